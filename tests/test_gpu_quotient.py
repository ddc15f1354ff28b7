"""The quotients of fast mode's back substitution by a reciprocal and one correction
(quot in common.cuh) against IEEE division, on batched systems of one equation
(lair divides, src/lapack/getrs.rs:35): divisors across and around the guard
(1e-30 .. 1e30), subnormal operands, and quotients at the end of the range, where
the product with the reciprocal overflows and the division does not."""
import numpy as np
import pytest

from lair_gb300 import batched

pytestmark = pytest.mark.gpu


def quotients(y, d, dtype):
    n = len(y)
    a, b = d.astype(dtype).copy(), y.astype(dtype).copy()
    _, info = batched.BatchSolver([1] * n, dtype=dtype, mode="fast").solve(a, b)
    assert (info < 0).all()
    return b


def mantissas(rng, n, dtype):
    return (rng.uniform(1, 2, n) * rng.choice([-1.0, 1.0], n)).astype(dtype)


# Powers of two of (y, d); `ulps` of the correctly rounded quotient: one where y - q d
# is exact (the smallest bit of q d above the subnormal grid), two below, none where
# the division itself is taken.
RANGES = {
    np.float64: [("usual", (-60, 60), (-60, 60), 1), ("guard, small divisors", (-300, 300), (-99, -98), 1),
                 ("guard, large divisors", (-300, 300), (98, 99), 1), ("beyond, small", (-300, 300), (-1000, -101), 0),
                 ("beyond, large", (-300, 300), (101, 1000), 0), ("subnormal y", (-1074, -1022), (-99, 98), 2),
                 ("subnormal quotient", (-1000, -975), (60, 98), 2), ("subnormal d", (-1074, -1022), (-1074, -1022), 0)],
    np.float32: [("usual", (-20, 20), (-20, 20), 1), ("guard, small divisors", (-60, 20), (-99, -98), 1),
                 ("guard, large divisors", (-20, 20), (98, 99), 1), ("beyond, small", (-60, -20), (-120, -101), 0),
                 ("beyond, large", (-20, 20), (101, 120), 0), ("subnormal y", (-149, -126), (-20, 98), 2),
                 ("subnormal quotient", (-80, -60), (60, 80), 2), ("subnormal d", (-149, -126), (-149, -126), 0)],
}


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_quotients_against_division(dtype):
    rng = np.random.default_rng(17)
    n = 4000
    for name, ey, ed, ulps in RANGES[dtype]:
        y = np.ldexp(mantissas(rng, n, dtype), rng.integers(*ey, n)).astype(dtype)
        d = np.ldexp(mantissas(rng, n, dtype), rng.integers(*ed, n)).astype(dtype)
        keep = (d != 0) & (y != 0)
        y, d = y[keep], d[keep]
        with np.errstate(all="ignore"):
            want = y / d
        got = quotients(y, d, dtype)
        over = np.isinf(want)
        assert np.array_equal(got[over], want[over]), name
        got, want = got[~over], want[~over]
        assert (np.abs(got - want) <= ulps * np.spacing(np.abs(want))).all(), name


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_quotients_at_the_end_of_the_range(dtype):
    rng = np.random.default_rng(18)
    big = np.finfo(dtype).max
    d = rng.uniform(0.5, 1, 20000).astype(dtype)
    y = (d * big).astype(dtype)  # quotients of max, or a few units below
    y = np.where(np.arange(len(y)) % 2 == 0, y, np.nextafter(y, dtype(0)))
    with np.errstate(over="ignore"):
        want, product = y / d, y * (dtype(1) / d)
    assert (np.isinf(product) & np.isfinite(want)).any()  # the case is among them
    got = quotients(y, d, dtype)
    assert np.array_equal(np.isinf(got), np.isinf(want))
    fin = np.isfinite(want)
    assert (np.abs(got[fin] - want[fin]) <= 2 * np.spacing(want[fin] / 2)).all()
    for y, d in ((np.inf, 2.0), (np.nan, 2.0), (0.0, 3.0), (-0.0, 3.0)):
        assert np.array_equal(quotients(np.array([y]), np.array([d]), dtype), np.array([y / d], dtype), equal_nan=True)
