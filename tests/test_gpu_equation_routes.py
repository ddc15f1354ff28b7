"""equation.solve and solve_matrix by one device call (FP64) against factoring and
solving by two: the same bits for every layout of a and b that they take, both
modes, the same errors, and a and b as they were."""
import numpy as np
import pytest

from lair_gb300 import equation, lu
from lair_gb300.errors import InvalidInput

pytestmark = pytest.mark.gpu


def views(n, rng):
    a = rng.uniform(-1, 1, (n, n))
    big = rng.uniform(-1, 1, (2 * n, 3 * n))
    raw = np.zeros(8 * n * n + 1, dtype=np.uint8)
    odd = raw[1:].view(np.float64).reshape(n, n)
    odd[:] = a
    ro = a.copy()
    ro.flags.writeable = False
    return {"c": a, "f": np.asfortranarray(a), "reversed": a[::-1], "both": a[::-1, ::-1], "f reversed": a.T[:, ::-1],
            "strided": big[::2, ::3], "transposed strided": big[::2, ::3].T, "unaligned": odd, "read-only": ro}


@pytest.mark.parametrize("mode", ["fast", "exact"])
@pytest.mark.parametrize("n", [1, 2, 65, 130, 300])
def test_one_call_matches_two(n, mode):
    rng = np.random.default_rng(n)
    b2 = rng.uniform(-1, 1, (n, 6))
    bs = [b2[:, 0], b2[::-1, 1], np.ascontiguousarray(b2[:, 2]), np.broadcast_to(np.array([0.5]), (n,))]
    for name, a in views(n, rng).items():
        keep = a.copy()
        for b in bs:
            want = lu.Factorized(equation._to_owned(a), mode=mode).solve(b)
            got = equation.solve(a, b, mode=mode)
            assert got.shape == want.shape and np.array_equal(got, want), name
        for b in (b2, np.asfortranarray(b2), b2[:, ::-2]):
            want = lu.Factorized(equation._to_owned(a), mode=mode).solve_matrix(b)
            got = equation.solve_matrix(a, b, mode=mode)
            assert got.shape == want.shape and np.array_equal(got, want), name
        assert np.array_equal(a, keep)


def test_errors_are_the_same():
    a = np.ones((4, 4))
    with pytest.raises(InvalidInput):
        equation.solve(a, np.ones(4))
    with pytest.raises(InvalidInput):
        equation.solve(a, np.ones(4, np.float32))  # singular before mistyped
    with pytest.raises(TypeError):
        equation.solve(np.eye(4), np.ones(4, np.float32))
    with pytest.raises(InvalidInput):
        equation.solve(np.eye(4), np.ones(3))
    assert equation.solve(np.zeros((0, 0)), np.zeros(0)).shape == (0,)
    x = equation.solve(np.eye(3, dtype=np.float32), np.ones(3, np.float32))
    assert x.dtype == np.float32 and np.array_equal(x, np.ones(3, np.float32))
