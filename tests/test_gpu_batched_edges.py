"""Batched systems in exact mode, bit for bit against the oracle, where the
panel warp's search leaves its short path (ties, zero and NaN columns, infinite
and subnormal pivots) and around the edges of the size classes."""
import numpy as np
import pytest

import oracle
from lair_gb300 import batched

pytestmark = pytest.mark.gpu

SIZES = [1, 3, 8, 9, 16, 17, 31, 32, 33, 64, 65, 97, 128, 129, 161, 168, 169, 235, 236, 256]


@pytest.mark.parametrize("kind", ["ties", "zero", "nan", "wide"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_exact_edges(dtype, kind):
    rng = np.random.default_rng(7)
    mats = []
    for n in SIZES:
        a = rng.uniform(-1, 1, (n, n))
        if kind == "ties":
            a = np.round(a * 2) / 2 + 2 * np.eye(n)[::-1]
        elif kind == "zero":
            a[:, n // 2] = 0.0
        elif kind == "nan":
            a[:, n - 1] = np.nan
        else:
            a *= np.exp2(rng.integers(-100, 100, (n, 1)) if dtype == np.float32 else rng.integers(-500, 500, (n, 1)))
            a[0, 0] = np.inf
        mats.append(a.astype(dtype))
    rhs = [rng.uniform(-1, 1, n).astype(dtype) for n in SIZES]
    a, b = batched.pack(mats, rhs, dtype)
    piv, info = batched.BatchSolver(SIZES, dtype=dtype, mode="exact").solve(a, b)
    with np.errstate(all="ignore"):
        for (lu, x, pv), m, r, s in zip(batched.unpack(SIZES, a, b, piv), mats, rhs, info):
            ref = m.copy()
            piv_r, sing_r = oracle.getrf(ref)
            assert list(pv) == piv_r and (s if s >= 0 else None) == sing_r
            assert np.array_equal(lu, ref, equal_nan=True)
            assert np.array_equal(x, oracle.getrs(ref, piv_r, r.copy()), equal_nan=True)
