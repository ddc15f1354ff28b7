"""Both forms of the batched kernel (matrices in shared memory, in scratch) in every size
bucket, whichever the autotuner would take: exact mode bit for bit against the
oracle (lair's getrf and getrs per system), where the panel warp's search leaves
its short path and around the edges of the buckets."""
import numpy as np
import pytest

import oracle
from lair_gb300 import _lib, batched

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 7, 8, 9, 15, 16, 17, 31, 32, 33, 63, 64, 65, 96, 97, 127, 128, 129, 160, 161, 167, 168, 192, 193, 224, 225,
         235, 236, 255, 256]


def systems(kind, dtype, rng):
    mats = []
    for n in SIZES:
        a = rng.uniform(-1, 1, (n, n))
        if kind == "ties":
            a = np.round(a * 2) / 2 + 2 * np.eye(n)[::-1]
        elif kind == "zero":
            a[:, n // 2] = 0.0
        elif kind == "nan":
            a[:, n - 1] = np.nan
        elif kind == "wide":
            a *= np.exp2(rng.integers(-100, 100, (n, 1)))
            a[0, 0] = np.inf
        mats.append(a.astype(dtype))
    return mats, [rng.uniform(-1, 1, n).astype(dtype) for n in SIZES]


@pytest.mark.parametrize("kind", ["plain", "ties", "zero", "nan", "wide"])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_both_forms(dtype, kind):
    mats, rhs = systems(kind, dtype, np.random.default_rng(23))
    plan = batched.BatchSolver(SIZES, dtype=dtype, mode="exact")
    want = []
    with np.errstate(all="ignore"):
        for m, r in zip(mats, rhs):
            lu = m.copy()
            piv, sing = oracle.getrf(lu)
            want.append((lu, oracle.getrs(lu, piv, r.copy()), piv, sing))
    for form in (0, 1):
        _lib.check(_lib.load().luhot_selftest_batch_form(plan._h, form), _lib.context())
        a, b = batched.pack(mats, rhs, dtype)
        piv, info = plan.solve(a, b)
        for (lu, x, p), s, (lu_w, x_w, p_w, s_w) in zip(batched.unpack(SIZES, a, b, piv), info, want):
            assert list(p) == p_w and (s if s >= 0 else None) == s_w
            assert np.array_equal(lu, lu_w, equal_nan=True) and np.array_equal(x, x_w, equal_nan=True)


@pytest.mark.parametrize("dtype,eps", [(np.float64, 2.0 ** -53), (np.float32, 2.0 ** -24)])
def test_fast_mode_in_both_forms(dtype, eps):
    rng = np.random.default_rng(29)
    mats, rhs = systems("plain", dtype, rng)
    plan = batched.BatchSolver(SIZES, dtype=dtype, mode="fast")
    outs = []
    for form in (0, 1):
        _lib.check(_lib.load().luhot_selftest_batch_form(plan._h, form), _lib.context())
        a, b = batched.pack(mats, rhs, dtype)
        plan.solve(a, b)
        outs.append((a, b))
        for (lu, x, _), m, r in zip(batched.unpack(SIZES, a, b, np.zeros(len(b), np.int32)), mats, rhs):
            m, x, r = m.astype(np.float64), x.astype(np.float64), r.astype(np.float64)
            n = len(r)
            # the bound of the batched tests: backward error 10 n eps
            assert np.abs(r - m @ x).max() <= 10 * n * eps * (np.abs(m).sum(1).max() * np.abs(x).max() + np.abs(r).max())
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])
