"""Batched plans of one size class and of several, before and after the autotuner's
look at sample systems (more than it takes, and fewer): exact mode's bits (lair's
getrf and getrs per system) do not depend on the plan, and the samples are only
read."""
import numpy as np
import pytest

import oracle
from lair_gb300 import batched

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("lo,hi,count", [(1, 1, 3), (8, 24, 50), (8, 24, 700), (60, 70, 40), (1, 256, 120)])
def test_plans(lo, hi, count, dtype):
    rng = np.random.default_rng(hi + count)
    sizes = [int(n) for n in rng.integers(lo, hi + 1, count)]
    mats = [rng.uniform(-1, 1, (n, n)).astype(dtype) for n in sizes]
    rhs = [rng.uniform(-1, 1, n).astype(dtype) for n in sizes]
    a0, b0 = batched.pack(mats, rhs, dtype)
    want = []
    for m, r in zip(mats, rhs):
        lu = m.copy()
        piv, _ = oracle.getrf(lu)
        want.append((lu, oracle.getrs(lu, piv, r.copy()), piv))
    plan = batched.BatchSolver(sizes, dtype=dtype, mode="exact")
    d_a, d_b = torch.from_numpy(a0).cuda(), torch.from_numpy(b0).cuda()
    torch.cuda.synchronize()
    for tuned in (False, True):
        if tuned:
            plan.autotune(d_a.data_ptr(), d_b.data_ptr())
            assert np.array_equal(d_a.cpu().numpy(), a0) and np.array_equal(d_b.cpu().numpy(), b0)
        a, b = a0.copy(), b0.copy()
        piv, info = plan.solve(a, b)
        assert (info < 0).all()
        for (lu, x, p), (lu_w, x_w, p_w) in zip(batched.unpack(sizes, a, b, piv), want):
            assert list(p) == p_w and np.array_equal(lu, lu_w) and np.array_equal(x, x_w)
