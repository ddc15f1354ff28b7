"""Parts of the solve at their edges: the interchange composition (perm_kernel)
on pivots that collide, point backwards or are all alike, and the fast sweeps
with every chain width, around 64-row blocks, plain and transposed."""
import numpy as np
import pytest

import oracle
from lair_gb300 import lapack

pytestmark = pytest.mark.gpu

EPS64 = 2.0 ** -53


def pivots(n, kind, rng):
    if kind == "random":
        return [int(rng.integers(i, n)) for i in range(n)]
    if kind == "any":
        return [int(v) for v in rng.integers(0, n, n)]
    if kind == "last":
        return [n - 1] * n
    if kind == "next":
        return [min(i + 1, n - 1) for i in range(n)]
    return [i ^ 1 if (i ^ 1) < n else i for i in range(n)]


@pytest.mark.parametrize("kind", ["random", "any", "last", "next", "pairs"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 1000, 20000])
def test_interchanges_of_any_pivots(n, kind):
    # L = U = I: the solve returns the permuted right-hand side exactly
    if n > 4000:
        from lair_gb300 import _lib
        import ctypes
        import torch

        rng = np.random.default_rng(n)
        piv = pivots(n, kind, rng)
        lu = torch.zeros((n, n), dtype=torch.float32, device="cuda")
        lu.diagonal().fill_(1.0)
        b = np.arange(n, dtype=np.float32)
        x = torch.from_numpy(b.copy()).cuda()
        p = torch.tensor(piv, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        lib, ctx = _lib.load(), _lib.context()
        _lib.check(lib.luhot_sgetrs_dev(ctx, n, 1, ctypes.c_void_p(lu.data_ptr()), n, ctypes.c_void_p(p.data_ptr()),
                                        ctypes.c_void_p(x.data_ptr()), 1, 0, _lib.MODE_FAST), ctx)
        got = x.cpu().numpy()
    else:
        rng = np.random.default_rng(n)
        piv = pivots(n, kind, rng)
        b = np.arange(n, dtype=np.float64)
        got = lapack.getrs(np.eye(n), piv, b)
    want = b.copy()
    for i, q in enumerate(piv):
        want[i], want[q] = want[q], want[i]
    assert np.array_equal(got, want)


@pytest.mark.parametrize("trans", [False, True])
@pytest.mark.parametrize("dtype,eps", [(np.float64, EPS64), (np.float32, 2.0 ** -24)])
@pytest.mark.parametrize("n,nrhs", [(1, 1), (63, 2), (64, 3), (65, 4), (129, 5), (200, 16), (257, 17), (2600, 16)])
def test_fast_sweeps(n, nrhs, dtype, eps, trans):
    rng = np.random.default_rng(n * 7 + nrhs)
    a = (rng.uniform(-1, 1, (n, n)) / np.sqrt(n) + 2 * np.eye(n)).astype(dtype)
    b = rng.uniform(-1, 1, (n, nrhs)).astype(dtype)
    lu = a.copy()
    piv, _ = oracle.getrf(lu)
    x = lapack.getrs(lu, piv, b, trans=trans)
    op = (a.T if trans else a).astype(np.float64)
    # normwise backward error of a backward-stable solve: n eps, with the
    # factors' own error of the same size
    r = np.abs(op @ x.astype(np.float64) - b).max()
    assert r <= 4 * n * eps * (np.abs(op).sum(1).max() * np.abs(x).max() + np.abs(b).max())
