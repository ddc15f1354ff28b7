"""The triangular sweeps of fast-mode solves (trsv_cluster.cu): orders around the
edges of a CTA's 16 rows and of the 64-row blocks, one to seventeen right-hand
sides (a launch takes 16; FP32 chains of four), a wide B, both transposes, more
blocks than the chip holds at once, and the FP64 sweeps on FP32 factors.

A = n I + U(-1, 1) has a condition number below 4 in the infinity norm and grows
little, so that solutions agree with an FP64 solve to 8 n eps; the general path,
exact mode's sweeps, to twice that."""
import ctypes

import numpy as np
import pytest

from lair_gb300 import _lib, lapack, lu

pytestmark = pytest.mark.gpu


def system(n, nrhs, dtype, seed):
    rng = np.random.default_rng(seed)
    a = (rng.uniform(-1, 1, (n, n)) + n * np.eye(n)).astype(dtype)
    return a, rng.standard_normal((n, nrhs)).astype(dtype)


def solve_dev(torch, fac, piv, b, ldb, trans, mode):
    lib, ctx = _lib.load(), _lib.context()
    n, nrhs = b.shape
    wide = np.full((n, ldb), 7.0, b.dtype)
    wide[:, :nrhs] = b
    d_lu, d_b = torch.from_numpy(fac).cuda(), torch.from_numpy(wide).cuda()
    d_p = torch.tensor(piv, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    fn = lib.luhot_dgetrs_dev if b.dtype == np.float64 else lib.luhot_sgetrs_dev
    _lib.check(fn(ctx, n, nrhs, ctypes.c_void_p(d_lu.data_ptr()), n, ctypes.c_void_p(d_p.data_ptr()),
                  ctypes.c_void_p(d_b.data_ptr()), ldb, trans, mode), ctx)
    out = d_b.cpu().numpy()
    assert np.all(out[:, nrhs:] == 7.0)
    return out[:, :nrhs]


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,nrhs,pad", [(1, 1, 0), (2, 17, 0), (15, 1, 3), (16, 2, 0), (17, 3, 0), (48, 4, 1),
                                        (63, 5, 0), (64, 1, 0), (65, 16, 2), (80, 17, 0), (129, 33, 0), (255, 1, 0),
                                        (1000, 7, 0), (1874, 15, 0), (1876, 16, 5), (2500, 18, 0)])
def test_sweeps(n, nrhs, pad, dtype):
    torch = pytest.importorskip("torch")
    a, b = system(n, nrhs, dtype, 3 * n + nrhs)
    fac = a.copy()
    piv, _ = lapack.getrf(fac, mode="fast")
    eps = np.finfo(dtype).eps
    for trans in (0, 1):
        want = np.linalg.solve((a.T if trans else a).astype(np.float64), b.astype(np.float64))
        tol = 8 * n * eps * np.abs(want).max()
        got = solve_dev(torch, fac, piv, b, nrhs + pad, trans, 0)
        assert np.abs(got - want).max() <= tol
        exact = solve_dev(torch, fac, piv, b, nrhs + pad, trans, 1)
        assert np.abs(got - exact).max() <= 2 * tol


def test_sweeps_many_blocks():
    """9001 rows: 141 blocks of 4 CTAs for each of 5 right-hand sides."""
    torch = pytest.importorskip("torch")
    n, nrhs = 9001, 5
    a, b = system(n, nrhs, np.float64, 1)
    fac = a.copy()
    piv, _ = lapack.getrf(fac, mode="fast")
    for trans in (0, 1):
        got = solve_dev(torch, fac, piv, b, nrhs, trans, 0)
        res = np.abs((a.T if trans else a) @ got - b).max()
        assert res <= 8 * n * np.finfo(float).eps * np.abs(b).max()


@pytest.mark.parametrize("n", [1, 63, 64, 65, 128, 129, 255, 256, 257, 320, 321, 1000, 2049])
def test_resident_sweeps_in_clusters(n):
    """One right-hand side on resident factors (trsv_scaled.cu): fewer blocks than
    a cluster takes, whole clusters, one block and one row more; solved twice."""
    a, b = system(n, 1, np.float64, 11 * n)
    f = lu.Factorized(a.copy(), device_resident=True)
    want = np.linalg.solve(a, b[:, 0])
    for _ in range(2):
        got = np.asarray(f.solve(b[:, 0]))
        assert np.abs(got - want).max() <= 8 * n * np.finfo(float).eps * np.abs(want).max()
