"""Transposed FP32 solves wide enough for chains of four right-hand sides
(trsv_cluster_wide_kernel): orders around a CTA's 16 rows and the 64-row blocks,
whole and partial chains, a wide B; a launch takes 16 right-hand sides.

A = n I + U(-1, 1) has a condition number below 4 in the infinity norm and grows
little, so that solutions agree with an FP64 solve to 8 n eps."""
import ctypes

import numpy as np
import pytest

from lair_gb300 import _lib, lapack

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,nrhs,pad", [(1876, 16, 0), (2001, 15, 3), (2048, 17, 0), (2500, 13, 1), (6001, 5, 0),
                                        (10007, 3, 0), (2511, 33, 2), (4033, 64, 0)])
def test_wide_transposed_sweeps(n, nrhs, pad):
    assert n * min(nrhs, 16) > 30000 and min(nrhs, 16) > 2  # the rule
    rng = np.random.default_rng(n)
    a = (rng.uniform(-1, 1, (n, n)) + n * np.eye(n)).astype(np.float32)
    b = rng.standard_normal((n, nrhs)).astype(np.float32)
    fac = a.copy()
    piv, _ = lapack.getrf(fac, mode="fast")
    lib, ctx = _lib.load(), _lib.context()
    wide = np.full((n, nrhs + pad), 7.0, np.float32)
    wide[:, :nrhs] = b
    d_lu, d_b = torch.from_numpy(fac).cuda(), torch.from_numpy(wide).cuda()
    d_p = torch.tensor(piv, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    _lib.check(lib.luhot_sgetrs_dev(ctx, n, nrhs, ctypes.c_void_p(d_lu.data_ptr()), n, ctypes.c_void_p(d_p.data_ptr()),
                                    ctypes.c_void_p(d_b.data_ptr()), nrhs + pad, 1, 0), ctx)
    out = d_b.cpu().numpy()
    assert np.all(out[:, nrhs:] == 7.0)
    want = torch.linalg.solve(torch.from_numpy(a).cuda().double().T, torch.from_numpy(b).cuda().double()).cpu().numpy()
    assert np.abs(out[:, :nrhs] - want).max() <= 8 * n * np.finfo(np.float32).eps * np.abs(want).max()
