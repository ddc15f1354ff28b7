"""Fast-mode getrf with the next panel beside the rest of a step (la_loop in
getrf.cu, taken while the block behind the next panel is large) against exact
mode, which goes step by step, and against the definition.

Square, wide, tall and odd sizes, the first sizes that take it (FP64 1128, FP32
836) and ones below; FP64: the pivots of exact mode, factors to 1e-11 of max |LU|;
both types: |L| <= 1 and max |PA - LU| < n eps max |A|; the caller's stream."""
import ctypes

import numpy as np
import pytest

from lair_gb300 import _lib, lapack

pytestmark = pytest.mark.gpu


def permuted(a, piv):
    pa = a.copy()
    for i, p in enumerate(piv):
        pa[[i, p]] = pa[[p, i]]
    return pa


def check(a0, lu, piv):
    k = min(a0.shape)
    lo, up = np.tril(lu[:, :k], -1).astype(np.float64), np.triu(lu[:k]).astype(np.float64)
    assert np.abs(lo).max() <= 1.0
    lo[np.arange(k), np.arange(k)] = 1.0
    err = np.abs(permuted(a0, piv).astype(np.float64) - lo @ up).max()
    assert err < k * np.finfo(a0.dtype).eps * np.abs(a0).max()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m,n", [(835, 835), (836, 836), (1127, 1127), (1128, 1128), (1999, 2003), (300, 9000),
                                 (9000, 300), (2700, 1301)])
def test_lookahead(m, n, dtype):
    rng = np.random.default_rng(m + 2 * n)
    a0 = rng.standard_normal((m, n)).astype(dtype)
    lu = a0.copy()
    piv, sing = lapack.getrf(lu, mode="fast")
    assert sing is None
    check(a0, lu, piv)
    if dtype == np.float64:
        ex = a0.copy()
        piv_e, _ = lapack.getrf(ex, mode="exact")
        assert list(piv) == list(piv_e)
        assert np.abs(lu - ex).max() <= 1e-11 * np.abs(ex).max()


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_lookahead_on_a_stream(dtype):
    """Input written on the caller's stream just before, result read on it."""
    torch = pytest.importorskip("torch")
    lib, ctx = _lib.load(), _lib.context()
    n = 1500
    a0 = np.random.default_rng(5).standard_normal((n, n)).astype(dtype)
    want = a0.copy()
    piv_w, _ = lapack.getrf(want, mode="fast")
    st = torch.cuda.Stream()
    fn = lib.luhot_dgetrf_dev if dtype == np.float64 else lib.luhot_sgetrf_dev
    try:
        _lib.check(lib.luhot_set_stream(ctx, ctypes.c_void_p(st.cuda_stream)), ctx)
        with torch.cuda.stream(st):
            src = torch.from_numpy(a0).cuda()
            for _ in range(3):
                d = src * 1.0
                piv = torch.zeros(n, dtype=torch.int32, device="cuda")
                sing = ctypes.c_int64()
                _lib.check(fn(ctx, n, n, ctypes.c_void_p(d.data_ptr()), n, ctypes.c_void_p(piv.data_ptr()),
                              ctypes.byref(sing), 0), ctx)
                got = (d * 1.0).cpu().numpy()
                assert np.array_equal(got, want) and piv.cpu().tolist() == list(piv_w)
    finally:
        _lib.check(lib.luhot_set_stream(ctx, None), ctx)
