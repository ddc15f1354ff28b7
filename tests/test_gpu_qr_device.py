"""luhot_dgeqrf_dev in fast mode (lair's lapack::geqrf, src/lapack/geqrf.rs:9-27,
on a device matrix): the blocked form's result is complete, and its status read,
when the call returns, so that a call on another stream right behind it shares
the context's workspace safely; leading dimensions above n; calls under capture."""
import ctypes

import numpy as np
import pytest

from lair_gb300 import _lib, lapack, qr

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def on_stream(lib, ctx, st):
    _lib.check(lib.luhot_set_stream(ctx, ctypes.c_void_p(st.cuda_stream) if st else None), ctx)


def geqrf_dev(lib, ctx, d, tau, m, n, lda):
    _lib.check(lib.luhot_dgeqrf_dev(ctx, m, n, ctypes.c_void_p(d.data_ptr()), lda, ctypes.c_void_p(tau.data_ptr()), 0), ctx)


@pytest.mark.parametrize("m,n,lda", [(32, 32, 37), (700, 300, 301), (300, 700, 1024), (2100, 1000, 1003)])
def test_device_entry_matches_host_entry(m, n, lda):
    lib, ctx = _lib.load(), _lib.context()
    a0 = np.random.default_rng(m + lda).standard_normal((m, n))
    host = a0.copy()
    tau_h = qr.geqrf(host)
    d = torch.full((m, lda), 7.0, dtype=torch.float64, device="cuda")
    d[:, :n] = torch.from_numpy(a0)
    tau = torch.zeros(min(m, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    geqrf_dev(lib, ctx, d, tau, m, n, lda)
    torch.cuda.synchronize()
    assert np.array_equal(d[:, :n].cpu().numpy(), host) and np.array_equal(tau.cpu().numpy(), tau_h)
    assert bool((d[:, n:] == 7.0).all())


def test_result_is_complete_on_return_and_streams_may_change():
    lib, ctx = _lib.load(), _lib.context()
    rng = np.random.default_rng(3)
    qm, qn, ln = 2000, 1500, 1500
    a0, b0 = rng.standard_normal((qm, qn)), rng.standard_normal((ln, ln))
    qr_w, lu_w = a0.copy(), b0.copy()
    tau_w = qr.geqrf(qr_w)
    piv_w, _ = lapack.getrf(lu_w, mode="fast")
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    try:
        for _ in range(3):
            a, b = torch.from_numpy(a0).cuda(), torch.from_numpy(b0).cuda()
            tau = torch.zeros(qn, dtype=torch.float64, device="cuda")
            piv = torch.zeros(ln, dtype=torch.int32, device="cuda")
            torch.cuda.synchronize()
            on_stream(lib, ctx, s1)
            geqrf_dev(lib, ctx, a, tau, qm, qn, qn)
            assert s1.query()  # nothing of it is still under way
            on_stream(lib, ctx, s2)
            sing = ctypes.c_int64()
            _lib.check(lib.luhot_dgetrf_dev(ctx, ln, ln, ctypes.c_void_p(b.data_ptr()), ln,
                                            ctypes.c_void_p(piv.data_ptr()), ctypes.byref(sing), 0), ctx)
            torch.cuda.synchronize()
            assert np.array_equal(a.cpu().numpy(), qr_w) and np.array_equal(tau.cpu().numpy(), tau_w)
            assert np.array_equal(b.cpu().numpy(), lu_w) and piv.cpu().tolist() == list(piv_w)
    finally:
        on_stream(lib, ctx, None)


def test_under_capture():
    """The call records on a stream under capture (its workspace made by an earlier
    call), and every replay factors what is in the buffer then."""
    lib, ctx = _lib.load(), _lib.context()
    m, n = 120, 64
    rng = np.random.default_rng(8)
    d = torch.zeros((m, n), dtype=torch.float64, device="cuda")
    tau = torch.zeros(n, dtype=torch.float64, device="cuda")
    st = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    try:
        on_stream(lib, ctx, st)
        geqrf_dev(lib, ctx, d, tau, m, n, n)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=st):
            geqrf_dev(lib, ctx, d, tau, m, n, n)
        for _ in range(2):
            a0 = rng.standard_normal((m, n))
            d.copy_(torch.from_numpy(a0))
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            want = a0.copy()
            tau_w = qr.geqrf(want, mode="exact")
            # two roundings of the same reflectors: the bounds of the fast QR tests
            assert np.abs(d.cpu().numpy() - want).max() <= 1e-10 * np.abs(a0).max() * np.sqrt(m)
            assert np.abs(tau.cpu().numpy() - tau_w).max() <= 1e-10
    finally:
        on_stream(lib, ctx, None)
