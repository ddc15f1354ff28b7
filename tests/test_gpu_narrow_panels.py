"""Fast-mode getrf with panels narrower than 64 columns (luhot_set_block), in particular
beside the rest of a step (look-ahead, from 1e6 / 5e5 elements on) and in front of
slice updates, whose K is the panel's width: the pivots of exact mode (FP64) and
max |PA - LU| < n eps max |A| (lair's getrf, src/lapack/getrf.rs:46-120)."""
import numpy as np
import pytest

from lair_gb300 import _lib, lapack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nb", [5, 16, 17, 33, 48, 63])
@pytest.mark.parametrize("m,n", [(300, 300), (1200, 1200), (1100, 1700), (2501, 1003)])
def test_narrow_panels(m, n, nb, dtype):
    lib, ctx = _lib.load(), _lib.context()
    a0 = np.random.default_rng(m + nb).standard_normal((m, n)).astype(dtype)
    a, ex = a0.copy(), a0.copy()
    try:
        _lib.check(lib.luhot_set_block(ctx, nb), ctx)
        piv, sing = lapack.getrf(a, mode="fast")
    finally:
        _lib.check(lib.luhot_set_block(ctx, 0), ctx)
    assert sing is None
    if dtype == np.float64:
        assert piv == lapack.getrf(ex, mode="exact")[0]
    pa = a0.astype(np.float64)
    for i, p in enumerate(piv):
        pa[[i, p]] = pa[[p, i]]
    k = min(m, n)
    f = a.astype(np.float64)
    lo = np.tril(f, -1)[:, :k] + np.eye(m, k)
    assert np.abs(lo).max() <= 1.0
    assert np.abs(pa - lo @ np.triu(f)[:k]).max() < k * np.finfo(dtype).eps * np.abs(a0).max()
