"""Around the rows up to which a panel runs in one cluster (panel_cluster.cu: FP64 3072
rows in fast mode and 1792 in exact mode, FP32 6144): exact mode bit for bit against
the oracle, fast mode with one and two rows per owner thread against the
definition and exact mode's pivots (lair's getrf, src/lapack/getrf.rs:46-120)."""
import numpy as np
import pytest

import oracle
from lair_gb300 import lapack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n", [(1777, 64), (1792, 64), (1793, 64), (1792, 33), (1821, 70), (2000, 64), (3841, 64)])
def test_exact_limit_bitwise(m, n):
    a = np.random.default_rng(m).uniform(-1, 1, (m, n))
    ref = a.copy()
    piv, sing = lapack.getrf(a, mode="exact")
    piv_r, sing_r = oracle.getrf(ref)
    assert piv == piv_r and sing == sing_r and np.array_equal(a, ref)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m,n", [(2048, 64), (2049, 64), (2560, 64), (2561, 20), (3071, 64), (3072, 64), (3073, 64),
                                 (3072, 200), (6144, 64), (6145, 64)])
def test_fast_limit(m, n, dtype):
    a0 = np.random.default_rng(m + n).standard_normal((m, n)).astype(dtype)
    a, ex = a0.copy(), a0.copy()
    piv, sing = lapack.getrf(a, mode="fast")
    piv_e, _ = lapack.getrf(ex, mode="exact")
    assert sing is None
    if dtype == np.float64:
        assert piv == piv_e
    pa = a0.astype(np.float64)
    for i, p in enumerate(piv):
        pa[[i, p]] = pa[[p, i]]
    lo = np.tril(a.astype(np.float64), -1) + np.eye(m, n)
    assert np.abs(lo).max() <= 1.0
    assert np.abs(pa - lo @ np.triu(a.astype(np.float64))[:n]).max() < n * np.finfo(dtype).eps * np.abs(a0).max()
