"""The cluster panel's split of rows over owner warps and threads
(panel_cluster.cu): one to four owner warps, one and two rows per owner thread
(FP64 from 2049 rows on), the largest panel the cluster takes (FP64 2560 rows),
and the widths at which a column's exchange changes (no next column, no
segment, segments of one piece).  Exact mode against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
from lair_gb300 import lapack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["plain", "ties", "singular"])
@pytest.mark.parametrize("m,n", [(512, 3), (513, 2), (1024, 4), (1025, 64), (1537, 33), (2050, 64), (2560, 48),
                                 (2561, 48), (300, 128), (512, 128), (513, 128)])
@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_panel_roles_bitwise(m, n, dtype, kind):
    rng = np.random.default_rng(7 * m + n)
    a = rng.uniform(-1, 1, (m, n))
    if kind == "ties":
        a = np.round(a * 4) / 4
    elif kind == "singular":
        a[:, n // 2] = 0.0
        a[:, n - 1] = np.nan
        a[m // 3] = 0.0
    a = a.astype(dtype)
    ref = a.copy()
    piv, sing = lapack.getrf(a, mode="exact")
    piv_r, sing_r = oracle.getrf(ref)
    assert piv == piv_r and sing == sing_r
    assert np.array_equal(a, ref, equal_nan=True)
