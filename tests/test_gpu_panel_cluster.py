"""The cluster form of the panel factorization (panel_cluster.cu) against the
oracle, bit for bit in exact mode: CTAs with no, one, few and several rows per
owner thread, the edges of the owner warps and of the rule that picks the form
(FP64 2048 rows, FP32 6144), ties, zero and NaN columns, zero rows."""
import numpy as np
import pytest

import oracle
from lair_gb300 import lapack

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (2, 1), (7, 3), (16, 16), (17, 17), (33, 32), (65, 5), (100, 100), (128, 127), (128, 128),
          (129, 128), (257, 64), (513, 64), (515, 128), (1030, 64), (2048, 64), (2049, 40)]


def matrix(m, n, dtype, kind):
    rng = np.random.default_rng(m * 131 + n)
    a = rng.uniform(-1, 1, (m, n))
    if kind == "ties":
        a = np.round(a * 4) / 4
    elif kind == "singular":
        a[:, n // 2] = 0.0
        a[:, n - 1] = np.nan
        a[m // 3] = 0.0
    return a.astype(dtype)


@pytest.mark.parametrize("kind", ["plain", "ties", "singular"])
@pytest.mark.parametrize("m,n,dtype", [(m, n, np.float64) for m, n in SHAPES] +
                         [(m, n, np.float32) for m, n in SHAPES + [(4100, 64), (6144, 33), (6145, 33)]])
def test_cluster_panel_bitwise(m, n, dtype, kind):
    a = matrix(m, n, dtype, kind)
    ref = a.copy()
    piv, sing = lapack.getrf(a, mode="exact")
    piv_r, sing_r = oracle.getrf(ref)
    assert piv == piv_r and sing == sing_r
    assert np.array_equal(a, ref, equal_nan=True)
