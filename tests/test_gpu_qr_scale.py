"""Blocked QR (geqrf_blocked.cu, fast mode, FP64) on rows of mixed scale: columns of
the first panel that fall into two groups of rows with nothing in common factor as
two problems, each to its own scale (lair's larf::left is FP64 throughout,
src/lapack/larf.rs)."""
import numpy as np
import pytest

import oracle
from lair_gb300 import qr

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


@pytest.mark.parametrize("scale", [1.0, 1e6, 1e12])
@pytest.mark.parametrize("m,n", [(300, 200), (1200, 732), (2600, 900)])
def test_decoupled_rows_keep_their_scale(m, n, scale):
    rng = np.random.default_rng(m)
    first = np.zeros(m, bool)
    first[:16] = True
    first[32:m // 2] = True
    a0 = rng.standard_normal((m, n))
    a0[np.ix_(~first, np.arange(16))] = 0.0
    a0[np.ix_(first, np.arange(16, 32))] = 0.0
    a0[first, 32:] *= scale
    f = qr.Factorized(a0.copy())
    for rows, cols in ((first, slice(0, 16)), (~first, slice(16, 32))):
        part = np.hstack([a0[rows, cols], a0[rows, 32:]])
        ref = part.copy()
        oracle.geqrf(ref)
        want = np.triu(ref)[:16]
        got = np.hstack([np.triu(f.qr[cols, cols]), f.qr[cols, 32:]])
        # the bound of the fast QR tests, 20 k eps, of each column's own norm
        norms = np.linalg.norm(part, axis=0)
        assert (np.abs(got - want) <= 20 * 32 * EPS * norms).all()
