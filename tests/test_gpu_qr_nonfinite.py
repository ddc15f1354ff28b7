"""FP64 fast QR of matrices with a NaN or an infinity, against lair's arithmetic (the
oracle's geqrf): a reflector reaches the rows from its own to its last non-zero one
(src/lapack/larf.rs, ilalr), so the rows of R above the first reflector that meets
the element stay what they are, and so does a matrix whose tau are all zero."""
import numpy as np
import pytest

import oracle
from lair_gb300 import qr

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def matrix(kind, m, n):
    a = np.random.default_rng(m * 3 + n).standard_normal((m, n))
    if kind == "nan early":
        a[3, 5] = np.nan
    elif kind == "inf in the middle":
        a[m // 2, n // 2] = np.inf
    elif kind == "nan last":
        a[-1, -1] = np.nan
    elif kind == "banded, nan":
        a = np.tril(np.triu(a, -2), 4)
        k = min(m, n) - 3
        a[k, k] = np.nan
    elif kind == "upper triangular, inf":
        a = np.triu(a)
        a[2, n - 2] = -np.inf
    return a


@pytest.mark.parametrize("kind", ["nan early", "inf in the middle", "nan last", "banded, nan", "upper triangular, inf"])
@pytest.mark.parametrize("m,n", [(32, 33), (100, 70), (90, 200), (500, 129)])
def test_rows_the_element_does_not_reach(m, n, kind):
    a0 = matrix(kind, m, n)
    ref = a0.copy()
    tau_r = oracle.geqrf(ref)
    f = qr.Factorized(a0.copy())
    ok = np.isfinite(ref)
    assert np.array_equal(np.isfinite(f.qr), ok)
    assert np.array_equal(np.isfinite(f.tau), np.isfinite(tau_r))
    # the bound of the fast QR tests, 20 k eps, of each column's norm
    finite = np.where(np.isfinite(a0), a0, 0.0)
    tol = np.broadcast_to(20 * min(m, n) * EPS * np.linalg.norm(finite, axis=0), a0.shape)
    upper = np.triu(np.ones((m, n), bool)) & ok
    assert (np.abs(f.qr - np.where(ok, ref, 0.0))[upper] <= tol[upper]).all()
