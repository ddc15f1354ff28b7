"""Blocked QR (geqrf_blocked.cu, fast mode, FP64) with columns at the ends of FP64's range,
against lair's arithmetic (the oracle's geqrf): each column's R to its own scale,
tau, and the columns whose squares underflow (tau = 0, kept as they are:
src/lapack/larfg.rs:9-16)."""
import numpy as np
import pytest

import oracle
from lair_gb300 import qr

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
SCALES = {"mixed small": [1e-150, 1e-180, 1e-100, 1.0, 1e-230, 1e-300], "large and small": [1e140, 1e-140, 1.0, 1e-200],
          "uniformly small": [1e-145], "uniformly large": [1e150], "subnormal": [1.0, 1e-310, 1e-150]}


@pytest.mark.parametrize("kind", sorted(SCALES))
@pytest.mark.parametrize("m,n", [(40, 33), (200, 64), (700, 100), (90, 200)])
def test_columns_at_the_ends_of_the_range(m, n, kind):
    rng = np.random.default_rng(m + n)
    scale = np.resize(SCALES[kind], n)
    a0 = rng.standard_normal((m, n)) * scale
    ref = a0.copy()
    tau_r = oracle.geqrf(ref)
    f = qr.Factorized(a0.copy())
    k = min(m, n)
    # the bound of the fast QR tests, 20 k eps, of each column's own norm; and on the
    # subnormal grid a sum of m products per reflector
    norms = np.abs(a0).max(axis=0) * np.sqrt(m)
    tol = 20 * k * EPS * norms + m * k * 5e-324
    assert (np.abs(np.triu(f.qr) - np.triu(ref)) <= tol).all()
    assert np.array_equal(f.tau == 0.0, tau_r == 0.0)
    np.testing.assert_allclose(f.tau, tau_r, rtol=0, atol=1e-10)
    kept = tau_r == 0.0
    below = np.tril(np.ones((m, k), bool), -1) & kept
    assert (np.abs(f.qr[:, :k] - ref[:, :k]) <= tol[:k])[below].all()
