"""Blocked QR (geqrf_blocked.cu, fast mode, FP64) at the edges of its panels,
cluster splits, row ranges and update kernels: A = QR and Q^T Q = I, R and tau
against LAPACK's (same sign convention), zero columns and dependent columns."""
import numpy as np
import pytest

from lair_gb300 import qr

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53
SHAPES = [(32, 32), (33, 32), (32, 33), (40, 200), (63, 64), (100, 33), (129, 65), (300, 300), (257, 100), (1000, 70),
          (1500, 700), (4200, 40)]


def check(a0, f):
    m, n = a0.shape
    k = min(m, n)
    q, r = f.q(), f.r()
    scale = np.abs(a0).max()
    # the bounds of the fast-mode QR tests: 20 k eps
    assert np.abs(q @ r - a0).max() <= 20 * max(k, 32) * 2 * EPS * max(scale, 1.0)
    assert np.abs(q.T @ q - np.eye(m)).max() <= 20 * max(k, 32) * 2 * EPS


@pytest.mark.parametrize("m,n", SHAPES)
def test_blocked_qr(m, n):
    rng = np.random.default_rng(m * 3 + n)
    a0 = rng.standard_normal((m, n))
    f = qr.Factorized(a0.copy())
    check(a0, f)
    h, tau = np.linalg.qr(a0, mode="raw")
    np.testing.assert_allclose(f.tau, tau, rtol=0, atol=1e-10)
    np.testing.assert_allclose(np.triu(f.qr), np.triu(h.T), rtol=0, atol=1e-10 * np.abs(a0).max() * np.sqrt(m))


def test_blocked_qr_zero_and_dependent_columns():
    rng = np.random.default_rng(1)
    a0 = rng.standard_normal((200, 90))
    a0[:, 5] = 0.0
    a0[:, 40] = 0.0
    a0[:, 60] = a0[:, 3]
    a0[50:, 70] = 0.0
    f = qr.Factorized(a0.copy())
    check(a0, f)
    assert f.tau[5] == 0.0
