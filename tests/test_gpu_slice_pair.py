"""Fast-mode FP64 getrf's paired panels: two panels of 64 columns and one
trailing update with K = 128 on the FP16 slice products
(lair_gb300/csrc/getrf.cu, ozaki.cu), taken while the block behind the pair has
at least 16e6 elements.

The K = 128 product against its integer restatement, bit for bit, and the
paired factorization against the DMMA engine, which updates panel by panel
(lair's trailing update is FP64 inside getrf_row_major,
src/lapack/getrf.rs:46-120).
"""
import numpy as np
import pytest

import ozaki_emulation as oz
from lair_gb300 import _lib, lapack

pytestmark = pytest.mark.gpu


def product_row(c, l, u):
    """c - l u for one row of C (l: 128 elements, u: 128 x N) in the kernel's
    arithmetic: integer group sums, R = floor(sum_G T_G 2^(38 - 8 G)), one
    rounding of R and one of the subtraction."""
    ea, eb = oz.exponents(l[None, :], 1), oz.exponents(u, 0)
    a, b = oz.digits(l[None, :], ea[:, None]), oz.digits(u, eb[None, :])
    r = None
    for g in range(oz.GROUPS - 1, -1, -1):
        t = sum(a[p] @ b[g - p] for p in range(g + 1)) << oz.FRAC
        r = t if r is None else t + (r >> 8)
    s = (ea[:, None] + eb[None, :] - (oz.FRAC + 16)).astype(np.int32)
    return (c - np.ldexp(r.astype(np.float64), s))[0]


@pytest.mark.parametrize("kind", ["random", "extreme", "zeros"])
def test_pair_product_bit_exact(kind):
    """[[I, W], [V, C]] with |V| < 1: the pair leaves V and W as they are, and the
    row that the 129th pivot picks is one row of C - V W, all of it in U."""
    rng = np.random.default_rng(len(kind))
    m, n, k = 4141, 4203, 128
    full = rng.standard_normal((m, n))
    full[:k, :k] = np.eye(k)
    if kind == "extreme":
        # Digits 255, 127, .., 127, 120: the groups' sums come as near to 2^24 as
        # they can with all products of one sign (and past it for group 6).
        x = 255.0 / 256 + sum(127.0 * 256.0 ** -(p + 1) for p in range(1, 6)) + 120.0 * 256.0 ** -7
        full[k:, :k] = x * rng.choice([-1.0, 1.0], (m - k, 1))
        full[:k, k:] = x * rng.choice([-1.0, 1.0], (1, n - k)) * np.exp2(rng.integers(-9, 9, (1, n - k)))
    else:
        full[k:, :k] = rng.uniform(-1, 1, (m - k, k))
        full[:k, k:] *= np.exp2(rng.integers(-30, 30, (1, n - k)))
        if kind == "zeros":
            full[k:, :k] *= rng.random((m - k, k)) < 0.02
            full[:k, k::3] = 0.0
    lu = full.copy()
    piv, sing = lapack.getrf(lu, mode="fast")
    assert sing is None or sing < 0
    assert list(piv[:k]) == list(range(k))
    p = piv[k]
    want = product_row(full[p, k:], full[p, :k], full[:k, k:])
    assert np.array_equal(lu[k, k:], want)


@pytest.mark.parametrize("m,n", [(4131, 4131), (4100, 4900), (4900, 4100)])
def test_pair_matches_dmma(m, n):
    rng = np.random.default_rng(m + 3 * n)
    a0 = rng.standard_normal((m, n))
    outs = []
    try:
        for engine in ("dmma", "auto"):
            _lib.set_fp64_update(engine)
            a = a0.copy()
            piv, _ = lapack.getrf(a, mode="fast")
            outs.append((a, list(piv)))
    finally:
        _lib.set_fp64_update("auto")
    (a_d, piv_d), (a_p, piv_p) = outs
    assert piv_p == piv_d
    assert np.abs(a_p - a_d).max() <= 1e-11 * np.abs(a_d).max()
    w = min(m, n)
    lo, up = np.tril(a_p[:, :w], -1), np.triu(a_p[:w])
    lo[np.arange(w), np.arange(w)] = 1.0
    pa = a0.copy()
    for i, p in enumerate(piv_p):
        pa[[i, p]] = pa[[p, i]]
    assert np.abs(pa - lo @ up).max() < w * np.finfo(float).eps * np.abs(a0).max()
