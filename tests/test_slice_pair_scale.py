"""The K = 128 slice product of fast-mode FP64 getrf (lair_gb300/csrc/ozaki.cu) where the
two K halves differ in scale (lair's update is FP64 throughout,
src/lapack/getrf.rs:76-89): the halves share their exponents unless some row's and
some column's halves lie more than two bits apart; then the product is that of two
of K = 64.

The rule on its integer restatement, against exact arithmetic (CPU), and the
paired factorization's product against the restatement, bit for bit (GPU)."""
import numpy as np
import pytest

import ozaki_emulation as oz

APART = 2


def half_exponents(x, axis):
    """Exponents of both halves along `axis` (length 128), zero halves as oz.ZERO."""
    out = []
    for part in np.split(x, 2, axis=axis):
        e = oz.exponents(part, axis)
        out.append(np.where((part == 0).all(axis=axis), oz.ZERO, e))
    return out


def group_sums(l, u, ea, eb):
    """R = floor(sum_G T_G 2^(38 - 8G)) for one row l and all columns of u."""
    a, b = oz.digits(l[None, :], ea), oz.digits(u, eb[None, :])
    r = None
    for g in range(oz.GROUPS - 1, -1, -1):
        t = sum(a[p] @ b[g - p] for p in range(g + 1)) << oz.FRAC
        r = t if r is None else t + (r >> 8)
    return r[0]


def pair_row(c, l, u, rows_apart=None):
    """c - l u (l: 128 elements, u: 128 x N) as the GPU computes it; rows_apart: whether
    any row of L has its halves apart (default: this one)."""
    el, eu = half_exponents(l, 0), half_exponents(u, 0)
    if rows_apart is None:
        rows_apart = abs(el[0] - el[1]) > APART
    apart = rows_apart and (np.abs(eu[0] - eu[1]) > APART).any()
    if not apart:
        el, eu = [np.maximum(*el)] * 2, [np.maximum(*eu)] * 2
    el, eu = [np.where(e == oz.ZERO, 0, e) for e in el], [np.where(e == oz.ZERO, 0, e) for e in eu]
    halves = [slice(0, 64), slice(64, 128)] if apart else [slice(0, 128)]
    out = c
    for h, ks in enumerate(halves):
        s = np.clip(el[h] + eu[h] - (oz.FRAC + 16), -4000, 4000).astype(np.int32)
        with np.errstate(over="ignore", invalid="ignore"):
            out = out - np.ldexp(group_sums(l[ks], u[ks], el[h], eu[h]).astype(np.float64), s)
        out = np.where((el[h] >= oz.NONFINITE) | (eu[h] >= oz.NONFINITE), np.nan, out)
    return out


def worst(got, c, l, u):
    ld = np.longdouble
    exact = c.astype(ld) - (l.astype(ld)[:, None] * u.astype(ld)).sum(0)
    return float((np.abs(got - exact) / (np.abs(c) + np.abs(l) @ np.abs(u))).max())


@pytest.mark.parametrize("bits", [0, 1, 2, 3, 5, 20, 33, 200])
@pytest.mark.parametrize("zero", [0, 1])
def test_scaled_half_against_zeros(bits, zero):
    """One half of U's rows scaled up, a row of L that is zero against it, and a row
    that is not: within the rounding of an FP64 sum at every scale (a shared exponent
    leaves 2^bits of 2^-53 there)."""
    rng = np.random.default_rng(bits)
    u = rng.standard_normal((128, 300))
    l = rng.uniform(-1, 1, 128)
    c = rng.standard_normal(300)
    big = slice(64 * zero, 64 * zero + 64)
    u[big] *= 2.0 ** bits
    assert worst(pair_row(c, l, u), c, l, u) <= 2.0 ** -50
    l[big] = 0.0
    assert worst(pair_row(c, l, u), c, l, u) <= 2.0 ** -50


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["first", "second", "some columns", "two bits", "three bits", "zero half", "graded",
                                  "tiny", "nan", "rows alone", "columns alone"])
def test_pair_with_halves_apart_bit_exact(kind):
    """[[I, W], [V, C]] with |V| < 1: the pair leaves V and W as they are, and the row
    that the 129th pivot picks (given a large first element) is one row of C - V W."""
    from lair_gb300 import lapack

    rng = np.random.default_rng(len(kind))
    m, n, k = 4141, 4203, 128
    full = rng.standard_normal((m, n))
    full[:k, :k] = np.eye(k)
    full[k:, :k] = rng.uniform(-1, 1, (m - k, k))
    p = k + 77 * len(kind)
    v, w = full[:, :k], full[:k, k:]
    if kind == "first":
        w[:64] *= 1e6
        v[p, :64] = 0.0
    elif kind == "second":
        w[64:] *= 1e10
        v[p, 64:] = 0.0
    elif kind == "some columns":
        w[:64, 5::7] *= 2.0 ** 30
        v[p, :64] *= 2.0 ** -40
    elif kind in ("two bits", "three bits"):
        w[:] = np.sign(w) * 0.75
        w[64:] *= 4.0 if kind == "two bits" else 8.0
        v[p, 64:] = 0.0
    elif kind == "zero half":
        w[:64, 3::5] = 0.0
        w[64:, 4::5] = 0.0
        v[p, :64] = 0.0
    elif kind == "graded":
        w *= 10.0 ** -np.arange(k)[:, None]
        v[p] *= 10.0 ** -np.arange(k)[::-1]
    elif kind == "tiny":
        w[:64] *= 2.0 ** -1040
        v[p, 64:] = 0.0
    elif kind == "rows alone":
        v[p, 64:] *= 2.0 ** -20
    elif kind == "columns alone":
        w[64:] *= 1e8
    else:
        w[3, 11] = np.nan
        w[100, 12] = np.inf
        v[p, 64:] *= 2.0 ** -20
    full[p, k] = 2.0 ** 60  # the 129th pivot
    c = full[p, k:].copy()
    e0, e1 = half_exponents(v[k:], 1)
    want = pair_row(c, v[p].copy(), w.copy(), (np.abs(e0 - e1) > APART).any())
    if kind not in ("nan", "tiny"):
        assert worst(want, c, v[p], w) <= 2.0 ** -50
    lu = full.copy()
    piv, _ = lapack.getrf(lu, mode="fast")
    assert list(piv[:k]) == list(range(k)) and piv[k] == p
    assert np.array_equal(lu[k, k:], want, equal_nan=True)
