"""Which engine the default (AUTO) takes for a trailing update of fast-mode FP64
getrf (lair's update is FP64 throughout, src/lapack/getrf.rs:76-89): the integer
slices from 256 x 256 on, FP64 MMAs below, also where the update is cut into
parts; and the error of the blocks below on rows of mixed scale."""
import numpy as np
import pytest

from lair_gb300 import _lib, lapack

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def update(full, k, engine):
    lib, ctx = _lib.load(), _lib.context()
    m, n = full.shape
    d = torch.from_numpy(full).cuda()
    torch.cuda.synchronize()
    _lib.check(lib.luhot_dschur_update_dev(ctx, m, n, k, d.data_ptr(), n, _lib.FP64_UPDATES[engine]), ctx)
    return d.cpu().numpy()


@pytest.mark.parametrize("m,n,engine", [(255, 255, "dmma"), (255, 5000, "dmma"), (5000, 255, "dmma"), (128, 64, "dmma"),
                                        (128, 4000, "dmma"), (4000, 64, "dmma"), (256, 256, "ozaki"), (256, 900, "ozaki"),
                                        (2000, 257, "ozaki")])
def test_rule_of_one_update(m, n, engine):
    full = np.random.default_rng(m + n).standard_normal((m + 64, n + 64))
    assert np.array_equal(update(full, 64, "auto"), update(full, 64, engine))


@pytest.mark.parametrize("m,n", [(319, 319), (3000, 160), (160, 3000), (319, 8000), (8000, 319)])
def test_factorizations_below_the_rule(m, n):
    """No trailing block reaches 256 x 256 (with and without look-ahead): every bit is
    the DMMA engine's."""
    a0 = np.random.default_rng(m * 3 + n).standard_normal((m, n))
    outs = []
    try:
        for engine in ("dmma", "auto"):
            _lib.set_fp64_update(engine)
            a = a0.copy()
            outs.append((a, list(lapack.getrf(a, mode="fast")[0])))
    finally:
        _lib.set_fp64_update("auto")
    assert outs[0][1] == outs[1][1] and np.array_equal(outs[0][0], outs[1][0])


@pytest.mark.parametrize("m,n", [(1000, 200), (200, 1000), (255, 255), (4000, 64)])
def test_rows_of_mixed_scale_below_the_rule(m, n):
    rng = np.random.default_rng(m)
    full = rng.standard_normal((m + 64, n + 64))
    full[:32, 64:] *= 1e10       # the first half of U12's rows
    full[64:64 + m // 2, :32] = 0.0  # meets zeros in half of L21's rows
    got = update(full, 64, "auto")[64:, 64:]
    c, l, u = full[64:, 64:], full[64:, :64], full[:64, 64:]
    exact = c.astype(np.longdouble) - l.astype(np.longdouble) @ u.astype(np.longdouble)
    # a K-term sum of FP64 products: (K + 1) eps of |C| + |L||U|
    assert float((np.abs(got - exact) / (np.abs(c) + np.abs(l) @ np.abs(u))).max()) <= 65 * 2.0 ** -53
