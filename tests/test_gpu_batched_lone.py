"""Batched plans of no more systems than SMs, whose large FP64 systems in scratch run on
CTAs of eight warps (kLone in batched.cu), and of one more: exact mode bit for bit
against the oracle, and fast mode the same bits whatever the plan."""
import numpy as np
import pytest

import oracle
from lair_gb300 import batched

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[256], [129], [168, 200, 255], [256, 1, 64, 170], [129] * 3 + [8] * 40])
def test_few_systems_exact(sizes):
    rng = np.random.default_rng(sum(sizes))
    mats = [rng.uniform(-1, 1, (n, n)) for n in sizes]
    rhs = [rng.uniform(-1, 1, n) for n in sizes]
    a, b = batched.pack(mats, rhs)
    piv, info = batched.BatchSolver(sizes, mode="exact").solve(a, b)
    assert (info < 0).all()
    for (lu, x, p), m, r in zip(batched.unpack(sizes, a, b, piv), mats, rhs):
        ref = m.copy()
        piv_r, _ = oracle.getrf(ref)
        assert list(p) == piv_r and np.array_equal(lu, ref) and np.array_equal(x, oracle.getrs(ref, piv_r, r.copy()))


def test_the_plan_does_not_change_the_bits():
    torch = pytest.importorskip("torch")
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rng = np.random.default_rng(5)
    n = 173
    mats = [rng.uniform(-1, 1, (n, n)) for _ in range(sms + 1)]
    rhs = [rng.uniform(-1, 1, n) for _ in range(sms + 1)]
    outs = []
    for count in (1, sms, sms + 1):
        a, b = batched.pack(mats[:count], rhs[:count])
        piv, _ = batched.BatchSolver([n] * count).solve(a, b)
        outs.append((a, b, piv))
    for a, b, piv in outs[:2]:
        assert np.array_equal(a, outs[2][0][:a.size]) and np.array_equal(b, outs[2][1][:b.size])
        assert np.array_equal(piv, outs[2][2][:piv.size])
