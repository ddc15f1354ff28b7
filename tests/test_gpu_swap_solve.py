"""Fast-mode getrf where the launch between panel and update (swap_solve.cu)
and the update's choice of kernel can go wrong: column groups of 8 and 16 with
remainders, panels narrower than 64, blocks on both sides of the tensor-core
rule (200 000 elements) and of the fine FP64 tiles, wide and tall shapes."""
import numpy as np
import pytest

from lair_gb300 import lapack, lu

pytestmark = pytest.mark.gpu

SHAPES = [(65, 66), (66, 65), (70, 200), (200, 73), (129, 700), (700, 129), (511, 460), (512, 470), (513, 513),
          (65, 4200), (1100, 1090), (2100, 1999)]


@pytest.mark.parametrize("dtype,eps", [(np.float64, 2.0 ** -53), (np.float32, 2.0 ** -24)])
@pytest.mark.parametrize("m,n", SHAPES)
def test_fast_factors(m, n, dtype, eps):
    rng = np.random.default_rng(m * 17 + n)
    a0 = rng.standard_normal((m, n)).astype(dtype)
    a = a0.copy()
    piv, sing = lapack.getrf(a, mode="fast")
    assert sing is None
    pa = a0.astype(np.float64)[lu.permutation(m, piv)]
    k = min(m, n)
    lo = np.tril(a.astype(np.float64), -1)[:, :k] + np.eye(m, k)
    up = np.triu(a.astype(np.float64))[:k]
    assert np.abs(lo).max() <= 1.0 + 4 * eps  # partial pivoting
    # the bound of the factorization tests: max |PA - LU| <= 10 n eps max |A|
    assert np.abs(pa - lo @ up).max() <= 10 * max(m, n) * eps * np.abs(a0).max()
