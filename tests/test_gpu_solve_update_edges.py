"""Fast-mode getrf where the launch between panel and update (swap_solve.cu) and the
update's engine change: trailing blocks of 255, 256 and 257 rows or columns behind
the first panel, column groups of 8 and 16 with remainders
(max |PA - LU| <= 10 n eps max |A|, the bound of the factorization tests)."""
import numpy as np
import pytest

from lair_gb300 import lapack, lu

pytestmark = pytest.mark.gpu

SHAPES = [(319, 319), (320, 320), (321, 321), (319, 900), (320, 900), (900, 319), (900, 320), (900, 321), (320, 321),
          (384, 391), (391, 400), (128, 2000), (2000, 129)]


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
    assert np.abs(lo).max() <= 1.0 + 4 * eps
    assert np.abs(pa - lo @ up).max() <= 10 * max(m, n) * eps * np.abs(a0).max()
