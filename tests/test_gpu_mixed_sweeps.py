"""GMRES refinement applies the FP32 factors in FP64 sweeps (cluster_sweep<double, float>,
trsv_cluster.cu) until it has run long enough for block-scaled tiles: orders around
the 64-row blocks, to the accuracy of an FP64 solve."""
import numpy as np
import pytest

from lair_gb300 import refine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "bf16x3"])
@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 129, 500, 1001])
def test_gmres_on_fp32_factors(n, precision):
    rng = np.random.default_rng(n)
    a = rng.uniform(-1, 1, (n, n)) + n * np.eye(n)
    b = rng.standard_normal((n, 2))
    x, info = refine.gesv_ir(a, b, precision=precision, solver="gmres")
    assert info["converged"]
    want = np.linalg.solve(a, b)
    # condition number below 4: 8 n eps, as the sweeps' own tests
    assert np.abs(x - want).max() <= 8 * max(n, 8) * np.finfo(float).eps * np.abs(want).max()
