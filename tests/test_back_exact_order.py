"""Exact mode's back substitution (back_exact_kernel, lair_gb300/csrc/getrs.cu) on an
emulated warp whose lanes drift apart: lair's bits (src/lapack/getrs.rs:30-36) hold
whichever lane lags behind a barrier, with x in shared and in global memory."""
import numpy as np
import pytest

import warp_emulation as warp

BODY = r"""
static int lag;  // the lane that falls behind at every barrier; 32: all but lane 0
static void __syncwarp() {
  lanes_meet();
  if (lag == 32 ? threadIdx.x != 0 : threadIdx.x == lag) std::this_thread::sleep_for(std::chrono::microseconds(300));
}
static double mul_rn(double a, double b) { return a * b; }
static double chain_sub(double a, double b) { return a - b; }
alignas(16) static unsigned char smem_raw[1 << 16];
"""
MAIN = r"""
int main(int argc, char** argv) {
  const int n = atoi(argv[2]), use_smem = atoi(argv[3]);
  lag = atoi(argv[4]);
  std::vector<double> u((size_t)n * n), x(n);
  FILE* f = fopen(argv[1], "rb");
  if (!f || fread(u.data(), 8, u.size(), f) != u.size() || fread(x.data(), 8, n, f) != (size_t)n) return 1;
  fclose(f);
  run_warp([&](int) { back_exact_kernel<double>(u.data(), n, x.data(), 1, n, use_smem); });
  for (double v : x) printf("%a\n", v);
}
"""


def back_substitution(u, x):
    """lair's order: x[i] -= u[i][k] x[k] for increasing k, then the division."""
    x = x.copy()
    n = len(x)
    for i in range(n - 1, -1, -1):
        for k in range(i + 1, n):
            x[i] -= u[i, k] * x[k]
        x[i] /= u[i, i]
    return x


@pytest.mark.parametrize("lag", [0, 1, 31, 32])
@pytest.mark.parametrize("use_smem", [1, 0])
@pytest.mark.parametrize("n", [1, 33, 64, 65, 131])
def test_order_holds_when_lanes_drift(tmp_path, n, use_smem, lag):
    rng = np.random.default_rng(n)
    u = rng.uniform(-1, 1, (n, n)) + 3 * np.eye(n)
    x = rng.uniform(-1, 1, n)
    data = tmp_path / "in"
    data.write_bytes(u.tobytes() + x.tobytes())
    kernel = "template <typename T>\n" + warp.extract("getrs.cu", "__global__ void back_exact_kernel").replace(
        "extern __shared__ __align__(16) unsigned char smem_raw[];", "")
    out = warp.run(BODY + kernel, MAIN, [data, n, use_smem, lag])
    got = np.array([float.fromhex(v) for v in out.split()])
    assert np.array_equal(got, back_substitution(u, x))
