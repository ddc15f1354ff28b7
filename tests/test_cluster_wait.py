"""The bounded cluster wait (cl_wait_long, lair_gb300/csrc/cluster.cuh) on an
emulated warp: a wait that gives up has recorded the error, whichever lane's
clock passed the limit first, and one that another wait's abort ends has not."""
import pytest

import warp_emulation as warp

MAIN = r"""
int main(int argc, char** argv) {
  const int first = atoi(argv[1]);  // the lane whose clock passes the limit; -1: none, the abort is set
  st.abort = first < 0;
  ahead = first;
  std::atomic<int> gave_up{0};
  run_warp([&](int) { gave_up += !cl_wait_long(0, 0, &st, 7); });
  printf("%d %d %d %llu", gave_up.load(), st.error, st.abort, st.timeout_where);
}
"""
BODY = r"""
enum { kDevOk = 0, kDevBarrierTimeout = 1 };
struct DeviceStatus { int error = 0, abort = 0; unsigned long long timeout_where = 0, timeout_ns = 1000; } st;
static int ahead;
static unsigned long long global_timer_ns() {
  static thread_local int reads = 0;
  return threadIdx.x == ahead && reads++ > 0 ? 5000 : 100;  // the other clocks stand still
}
static unsigned cl_try(unsigned, unsigned) { return 0; }  // nothing ever arrives
static int ld_relaxed_i32(const int* p) { return __atomic_load_n(p, __ATOMIC_RELAXED); }
"""


@pytest.mark.parametrize("first", [0, 1, 31, -1])
def test_a_wait_that_gives_up_records_it(first):
    body = BODY + warp.extract("cluster.cuh", "static __device__ __noinline__ bool cl_wait_long")
    gave_up, error, abort, where = map(int, warp.run(body, MAIN, [first]).split())
    assert gave_up == 32
    assert (error, abort, where) == ((1, 1, 7) if first >= 0 else (0, 1, 0))
