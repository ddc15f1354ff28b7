// Exchange between the CTAs of one thread-block cluster through shared memory:
// stores that count their bytes on the receiver's mbarrier, bounded waits.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <set>
#include <utility>

#include "common.cuh"

namespace luhot {

__device__ __forceinline__ unsigned cl_smem(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned cl_peer(unsigned addr, int cta) {
  unsigned d;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(d) : "r"(addr), "r"(cta));
  return d;
}
// 16 bytes into a peer's shared memory, counted on the peer's mbarrier.
__device__ __forceinline__ void cl_push16(unsigned dst, unsigned bar, unsigned long long a, unsigned long long b) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
               "l"(a), "l"(b), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cl_push8(unsigned dst, unsigned bar, unsigned long long a) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(dst), "l"(a),
               "r"(bar)
               : "memory");
}
__device__ __forceinline__ void cl_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ unsigned cl_try(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, "
      "0, p;\n}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done;
}
// Bounded wait of a whole warp; false (for all lanes) once it gave up.  The loop is
// kept out of line: a column's chain runs through its code once a column on one
// warp, so that the length of that code is itself part of the chain.  The lanes read
// clocks of their own: whichever passes the limit first, lane 0 records it.
static __device__ __noinline__ bool cl_wait_long(unsigned bar, unsigned parity, DeviceStatus* st, int step) {
  unsigned long long t0 = 0;
  for (unsigned spins = 1;; ++spins) {
    if (__all_sync(0xffffffffu, cl_try(bar, parity) != 0)) return true;
    if ((spins & 15u) == 0) {
      const unsigned long long now = global_timer_ns();
      if (t0 == 0) t0 = now;
      const bool late = __any_sync(0xffffffffu, now - t0 > st->timeout_ns);
      if (late || __any_sync(0xffffffffu, ld_relaxed_i32(&st->abort) != 0)) {
        if (late && (threadIdx.x & 31) == 0) {
          atomicCAS(&st->error, kDevOk, kDevBarrierTimeout);
          atomicExch(&st->timeout_where, (unsigned long long)step);
          atomicExch(&st->abort, 1);
        }
        return false;
      }
    }
  }
}
__device__ __forceinline__ bool cl_wait(unsigned bar, unsigned parity, DeviceStatus* st, int step) {
  if (__all_sync(0xffffffffu, cl_try(bar, parity) != 0)) return true;
  return cl_wait_long(bar, parity, st, step);
}
__device__ __forceinline__ void cl_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// For a CTA that gave up a wait, behind the last cl_sync: pushes to it may still be
// under way, which have to land before it leaves.
static __device__ __noinline__ void cl_drain() {
  const unsigned long long t0 = global_timer_ns();
  while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
}

// Lets `kernel` launch with clusters of more than 8 CTAs; once per kernel and
// device, like allow_max_dynamic_smem.
inline cudaError_t allow_wide_clusters(const void* kernel) {
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> allowed;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  if (allowed.count({kernel, dev})) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) allowed.insert({kernel, dev});
  return e;
}

inline cudaLaunchConfig_t cl_config(int P, int threads, size_t smem, cudaStream_t stream, cudaLaunchAttribute* attr) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(P);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = P;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

}  // namespace luhot
