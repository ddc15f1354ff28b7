// Shared by the two panel kernels: the elimination update, the pivot search
// keys and the kernel arguments.
#pragma once

#include <climits>
#include <cstdint>

#include "common.cuh"
#include "luhot_internal.h"

namespace luhot {

// ---------------------------------------------------------------------------
// Arithmetic of one elimination update: c - l*u.
// ---------------------------------------------------------------------------
template <bool kExact>
__device__ __forceinline__ double upd(double c, double l, double u) {
  if (kExact) return __dsub_rn(c, __dmul_rn(l, u));
  return fma(-l, u, c);
}
template <bool kExact>
__device__ __forceinline__ float upd(float c, float l, float u) {
  if (kExact) return __fsub_rn(c, __fmul_rn(l, u));
  return fmaf(-l, u, c);
}
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }

template <typename T>
struct PanelArgs {
  T* a;
  int64_t lda;
  int m;          // rows of the whole matrix
  int k0;         // first row/column of the panel
  int w;          // panel width == elimination steps in this panel
  int rows_per;   // panel rows owned by each CTA
  int lds;        // shared-memory row stride (elements)
  int* piv;       // device pivots (global row index per step)
  unsigned long long* heads;  // [2][kMaxPanelCtas][kPanelHeaderWords] exchange headers
  unsigned long long* slots;  // [2][kMaxPanelCtas][kPanelSlotWords] exchange words
  int* moves;                 // (destination, source) rows of the panel's rows that moved
  int* move_count;            // zeroed before the launch
  DeviceStatus* st;
};

// Pivot search keys.  lair's iamax (src/blas/iamax.rs:6-21) takes the first
// index of the largest |x| with a strict `>`: larger value wins, equal values
// keep the smaller row, NaN never wins, and an all-zero/NaN column means a
// singular step.  For |x| >= 0 the IEEE bit pattern orders like the value,
// so the search compares integers (on the integer pipe; FP64 compares are
// slow on this part): key = bits of |x|, or 0 for NaN.  (key, row) ordered by
// key descending then row ascending is a total order, so any reduction tree
// gives the same answer; key 0 means "no positive entry".
template <typename T>
struct PivotKey;
template <>
struct PivotKey<float> {
  using K = unsigned int;
  __device__ static K of(float x) {
    const unsigned int b = __float_as_uint(x) & 0x7fffffffu;
    return b > 0x7f800000u ? 0u : b;
  }
  __device__ static K shfl(K k, int src) { return __shfl_sync(0xffffffffu, k, src); }
  __device__ static float value(K raw) { return __uint_as_float(raw); }
};
template <>
struct PivotKey<double> {
  using K = unsigned long long;
  __device__ static K of(double x) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
    return b > 0x7ff0000000000000ull ? 0ull : b;
  }
  __device__ static K shfl(K k, int src) { return __shfl_sync(0xffffffffu, k, src); }
  __device__ static double value(K raw) { return __longlong_as_double((long long)raw); }
};

template <typename K>
__device__ __forceinline__ void key_combine(K& k, int& i, int& s, K k2, int i2, int s2) {
  if (k2 > k || (k2 == k && i2 < i)) {
    k = k2;
    i = i2;
    s = s2;
  }
}
// Warp-wide reduction of (key, id, slot) on the integer reduce unit
// (redux.sync): the largest key, then the smallest id among the lanes that
// hold it; the slot comes from that lane, whose index is returned.  The
// order is total, so this is the answer of any key_combine tree.
__device__ __forceinline__ int key_reduce_redux(unsigned int& k, int& i, int& s) {
  const unsigned int m = __reduce_max_sync(0xffffffffu, k);
  const int mi = __reduce_min_sync(0xffffffffu, k == m ? i : INT_MAX);
  const int src = __ffs(__ballot_sync(0xffffffffu, k == m && i == mi)) - 1;
  s = __shfl_sync(0xffffffffu, s, src);
  k = m;
  i = mi;
  return src;
}
__device__ __forceinline__ int key_reduce_redux(unsigned long long& k, int& i, int& s) {
  const unsigned int hi = (unsigned int)(k >> 32);
  const unsigned int mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned int ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned int)k : 0u);
  const unsigned long long m = ((unsigned long long)mh << 32) | ml;
  const int mi = __reduce_min_sync(0xffffffffu, k == m ? i : INT_MAX);
  const int src = __ffs(__ballot_sync(0xffffffffu, k == m && i == mi)) - 1;
  s = __shfl_sync(0xffffffffu, s, src);
  k = m;
  i = mi;
  return src;
}

// Lane of a warp that holds the largest key (the smallest id among equal
// keys).  One redux and one vote unless (the high words of) keys tie.
__device__ __forceinline__ int warp_best(unsigned int k, int id) {
  const unsigned m = __reduce_max_sync(0xffffffffu, k);
  unsigned mask = __ballot_sync(0xffffffffu, k == m);
  if (mask & (mask - 1u)) {
    const int mi = __reduce_min_sync(0xffffffffu, k == m ? id : INT_MAX);
    mask = __ballot_sync(0xffffffffu, k == m && id == mi);
  }
  return __ffs(mask) - 1;
}
__device__ __forceinline__ int warp_best(unsigned long long k, int id) {
  const unsigned hi = (unsigned)(k >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  unsigned mask = __ballot_sync(0xffffffffu, hi == mh);
  if (mask & (mask - 1u)) {
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)k : 0u);
    const unsigned long long m = ((unsigned long long)mh << 32) | ml;
    const int mi = __reduce_min_sync(0xffffffffu, k == m ? id : INT_MAX);
    mask = __ballot_sync(0xffffffffu, k == m && id == mi);
  }
  return __ffs(mask) - 1;
}

// Cooperative form over one thread-block cluster (panel_cluster.cu): whether
// it takes a panel of `rows` rows and width w, and its launch.
template <typename T, bool kExact>
bool panel_cluster_fits(luhot_ctx* ctx, int rows, int w);
template <typename T, bool kExact>
int launch_panel_cluster(luhot_ctx* ctx, T* a, int64_t lda, int m, int k0, int w, int* piv, int* moves,
                         cudaStream_t stream);

}  // namespace luhot
