// Digit slices of FP64 rows and columns for the tensor-core update (ozaki.cu).
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

namespace luhot {

constexpr int kOzSlices = 7;
constexpr int kOzGroups = 7;   // G = p + q = 0 .. 6
constexpr int kOzK = 64;       // K of one update (one 128-byte box row of FP16)
constexpr int kOzNonFinite = 1 << 20;  // exponent of a row / column that holds Inf or NaN
constexpr int kOzZero = -(1 << 20);    // exponent of a zero element

// The e of frexp(x) (|x| < 2^e, |x| >= 2^(e-1)) from the bits; kOzZero for
// zeros, kOzNonFinite for Inf and NaN.
__device__ __forceinline__ int oz_exponent(double x) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const int E = (int)((u >> 52) & 0x7ff);
  const unsigned long long m = u & 0xFFFFFFFFFFFFFull;
  if (E == 0x7ff) return kOzNonFinite;
  if (E != 0) return E - 1022;
  if (m == 0) return kOzZero;
  return (64 - __clzll((long long)m)) - 1074;
}

// Seven balanced base-256 digits of round(|x| 2^(56-e)), signed like x, most
// significant first; |x| < 2^e.  Integer arithmetic only.
__device__ __forceinline__ void oz_digits(double x, int e, int (&d)[kOzSlices]) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const int E = (int)((u >> 52) & 0x7ff);
  unsigned long long m = u & 0xFFFFFFFFFFFFFull;
  int ex = -1074;
  if (E != 0) {
    m |= 1ull << 52;
    ex = E - 1075;
  }
  // |x| = m 2^ex < 2^e, so m 2^(ex - e + 56) < 2^56.
  const int sh = ex - e + 56;
  unsigned long long N;
  if (m == 0 || sh <= -64)
    N = 0;
  else if (sh >= 0)
    N = m << sh;
  else
    N = (m + (1ull << (-sh - 1))) >> (-sh);  // round half up; m < 2^53, so no overflow
  int carry = 0;
#pragma unroll
  for (int p = kOzSlices - 1; p >= 1; --p) {
    const int v = (int)(N & 255u) + carry;
    N >>= 8;
    carry = v >= 128 ? 1 : 0;
    d[p] = v - (carry << 8);
  }
  d[0] = (int)N + carry;  // N < 2^8 here: d_0 <= 256
  if (u >> 63) {
#pragma unroll
    for (int p = 0; p < kOzSlices; ++p) d[p] = -d[p];
  }
}

// One warp writes the digits of a 64-element row (x0 = element lane, x1 =
// element lane + 32) with the warp-reduced exponent e into slice rows
// dst[p * slice + 0..63].
__device__ __forceinline__ void oz_emit_row(double x0, double x1, int e, __half* __restrict__ dst, int64_t slice,
                                            int lane) {
  int d0[kOzSlices], d1[kOzSlices];
  if (e == kOzZero || e >= kOzNonFinite) {
#pragma unroll
    for (int p = 0; p < kOzSlices; ++p) d0[p] = d1[p] = 0;
  } else {
    oz_digits(x0, e, d0);
    oz_digits(x1, e, d1);
  }
#pragma unroll
  for (int p = 0; p < kOzSlices; ++p) {
    dst[p * slice + lane] = __int2half_rn(d0[p]);
    dst[p * slice + lane + 32] = __int2half_rn(d1[p]);
  }
}

__device__ __forceinline__ int oz_warp_max(int v) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, off));
  return v;
}

}  // namespace luhot
