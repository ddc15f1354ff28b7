// Between a panel and its trailing update, in one launch: the panel's row
// interchanges left and right of it, U12 <- L11^-1 A12, and (fast FP64) the
// digit slices of L21 and U12 for the tensor-core update (ozaki.cu).
//
// CTAs take one of three parts:
//   right   groups of 8 (FP64) or 16 (FP32) columns: a group's moved rows and its
//           rows of the panel are gathered (every load before any store), then
//           solved: a warp has two columns, 16 lanes each, a lane the rows
//           lane + 16 r; step k takes x_k by shuffle and subtracts l_ik x_k from
//           the rows below, so an element gets its updates one at a time in
//           increasing k (lair's order, src/lapack/getrf.rs:76-89: exact mode's
//           bits).  With a split, the 64 solved values of a column are turned
//           into digits where they are.
//   left    32 columns: the interchanges alone.
//   split   a warp per row of L21.
// FP64: a warp's FP64 instruction takes 64 cycles of its SM quarter's pipe
// whatever its lanes do, so the columns are spread over all quarters of the
// chip (two columns and 2.5 of 4 row registers a step keep 80 % of the lanes
// of those instructions busy) instead of a column per thread: a 64-row solve of
// 936 columns took 15 + 3 + 9 + 28 us as diagonal inverse, two splits and a slice
// product (and 84 us as one thread per column), the interchanges 7 and the
// update's own splits 4 + 9; this launch does all of it.
// Few columns (a CTA a group, one pass): memory latency and the 64-step chain bound
// it, so the list of moves, its count and 16 elements of L11 a thread are in
// flight at once (2500-column FP32 factorization: 14 -> 11 us a launch; 936 FP64
// columns 18.5 -> 17.4).
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "luhot_internal.h"
#include "ozaki_split.cuh"
#include "panel.cuh"
#include "swap_solve.cuh"

namespace luhot {

template <typename T>
struct SwapSolveArgs {
  T* a;
  int64_t lda;
  const int* moves;       // (destination, source) rows, or nullptr
  const int* move_count;
  int k0, w;
  int cl0, cl1, cr0, cr1;
  int right_ctas, left_ctas;
  SplitOut split;
};

template <typename T>
__host__ __device__ constexpr int ss_cols() {
  return sizeof(T) == 8 ? 8 : 16;
}
template <typename T>
__host__ __device__ constexpr int ss_threads() {
  return 16 * ss_cols<T>();  // a warp per two columns
}
constexpr int kSsLeftCols = 32;
static_assert(64 * 64 % (16 * ss_threads<float>()) == 0 && 64 * 64 % (16 * ss_threads<double>()) == 0,
              "L11 is staged in whole batches");

template <typename T, bool kExact, int W>
__global__ void __launch_bounds__(ss_threads<T>()) swap_solve_kernel(SwapSolveArgs<T> p) {
  constexpr int kCols = ss_cols<T>(), kTh = ss_threads<T>(), kWp = W + 1, kXp = kCols + 1;
  constexpr int kR = W / 16;  // rows of a lane, and row passes of the CTA
  constexpr unsigned kFull = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int mv[4 * kMaxPanelWidth];      // the (destination, source) pairs
  __shared__ int srcrow[W];                   // source of each of the panel's rows
  __shared__ int below[2 * kMaxPanelWidth];   // pairs whose destination lies below the panel's rows
  __shared__ int s_below;
  const int tid = threadIdx.x, lane = tid & 31;
  const int bid = blockIdx.x;

  if (bid >= p.right_ctas + p.left_ctas) {
    if constexpr (std::is_same<T, double>::value) {
      // Rows of L21: digits of a row's w elements (zero beyond w).
      const SplitOut& s = p.split;
      const int warps = (gridDim.x - p.right_ctas - p.left_ctas) * (kTh / 32);
      for (int i = (bid - p.right_ctas - p.left_ctas) * (kTh / 32) + (tid >> 5); i < s.M; i += warps) {
        const double* row = p.a + (int64_t)(s.r1 + i) * p.lda + p.k0;
        const double x0 = lane < p.w ? row[lane] : 0.0;
        const double x1 = lane + 32 < p.w ? row[lane + 32] : 0.0;
        const int e = oz_warp_max(max(oz_exponent(x0), oz_exponent(x1)));
        oz_emit_row(x0, x1, e, s.as + (int64_t)i * kOzK, (int64_t)s.M * kOzK, lane);
        if (lane == 0) s.ea[i] = e == kOzZero ? 0 : e;
      }
    }
    return;
  }

  // The list is read whole, beside its count: one trip to memory instead of two.
  const int capacity = p.moves ? 2 * min(p.w, kMaxPanelWidth) : 0;
  for (int i = tid; i < 2 * capacity; i += kTh) mv[i] = p.moves[i];
  const int count = p.moves ? min(*p.move_count, capacity) : 0;

  if (bid >= p.right_ctas) {
    // Interchanges alone: 32 columns, every load of a group before its stores.
    __syncthreads();
    T* vals = reinterpret_cast<T*>(smem_raw);  // [2w][32]
    const int tx = lane, ty = tid >> 5;
    constexpr int kTy = kTh / 32, kB = 8;
    const int groups = (p.cl1 - p.cl0 + kSsLeftCols - 1) / kSsLeftCols;
    for (int g = bid - p.right_ctas; g < groups; g += p.left_ctas) {
      const int c = p.cl0 + g * kSsLeftCols + tx;
      const bool on = c < p.cl1;
      for (int e0 = ty; e0 < count; e0 += kTy * kB) {
        T v[kB];
#pragma unroll
        for (int q = 0; q < kB; ++q) {
          const int e = e0 + q * kTy;
          v[q] = (on && e < count) ? p.a[(int64_t)mv[2 * e + 1] * p.lda + c] : T(0);
        }
#pragma unroll
        for (int q = 0; q < kB; ++q) {
          const int e = e0 + q * kTy;
          if (e < count) vals[e * kSsLeftCols + tx] = v[q];
        }
      }
      __syncthreads();
      for (int e = ty; e < count; e += kTy)
        if (on) p.a[(int64_t)mv[2 * e] * p.lda + c] = vals[e * kSsLeftCols + tx];
      __syncthreads();
    }
    return;
  }

  T* Lt = reinterpret_cast<T*>(smem_raw);  // [W][W + 1]: Lt[k][i] = L11(i, k) for i > k, else 0
  T* X = Lt + W * kWp;                     // [W][kCols + 1]
  __half* D = reinterpret_cast<__half*>(X + W * kXp);  // [7][kCols][64] (with a split)
  constexpr int kLoads = 16;  // in flight
  for (int base = tid; base < W * W; base += kLoads * kTh) {
    T l[kLoads];
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int idx = base + q * kTh, i = idx / W, k = idx - i * W;
      l[q] = (i < p.w && k < i) ? p.a[(int64_t)(p.k0 + i) * p.lda + p.k0 + k] : T(0);
    }
#pragma unroll
    for (int q = 0; q < kLoads; ++q) {
      const int idx = base + q * kTh, i = idx / W, k = idx - i * W;
      Lt[k * kWp + i] = l[q];
    }
  }
  if (tid < W) srcrow[tid] = p.k0 + tid;
  if (tid == 0) s_below = 0;
  __syncthreads();
  for (int e = tid; e < count; e += kTh) {
    const int dst = mv[2 * e];
    if (dst < p.k0 + p.w) {
      srcrow[dst - p.k0] = mv[2 * e + 1];
    } else {
      const int q = atomicAdd(&s_below, 1);
      if (q < kMaxPanelWidth) {
        below[2 * q] = dst;
        below[2 * q + 1] = mv[2 * e + 1];
      }
    }
  }
  __syncthreads();
  const int nbelow = min(s_below, W);  // a row moved out of the panel's rows for every row moved in
  const int tx = tid % kCols, ty = tid / kCols;  // ty: 0 .. 15
  const int half = lane >> 4, g16 = lane & 15;
  const int col = 2 * (tid >> 5) + half;
  const int groups = (p.cr1 - p.cr0 + kCols - 1) / kCols;
  for (int g = bid; g < groups; g += p.right_ctas) {
    const int cb = p.cr0 + g * kCols;
    const int c = cb + tx;
    const bool on = c < p.cr1;
    T v[kR], t[kR];
#pragma unroll
    for (int q = 0; q < kR; ++q) {
      const int e = ty + 16 * q;
      v[q] = (on && e < nbelow) ? p.a[(int64_t)below[2 * e + 1] * p.lda + c] : T(0);
      t[q] = (on && e < p.w) ? p.a[(int64_t)srcrow[e] * p.lda + c] : T(0);
    }
#pragma unroll
    for (int q = 0; q < kR; ++q) X[(ty + 16 * q) * kXp + tx] = t[q];
    __syncthreads();  // every load of this group's columns is done
#pragma unroll
    for (int q = 0; q < kR; ++q) {
      const int e = ty + 16 * q;
      if (on && e < nbelow) p.a[(int64_t)below[2 * e] * p.lda + c] = v[q];
    }
    T x[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) x[r] = X[(g16 + 16 * r) * kXp + col];
#pragma unroll
    for (int kb = 0; kb < kR; ++kb) {
      const int steps = min(16, p.w - kb * 16);
      for (int kk = 0; kk < steps; ++kk) {
        const T xk = __shfl_sync(kFull, x[kb], (lane & 16) | kk);
        const T* l = Lt + (kb * 16 + kk) * kWp + g16;
        if (kk < 15 && g16 > kk) x[kb] = upd<kExact>(x[kb], l[16 * kb], xk);
#pragma unroll
        for (int r = kb + 1; r < kR; ++r) x[r] = upd<kExact>(x[r], l[16 * r], xk);
      }
    }
#pragma unroll
    for (int r = 0; r < kR; ++r) X[(g16 + 16 * r) * kXp + col] = x[r];
    if constexpr (std::is_same<T, double>::value && W == kOzK && !kExact) {
      if (p.split.bs) {
        int e = kOzZero;
#pragma unroll
        for (int r = 0; r < kR; ++r) e = max(e, oz_exponent(x[r]));
#pragma unroll
        for (int off = 8; off > 0; off >>= 1) e = max(e, __shfl_xor_sync(kFull, e, off));
        if (g16 == 0 && cb + col < p.cr1) p.split.eb[cb + col - p.cr0] = e == kOzZero ? 0 : e;
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          int d[kOzSlices];
          if (e == kOzZero || e >= kOzNonFinite) {
#pragma unroll
            for (int q = 0; q < kOzSlices; ++q) d[q] = 0;
          } else {
            oz_digits(x[r], e, d);
          }
#pragma unroll
          for (int q = 0; q < kOzSlices; ++q) D[(q * kCols + col) * kOzK + g16 + 16 * r] = __int2half_rn(d[q]);
        }
      }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kR; ++q) {
      const int r = ty + 16 * q;
      if (on && r < p.w) p.a[(int64_t)(p.k0 + r) * p.lda + c] = X[r * kXp + tx];
    }
    if constexpr (std::is_same<T, double>::value && W == kOzK && !kExact) {
      if (p.split.bs) {
        // Slice rows of 128 bytes, 16 bytes a thread.
        const int64_t slice = (int64_t)(p.cr1 - p.cr0) * kOzK;
        for (int idx = tid; idx < kOzSlices * kCols * 8; idx += kTh) {
          const int q = idx / (kCols * 8), rest = idx - q * (kCols * 8), j = rest >> 3, part = rest & 7;
          if (cb + j < p.cr1)
            *reinterpret_cast<uint4*>(p.split.bs + q * slice + (int64_t)(cb + j - p.cr0) * kOzK + part * 8) =
                *reinterpret_cast<const uint4*>(D + (q * kCols + j) * kOzK + part * 8);
        }
      }
    }
    __syncthreads();
  }
}

template <typename T, bool kExact>
int launch_swap_solve(luhot_ctx* ctx, T* a, int64_t lda, const int* moves, int k0, int w, int cl0, int cl1, int cr0,
                      int cr1, const SplitOut* split, cudaStream_t stream) {
  const int nright = std::max(0, cr1 - cr0), nleft = moves ? std::max(0, cl1 - cl0) : 0;
  if (nright + nleft == 0) return LUHOT_OK;
  const int W = w <= 64 ? 64 : 128;
  constexpr int kCols = ss_cols<T>(), kTh = ss_threads<T>();
  SwapSolveArgs<T> args{};
  args.a = a;
  args.lda = lda;
  args.moves = moves;
  args.move_count = moves ? moves + 4 * kMaxPanelWidth : nullptr;
  args.k0 = k0;
  args.w = w;
  args.cl0 = cl0;
  args.cl1 = cl0 + nleft;
  args.cr0 = cr0;
  args.cr1 = cr0 + nright;
  if (split) args.split = *split;
  // A CTA stages L11 once and takes several groups where there are more than
  // four a multiprocessor (the CTAs that fit with 64 rows of FP64).
  args.right_ctas = std::min((nright + kCols - 1) / kCols, 4 * ctx->num_sms);
  args.left_ctas = std::min((nleft + kSsLeftCols - 1) / kSsLeftCols, 4 * ctx->num_sms);
  const int split_ctas = split ? std::min((split->M + 2 * (kTh / 32) - 1) / (2 * (kTh / 32)), 4 * ctx->num_sms) : 0;
  const size_t right = ((size_t)W * (W + 1) + (size_t)W * (kCols + 1)) * sizeof(T) +
                       (split ? (size_t)kOzSlices * kCols * kOzK * sizeof(__half) : 0);
  const size_t left = nleft ? (size_t)2 * w * kSsLeftCols * sizeof(T) : 0;
  const size_t smem = std::max(right, left);
  prof_begin(ctx, kProfTrsm);
  if (W == 64) {
    LUHOT_CUDA_TRY(ctx, allow_max_dynamic_smem(swap_solve_kernel<T, kExact, 64>));
    swap_solve_kernel<T, kExact, 64>
        <<<args.right_ctas + args.left_ctas + split_ctas, kTh, smem, stream>>>(args);
  } else {
    LUHOT_CUDA_TRY(ctx, allow_max_dynamic_smem(swap_solve_kernel<T, kExact, 128>));
    swap_solve_kernel<T, kExact, 128>
        <<<args.right_ctas + args.left_ctas + split_ctas, kTh, smem, stream>>>(args);
  }
  prof_end(ctx, kProfTrsm, (double)w * (w - 1) * nright,
           ((double)w * w + 2.0 * w * nright + 4.0 * w * (nleft + nright)) * sizeof(T) +
               (split ? (split->M * (8.0 * w + 14.0 * kOzK) + 14.0 * kOzK * nright) : 0.0));
  LUHOT_CUDA_TRY(ctx, cudaGetLastError());
  return LUHOT_OK;
}

template int launch_swap_solve<double, false>(luhot_ctx*, double*, int64_t, const int*, int, int, int, int, int, int,
                                              const SplitOut*, cudaStream_t);
template int launch_swap_solve<double, true>(luhot_ctx*, double*, int64_t, const int*, int, int, int, int, int, int,
                                             const SplitOut*, cudaStream_t);
template int launch_swap_solve<float, false>(luhot_ctx*, float*, int64_t, const int*, int, int, int, int, int, int,
                                             const SplitOut*, cudaStream_t);
template int launch_swap_solve<float, true>(luhot_ctx*, float*, int64_t, const int*, int, int, int, int, int, int,
                                            const SplitOut*, cudaStream_t);

}  // namespace luhot
