// Batched LU + solve of thousands of small uneven systems in one graph launch.
//
// Packed layout: system i is an n_i x n_i row-major matrix at element offset
// a_off[i] = sum_{j<i} n_j^2 and a right-hand side (overwritten by x) and
// int32 pivots at b_off[i] = sum_{j<i} n_j.  info[i] = last all-zero pivot
// step of system i (lair's Option<usize>) or -1.
//
// One CTA per system at a time; the CTAs of a size class draw its systems from
// an atomic counter, largest first, and the classes run side by side (branches
// of the graph), so each has the shared memory, threads and registers it needs:
// a class is a range of n whose matrices fit so many to an SM, and the systems
// that do not fit (or that the autotuner moved) use a scratch matrix per CTA in
// global memory, which stays in L2.
//
// Per system the matrix (and the right-hand side as column n) is copied in and
// factored in panels of NB columns:
//   panel   one warp, the active rows in registers (NI rows x NB columns a lane),
//           no block barrier inside: pivot by one redux and a vote, pivot row by
//           shuffle, rank-1 updates in registers.  Rows never move: a row's logical
//           index is relabelled, and the copy-out writes rows in logical order.
//   U12     a thread per column (the right-hand side among them, so the forward
//           substitution needs no pass of its own);
//   update  FP32: 8 rows x 4 columns a lane, vector loads of both operands; FP64,
//           bound by its pipe, where a warp instruction takes 64 cycles however
//           few lanes it has: (row, column) pairs flattened over the lanes.
// The back substitution is one warp's column sweep with the solution in
// registers.  Elements get their updates one at a time in elimination order
// with lair's roundings in exact mode (src/lapack/getrf.rs:76-89, getrs.rs:24-36),
// so each system's LU, pivots and x are bit-identical to lair's there.
//
// 10 000 FP32 systems of n ~ U{8..256} 15.0 -> 8.0 ms, 1500 FP64 7.3 -> 6.0 ms,
// against one 256-thread CTA per system with a block-wide search and four barriers
// per column.  FP64 is within 1.5 of its pipe's 4.1 ms.  FP32: the panel warps' steps (about
// 1100 cycles each, instruction fetches among them) are some 3 of the 8 ms; updates,
// U12 and copies run in turn with them in the same CTA, and systems of 164 to 235 rows
// have an SM to themselves.
#include <algorithm>
#include <climits>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "luhot_internal.h"
#include "panel.cuh"

namespace luhot {

constexpr int kBatchMaxN = 256;
constexpr int kBuckets = 9;         // n in (0,16], (16,32], (32,64], (64,96], ..., (224,256]
constexpr size_t kBatchSmem = 222 * 1024;
constexpr int kScratchLd = 260;     // row stride of a scratch matrix (256 + the right-hand side, whole 16 bytes)
constexpr size_t kScratchElems = (size_t)kBatchMaxN * kScratchLd;

__host__ __device__ inline int batch_bucket(int n) {
  if (n <= 16) return 0;
  if (n <= 32) return 1;
  if (n <= 64) return 2;
  return min(kBuckets - 1, 3 + (n - 65) / 32);
}

// Panel width: a lane's NI x NB panel values are registers; FP32 panels of more
// than 128 rows are kept to 64 registers so that 16 warps share an SM.
template <typename T>
__host__ __device__ constexpr int batch_nb(int ni) {
  return sizeof(T) == 8 || ni == 8 ? 8 : 16;
}
// Row stride in shared memory (n columns and the right-hand side): FP32 whole
// 16-byte pieces, an odd number of them (conflict-free panel loads); FP64 odd.
template <typename T>
__host__ __device__ inline int batch_ld(int n) {
  if (sizeof(T) == 8) return (n + 1) | 1;
  const int q = (n + 4) / 4;
  return 4 * (q | 1);
}

struct BatchMeta {
  const int* sizes;
  const int64_t* aoff;
  const int64_t* boff;
  const int* order;  // the class's systems, largest first
  int count;
};

// A22 -= L21 U12 for the active rows act[0, na) and the columns [c1, c1 + nc),
// panel columns [k0, k0 + w); steps in `mask` made no update.  FP32, kCV columns
// a lane: 4 (16 lanes, two groups of 8 rows a warp) or 1.
template <bool kExact, int kNB, int kCV, bool kMasked>
__device__ __forceinline__ void batch_update_f32(float* S, int ld, const int* act, int na, const int* prow, int k0,
                                                 int c1, int nc, unsigned mask) {
  constexpr int kRows = 8, kLanes = kCV == 4 ? 16 : 32, kGroups = 32 / kLanes;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int cgs = (nc + kLanes * kCV - 1) / (kLanes * kCV);
  const int rgs = (na + kRows * kGroups - 1) / (kRows * kGroups);
  for (int unit = warp; unit < rgs * cgs; unit += warps) {
    const int rg = unit / cgs, cg = unit - rg * cgs;
    const int cc = (cg * kLanes + lane % kLanes) * kCV;
    const bool on = cc < nc;
    const int c = c1 + (on ? cc : 0);
    const int q0 = (rg * kGroups + lane / kLanes) * kRows;
    int row[kRows];
    float acc[kRows][kCV];
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      row[r] = act[min(q0 + r, na - 1)] * ld;
      if constexpr (kCV == 4) {
        const float4 v = *reinterpret_cast<const float4*>(S + row[r] + c);
        acc[r][0] = v.x, acc[r][1] = v.y, acc[r][2] = v.z, acc[r][3] = v.w;
      } else {
        acc[r][0] = S[row[r] + c];
      }
    }
    // w is the whole panel width here: after a narrower (last) panel no row is left.
#pragma unroll
    for (int kb = 0; kb < kNB; kb += 4) {
      float4 l[kRows];
#pragma unroll
      for (int r = 0; r < kRows; ++r) l[r] = *reinterpret_cast<const float4*>(S + row[r] + k0 + kb);
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        if (kMasked && (mask >> (kb + kk)) & 1u) continue;
        const float* up = S + prow[k0 + kb + kk] * ld + c;
        float u[kCV];
        if constexpr (kCV == 4) {
          const float4 v = *reinterpret_cast<const float4*>(up);
          u[0] = v.x, u[1] = v.y, u[2] = v.z, u[3] = v.w;
        } else {
          u[0] = *up;
        }
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
          const float lv = kk == 0 ? l[r].x : kk == 1 ? l[r].y : kk == 2 ? l[r].z : l[r].w;
#pragma unroll
          for (int e = 0; e < kCV; ++e) acc[r][e] = upd<kExact>(acc[r][e], lv, u[e]);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      if (!on || q0 + r >= na) continue;
      if constexpr (kCV == 4)
        *reinterpret_cast<float4*>(S + row[r] + c) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
      else
        S[row[r] + c] = acc[r][0];
    }
  }
}
template <bool kExact, int kNB>
__device__ __forceinline__ void batch_update(float* S, int ld, const int* act, int na, const int* prow, int k0, int,
                                             int c1, int nc, unsigned mask) {
  if (mask)
    batch_update_f32<kExact, kNB, 1, true>(S, ld, act, na, prow, k0, c1, nc, mask);
  else if (nc > 32)
    batch_update_f32<kExact, kNB, 4, false>(S, ld, act, na, prow, k0, c1, nc, mask);
  else
    batch_update_f32<kExact, kNB, 1, false>(S, ld, act, na, prow, k0, c1, nc, mask);
}
template <bool kExact, int kNB>
__device__ __forceinline__ void batch_update(double* S, int ld, const int* act, int na, const int* prow, int k0,
                                             int w, int c1, int nc, unsigned mask) {
  constexpr int kE = 4;  // elements of a lane in flight
  const int total = na * nc, step = blockDim.x * kE;
  for (int base = threadIdx.x; base < total; base += step) {
    int crow[kE], cc[kE];
    double acc[kE];
#pragma unroll
    for (int e = 0; e < kE; ++e) {
      const int idx = min(base + e * (int)blockDim.x, total - 1);
      const int q = idx / nc;
      cc[e] = c1 + idx - q * nc;
      crow[e] = act[q] * ld;
      acc[e] = S[crow[e] + cc[e]];
    }
    for (int k = 0; k < w; ++k) {
      if ((mask >> k) & 1u) continue;
      const int ur = prow[k0 + k] * ld;
#pragma unroll
      for (int e = 0; e < kE; ++e) acc[e] = upd<kExact>(acc[e], S[crow[e] + k0 + k], S[ur + cc[e]]);
    }
#pragma unroll
    for (int e = 0; e < kE; ++e)
      if (base + e * (int)blockDim.x < total) S[crow[e] + cc[e]] = acc[e];
  }
}

// u[c] = P[ib][c] of lane src for c in [kC0, kCW) (ib and src uniform).
template <typename T, int NI, int kC0, int kCW>
__device__ __forceinline__ void batch_row(const T (&P)[NI][batch_nb<T>(NI)], int ib, int src, T (&u)[batch_nb<T>(NI)]) {
#pragma unroll
  for (int i = 0; i < NI; ++i)
    if (i == ib) {
#pragma unroll
      for (int c = kC0; c < kCW; ++c) u[c] = __shfl_sync(0xffffffffu, P[i][c], src);
    }
}

// Elimination step k = k0 + j of a panel, by one warp: P[i][kC0] is column k of
// the lane's row pr[i] (logical row lid[i], alive[i] all ones while it is active),
// P[i][kC0 + 1 ..) the panel's later columns.  kShift: the results move one
// register to the left, so the loop over the steps needs no unrolling (FP32: 16
// unrolled steps of 8 rows are over 100 KB of code, and the instruction fetches
// took ten times the step); FP64 steps are unrolled, since every FMA on a column
// past the panel would cost 64 cycles.  Finished multipliers go to S, the pivot
// row to pv[j][0 ..).
// The search looks at the top 32 bits of |a|; ties there, zeros, infinities and
// NaN take the full comparison (strict > in logical row order, NaN never wins).
template <typename T, bool kExact, int NI, int kC0, int kCW, bool kShift>
__device__ __forceinline__ void batch_step(T (&P)[NI][batch_nb<T>(NI)], int (&lid)[NI], unsigned (&alive)[NI],
                                           const int (&pr)[NI], int groups, T* S, int ld, int k, int j, int* piv,
                                           int* prow, T* pv, int& sing, unsigned& mask) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int NB = batch_nb<T>(NI);
  constexpr unsigned kInfTop = sizeof(T) == 8 ? 0x7ff00000u : 0x7f800000u;
  using K = typename PivotKey<T>::K;
  const int lane = threadIdx.x & 31;
  unsigned key[NI], m = 0;
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    key[i] = 0u;
    if (i >= groups) continue;  // no row beyond (uniform)
    unsigned top;
    if constexpr (sizeof(T) == 8)
      top = (unsigned)__double2hiint(P[i][kC0]);
    else
      top = __float_as_uint(P[i][kC0]);
    key[i] = top & 0x7fffffffu & alive[i];
    m = max(m, key[i]);
  }
  const unsigned best = __reduce_max_sync(kFull, m);
  const unsigned vote = __ballot_sync(kFull, m == best);
  int src = __ffs(vote) - 1, ib = 0, same = 0;
#pragma unroll
  for (int i = 0; i < NI; ++i)
    if (i < groups && key[i] == best) {
      ib = i;
      ++same;
    }
  ib = __shfl_sync(kFull, ib | (same > 1 ? 256 : 0), src);
  bool pivot = true;
  if (best == 0 || best >= kInfTop || (vote & (vote - 1u)) || ib >= 256) {
    K bk = 0;
    int bid = INT_MAX, bi = 0, at = -1;
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      const K full = PivotKey<T>::of(P[i][kC0]);
      if (alive[i] && (full > bk || (full == bk && lid[i] < bid))) {
        bk = full;
        bid = lid[i];
        bi = i;
      }
      if (alive[i] && lid[i] == k) at = i;
    }
    src = warp_best(bk, bid);
    pivot = __shfl_sync(kFull, bk, src) > 0;
    if (!pivot) {  // lair: no swap, no update; the row at k retires as it is
      src = __ffs(__ballot_sync(kFull, at >= 0)) - 1;
      bi = at;
      sing = k;
      mask |= 1u << j;
    }
    ib = __shfl_sync(kFull, bi, src);
  }
  T u[NB];
  batch_row<T, NI, kC0, kCW>(P, ib, src, u);
  // Relabel: the row at k takes the pivot's place, the pivot row retires as row k.
  int mine = 0, prr = 0;
#pragma unroll
  for (int i = 0; i < NI; ++i)
    if (i == ib) {
      mine = lid[i];
      prr = pr[i];
    }
  const int pl = __shfl_sync(kFull, mine, src);
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    if (i >= groups) continue;
    if (lid[i] == k) lid[i] = pl;
    if (i == ib && lane == src) {
      lid[i] = k;
      alive[i] = 0u;
    }
  }
  if (lane == src) {
    prow[k] = prr;
    piv[k] = pl;
  }
  if (lane == 0) {
#pragma unroll
    for (int c = kC0; c < kCW; ++c) pv[j * NB + c - kC0] = u[c];
  }
  if (!pivot) {
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      if (alive[i]) S[pr[i] * ld + k] = P[i][kC0];
#pragma unroll
      for (int c = kC0 + 1; c < kCW; ++c)
        if (kShift) P[i][c - 1] = P[i][c];
    }
    return;
  }
  const T recip = T(1) / u[kC0];
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    if (i >= groups) continue;
    const T l = mul_rn(P[i][kC0], recip);
    if (alive[i]) S[pr[i] * ld + k] = l;
#pragma unroll
    for (int c = kC0 + 1; c < kCW; ++c) P[i][kShift ? c - 1 : c] = upd<kExact>(P[i][c], l, u[c]);
  }
}
template <typename T, bool kExact, int NI, int J>
__device__ __forceinline__ void batch_steps_unrolled(T (&P)[NI][batch_nb<T>(NI)], int (&lid)[NI], unsigned (&alive)[NI],
                                                     const int (&pr)[NI], int groups, T* S, int ld, int k0, int w,
                                                     int* piv, int* prow, T* pv, int& sing, unsigned& mask) {
  if constexpr (J < batch_nb<T>(NI)) {
    if (J >= w) return;
    batch_step<T, kExact, NI, J, batch_nb<T>(NI), false>(P, lid, alive, pr, groups, S, ld, k0 + J, J, piv, prow, pv,
                                                       sing, mask);
    batch_steps_unrolled<T, kExact, NI, J + 1>(P, lid, alive, pr, groups, S, ld, k0, w, piv, prow, pv, sing, mask);
  }
}

// Factor and solve one system held in S (n rows of stride ld, the right-hand
// side in column n); prow: physical row of each logical row.  Returns (in warp
// pw, which runs the panels) the last singular step or -1.
template <typename T, bool kExact, int NI>
__device__ __forceinline__ int batch_factor(T* S, int ld, int n, int* piv, int* prow, int* act, int* slid, T* pv,
                                            int* s_na, unsigned* s_mask, int pw) {
  constexpr int NB = batch_nb<T>(NI);
  constexpr unsigned kFull = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int sing = -1;
  for (int k0 = 0; k0 < n; k0 += NB) {
    const int w = min(NB, n - k0);
    if (warp == pw) {
      // The active rows, in the order of act: lane's rows act[lane + 32 i].
      const int rows = n - k0, groups = (rows + 31) / 32;
      T P[NI][NB];
      int lid[NI], pr[NI];
      unsigned alive[NI];
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int q = lane + 32 * i;
        const bool on = q < rows;
        pr[i] = on ? act[q] : 0;
        lid[i] = on ? slid[pr[i]] : -1;
        alive[i] = on ? kFull : 0u;
        const T* row = S + pr[i] * ld + k0;
        if (sizeof(T) == 4 && w == NB) {
#pragma unroll
          for (int c = 0; c < NB; c += 4) {
            const float4 v = on ? *reinterpret_cast<const float4*>(row + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            P[i][c] = v.x, P[i][c + 1] = v.y, P[i][c + 2] = v.z, P[i][c + 3] = v.w;
          }
        } else {
#pragma unroll
          for (int c = 0; c < NB; ++c) P[i][c] = (on && c < w) ? row[c] : T(0);
        }
      }
      unsigned mask = 0;
      if constexpr (sizeof(T) == 8) {
        batch_steps_unrolled<T, kExact, NI, 0>(P, lid, alive, pr, groups, S, ld, k0, w, piv, prow, pv, sing, mask);
      } else {
        const int half = min(w, NB / 2);
        for (int j = 0; j < half; ++j)
          batch_step<T, kExact, NI, 0, NB, true>(P, lid, alive, pr, groups, S, ld, k0 + j, j, piv, prow, pv, sing, mask);
        for (int j = half; j < w; ++j)
          batch_step<T, kExact, NI, 0, NB / 2, true>(P, lid, alive, pr, groups, S, ld, k0 + j, j, piv, prow, pv, sing,
                                                     mask);
      }
      __syncwarp();  // act was read by every lane
      int na = 0;
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const bool rest = alive[i] != 0;
        const unsigned vote = __ballot_sync(kFull, rest);
        if (rest) {
          act[na + __popc(vote & ((1u << lane) - 1u))] = pr[i];
          slid[pr[i]] = lid[i];
        }
        na += __popc(vote);
      }
      if (lane == 0) {
        *s_na = na;
        *s_mask = mask;
      }
    }
    __syncthreads();
    // The pivot rows' panel part (columns k0 + j ..) from pv.
    for (int idx = tid; idx < w * NB; idx += blockDim.x) {
      const int j = idx / NB, c = idx - j * NB;
      if (j + c < w) S[prow[k0 + j] * ld + k0 + j + c] = pv[idx];
    }
    const int c1 = k0 + w, nc = n + 1 - c1, na = *s_na;
    const unsigned mask = *s_mask;
    for (int c = c1 + tid; c <= n; c += blockDim.x) {
      T t[NB];
#pragma unroll
      for (int i = 0; i < NB; ++i) t[i] = i < w ? S[prow[k0 + i] * ld + c] : T(0);
#pragma unroll
      for (int i = 1; i < NB; ++i) {
        if (i >= w) break;
        const T* l = S + prow[k0 + i] * ld + k0;
#pragma unroll
        for (int j = 0; j < NB; ++j)
          if (j < i && !((mask >> j) & 1u)) t[i] = upd<kExact>(t[i], l[j], t[j]);
        S[prow[k0 + i] * ld + c] = t[i];
      }
    }
    if (na > 0) {
      __syncthreads();
      batch_update<kExact, NB>(S, ld, act, na, prow, k0, w, c1, nc, mask);
    }
    __syncthreads();
  }
  return sing;
}

// Back substitution of the factored system; x to global memory.
template <typename T, bool kExact, int NI>
__device__ __forceinline__ void batch_back(T* S, int ld, int n, const int* prow, T* xg, int pw) {
  constexpr unsigned kFull = 0xffffffffu;
  if (kExact) {
    // lair's order: x[i] -= u[i][k] x[k] for k = i+1.. in increasing k.
    if ((int)threadIdx.x == 32 * pw)
      for (int i = n - 1; i >= 0; --i) {
        const T* u = S + prow[i] * ld;
        T acc = u[n];
        for (int k = i + 1; k < n; ++k) acc = upd<true>(acc, u[k], S[prow[k] * ld + n]);
        acc = acc / u[i];
        S[prow[i] * ld + n] = acc;
        xg[i] = acc;
      }
    return;
  }
  if ((int)(threadIdx.x >> 5) != pw) return;
  const int lane = threadIdx.x & 31;
  T x[NI], d[NI], rc[NI];
  const T* row[NI];
  bool good = true;
#pragma unroll
  for (int q = 0; q < NI; ++q) {
    const int i = lane + 32 * q;
    const bool on = i < n;
    row[q] = S + (on ? prow[i] : 0) * ld;
    x[q] = on ? row[q][n] : T(0);
    d[q] = on ? row[q][i] : T(1);
    rc[q] = T(1) / d[q];
    good = good && quot_plain(d[q], rc[q]);
  }
  good = __all_sync(kFull, good);
#pragma unroll
  for (int qb = NI - 1; qb >= 0; --qb) {
    if (32 * qb >= n) continue;
    for (int kk = min(31, n - 1 - 32 * qb); kk >= 0; --kk) {
      const int k = 32 * qb + kk;
      if (lane == kk) x[qb] = quot(x[qb], d[qb], rc[qb], good);
      const T xk = __shfl_sync(kFull, x[qb], kk);
#pragma unroll
      for (int q = 0; q < NI; ++q)
        if (q < qb || (q == qb && lane < kk)) x[q] = upd<false>(x[q], row[q][k], xk);
    }
  }
#pragma unroll
  for (int q = 0; q < NI; ++q)
    if (lane + 32 * q < n) xg[lane + 32 * q] = x[q];
}

// Threads of a CTA, and CTAs an SM's registers must hold.  (kLone: in a plan of no more
// systems than SMs each has an SM, and FP64 systems of more than 128 rows in scratch
// take eight warps, and all its registers, to cover the latency of L2: one of 256 rows
// 2996 -> 2125 us, 152 of them 3209 -> 2256.)
__host__ __device__ constexpr int batch_max_threads(size_t elem, int ni) { return elem == 4 && ni == 8 ? 256 : 128; }
__host__ __device__ constexpr int batch_min_ctas(size_t elem, int ni) {
  return ni <= 2 ? 5 : elem == 4 ? (ni == 4 ? 4 : 2) : (ni == 4 ? 3 : 2);
}

// kScratch: the matrix lives in this CTA's part of `scratch`.
constexpr int kLoneThreads = 256;
template <typename T, bool kExact, int NI, bool kScratch, bool kLone = false>
__global__ void __launch_bounds__(kLone ? kLoneThreads : batch_max_threads(sizeof(T), NI),
                                  kLone ? 1 : batch_min_ctas(sizeof(T), NI))
    batched_lu_kernel(BatchMeta m, T* a, T* b, int* piv, int* info, int* counter, T* scratch) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int prow[kBatchMaxN], act[kBatchMaxN], slid[kBatchMaxN];
  __shared__ __align__(16) T pv[batch_nb<T>(NI) * batch_nb<T>(NI)];
  __shared__ int s_item, s_na;
  __shared__ unsigned s_mask;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, warps = blockDim.x >> 5;
  // The panel warps of an SM's CTAs (numbers 152 apart as they are first placed)
  // on different quarters of it, whose FP64 pipes they occupy.
  const int pw = (blockIdx.x / kNumSmsGB300) & 3;
  for (;;) {
    if (tid == 0) s_item = atomicAdd(counter, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= m.count) break;
    const int sys = m.order[item];
    const int n = m.sizes[sys];
    T* A = a + m.aoff[sys];
    T* xg = b + m.boff[sys];
    T* S = kScratch ? scratch + (size_t)blockIdx.x * kScratchElems : reinterpret_cast<T*>(smem_raw);
    const int ld = kScratch ? kScratchLd : batch_ld<T>(n);
    if (n >= 32) {
      // 32-column pieces of rows, four loads of a lane in flight.
      const int pieces = (n + 31) / 32, items = n * pieces;
      for (int it = warp; it < items; it += 4 * warps) {
        T v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int q = it + e * warps, r = q / pieces, c = (q - r * pieces) * 32 + lane;
          v[e] = (q < items && c < n) ? A[r * n + c] : T(0);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int q = it + e * warps, r = q / pieces, c = (q - r * pieces) * 32 + lane;
          if (q < items && c < n) S[r * ld + c] = v[e];
        }
      }
    } else {
      for (int idx = tid; idx < n * n; idx += blockDim.x) S[(idx / n) * ld + idx % n] = A[idx];
    }
    for (int i = tid; i < n; i += blockDim.x) {
      S[i * ld + n] = xg[i];
      act[i] = slid[i] = i;
    }
    __syncthreads();
    const int sing = batch_factor<T, kExact, NI>(S, ld, n, piv + m.boff[sys], prow, act, slid, pv, &s_na,
                                                 &s_mask, pw);
    batch_back<T, kExact, NI>(S, ld, n, prow, xg, pw);
    if (n >= 32) {
      for (int r = warp; r < n; r += warps) {
        const T* src = S + prow[r] * ld;
        for (int c = lane; c < n; c += 32) A[r * n + c] = src[c];
      }
    } else {
      for (int idx = tid; idx < n * n; idx += blockDim.x) A[idx] = S[prow[idx / n] * ld + idx % n];
    }
    if (tid == 32 * pw) info[sys] = sing;
    __syncthreads();
  }
}

}  // namespace luhot

// ---------------------------------------------------------------------------
// Plan object (host).
// ---------------------------------------------------------------------------
namespace luhot {

// A launch: the systems order[first .. first + count) on CTAs of one kernel.
struct BatchClass {
  int first = 0, count = 0;
  int ni = 1;            // rows of a panel lane
  bool scratch = false;
  bool lone = false;     // an SM to each system (kLone)
  int threads = 0, grid = 0;
  size_t smem = 0;
};
constexpr int kMaxBatchClasses = 16;
constexpr int kBatchStreams = 4;  // the capturing stream and three branches

}  // namespace luhot

struct luhot_batch {
  luhot_ctx* ctx = nullptr;
  int dtype = 0;  // 0 f64, 1 f32
  int mode = LUHOT_MODE_FAST;
  int64_t count = 0;
  int64_t a_elems = 0, b_elems = 0;
  std::vector<int> sizes;
  std::vector<int64_t> aoff, boff;
  std::vector<int> order;
  std::vector<luhot::BatchClass> classes;
  int tune[luhot::kBuckets];  // 0: shared memory where it fits, else the panel width of the scratch form
  int smem_n = 0;
  // device metadata: sizes, aoff, boff, order, counters
  void* d_meta = nullptr;
  int* d_counter = nullptr;
  luhot::BatchMeta meta{};
  // matrices of the CTAs of scratch classes (none without such systems)
  void* d_scratch = nullptr;
  size_t scratch_ctas = 0;
  cudaStream_t branch[luhot::kBatchStreams - 1] = {nullptr, nullptr, nullptr};
  cudaEvent_t fork = nullptr, joined[luhot::kBatchStreams - 1] = {nullptr, nullptr, nullptr};
  // cached graph
  cudaGraphExec_t exec = nullptr;
  cudaGraph_t graph = nullptr;
  void* g_ptrs[4] = {nullptr, nullptr, nullptr, nullptr};
};

namespace luhot {

static size_t elem_size(int dtype) { return dtype == 0 ? sizeof(double) : sizeof(float); }
static size_t smem_bytes(int dtype, int n) {
  return dtype == 0 ? (size_t)n * batch_ld<double>(n) * sizeof(double) : (size_t)n * batch_ld<float>(n) * sizeof(float);
}
static int batch_width(int dtype) { return dtype == 0 ? batch_nb<double>(8) : batch_nb<float>(8); }

static int smem_n_for(int dtype, size_t budget) {
  int n = 8;
  while (n + 1 <= kBatchMaxN && smem_bytes(dtype, n + 1) <= budget) ++n;
  return n;
}

template <typename T, bool kExact>
static const void* batch_kernel_of(int ni, bool scratch) {
  if (scratch)
    return ni == 1   ? (const void*)batched_lu_kernel<T, kExact, 1, true>
           : ni == 2 ? (const void*)batched_lu_kernel<T, kExact, 2, true>
           : ni == 4 ? (const void*)batched_lu_kernel<T, kExact, 4, true>
                     : (const void*)batched_lu_kernel<T, kExact, 8, true>;
  return ni == 1   ? (const void*)batched_lu_kernel<T, kExact, 1, false>
         : ni == 2 ? (const void*)batched_lu_kernel<T, kExact, 2, false>
         : ni == 4 ? (const void*)batched_lu_kernel<T, kExact, 4, false>
                   : (const void*)batched_lu_kernel<T, kExact, 8, false>;
}
static const void* batch_kernel(int dtype, int mode, int ni, bool scratch, bool lone) {
  const bool ex = mode == LUHOT_MODE_EXACT;
  if (lone)
    return ex ? (const void*)batched_lu_kernel<double, true, 8, true, true>
              : (const void*)batched_lu_kernel<double, false, 8, true, true>;
  if (dtype == 0)
    return ex ? batch_kernel_of<double, true>(ni, scratch) : batch_kernel_of<double, false>(ni, scratch);
  return ex ? batch_kernel_of<float, true>(ni, scratch) : batch_kernel_of<float, false>(ni, scratch);
}

// Orders the systems (indices into sizes) by class, largest class and largest
// system first.  A class is a panel form (NI) and the number of its largest
// matrices that fit in an SM's shared memory (or the scratch form).  few: the plan
// has no more systems than SMs.
static void build_classes(luhot_ctx* ctx, int dtype, int mode, const int* tune, int smem_n, bool few,
                          const std::vector<int>& sizes, std::vector<int>& order, std::vector<BatchClass>& classes) {
  auto key_of = [&](int n) {
    const int ni = n <= 32 ? 1 : n <= 64 ? 2 : n <= 128 ? 4 : 8;
    const bool scratch = n > smem_n || tune[batch_bucket(n)] != 0;
    const size_t bytes = smem_bytes(dtype, n);
    int fit = 8;  // CTAs to an SM
    if (scratch)
      fit = 0;
    else
      for (int f : {6, 4, 3, 2, 1})
        if (bytes + 3 * 1024 > kBatchSmem / f) fit = f == 6 ? 4 : f == 4 ? 3 : f == 3 ? 2 : 1;
    return (8 - ni) * 16 + fit;  // larger rows first, then fewer to an SM
  };
  // Sizes by class and size, the systems of each in their order.
  int key[kBatchMaxN + 1], by_class[kBatchMaxN], at[kBatchMaxN + 1], count[kBatchMaxN + 1] = {};
  for (int n = 1; n <= kBatchMaxN; ++n) {
    key[n] = key_of(n);
    by_class[n - 1] = n;
  }
  std::sort(by_class, by_class + kBatchMaxN, [&](int x, int y) { return key[x] != key[y] ? key[x] < key[y] : x > y; });
  for (int n : sizes) ++count[n];
  int next = 0;
  for (int n : by_class) {
    at[n] = next;
    next += count[n];
  }
  order.resize(sizes.size());
  for (size_t i = 0; i < sizes.size(); ++i) order[at[sizes[i]]++] = (int)i;
  classes.clear();
  for (size_t i = 0; i < order.size();) {
    const int n = sizes[order[i]], k = key[n];
    size_t e = i;
    while (e < order.size() && key[sizes[order[e]]] == k) ++e;
    BatchClass c;
    c.first = (int)i;
    c.count = (int)(e - i);
    c.ni = 8 - k / 16;
    c.scratch = k % 16 == 0;
    c.smem = c.scratch ? 0 : smem_bytes(dtype, n);  // the class's first system is its largest
    // Few matrices of more than 128 rows fit in an SM's shared memory: 8 warps each.
    c.lone = few && dtype == 0 && c.ni == 8 && c.scratch;
    c.threads = c.lone ? kLoneThreads : c.scratch ? 128 : batch_max_threads(elem_size(dtype), c.ni);
    const void* kern = batch_kernel(dtype, mode, c.ni, c.scratch, c.lone);
    allow_max_dynamic_smem(kern);
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, c.threads, c.smem) != cudaSuccess) {
      cudaGetLastError();
      per_sm = 1;
    }
    c.grid = std::min(c.count, std::max(1, per_sm) * ctx->num_sms);
    classes.push_back(c);
    i = e;
  }
}

// Branches of a launch of `classes` classes (the first class's is the stream itself),
// made when a plan first has so many: a plan of one class makes none.
static int batch_branches(const std::vector<BatchClass>& classes) {
  return std::max(0, std::min((int)classes.size(), kBatchStreams) - 1);
}
static int make_branches(luhot_batch* p, const std::vector<BatchClass>& classes) {
  const int nb = batch_branches(classes);
  if (nb > 0 && !p->fork) LUHOT_CUDA_TRY(p->ctx, cudaEventCreateWithFlags(&p->fork, cudaEventDisableTiming));
  for (int q = 0; q < nb; ++q) {
    if (!p->branch[q]) LUHOT_CUDA_TRY(p->ctx, cudaStreamCreateWithFlags(&p->branch[q], cudaStreamNonBlocking));
    if (!p->joined[q]) LUHOT_CUDA_TRY(p->ctx, cudaEventCreateWithFlags(&p->joined[q], cudaEventDisableTiming));
  }
  return LUHOT_OK;
}

// The sample systems' matrices and right-hand sides, packed: sample q is system
// sys[q] of the plan.  Words of the element's size.
template <typename W>
__global__ void gather_samples_kernel(const W* __restrict__ a, const W* __restrict__ b, const int* __restrict__ sys,
                                      const int* __restrict__ sizes, const int64_t* __restrict__ aoff,
                                      const int64_t* __restrict__ boff, const int64_t* __restrict__ s_aoff,
                                      const int64_t* __restrict__ s_boff, W* __restrict__ pa, W* __restrict__ pb) {
  const int q = blockIdx.x, i = sys[q], n = sizes[q];
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) pa[s_aoff[q] + e] = a[aoff[i] + e];
  for (int e = threadIdx.x; e < n; e += blockDim.x) pb[s_boff[q] + e] = b[boff[i] + e];
}

// Clears the counters and launches every class, the branches' share on their
// streams between a fork and a join (so a capture of `stream` holds them all).
static cudaError_t launch_classes(luhot_batch* p, const std::vector<BatchClass>& classes, const BatchMeta& m,
                                  void* scratch, void* a, void* b, int* piv, int* info, int* counters,
                                  cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(counters, 0, kMaxBatchClasses * sizeof(int), stream);
  const int nb = batch_branches(classes);
  if (e == cudaSuccess && nb > 0) e = cudaEventRecord(p->fork, stream);
  for (int q = 0; q < nb && e == cudaSuccess; ++q) e = cudaStreamWaitEvent(p->branch[q], p->fork, 0);
  char* sp = static_cast<char*>(scratch);
  for (size_t i = 0; i < classes.size() && e == cudaSuccess; ++i) {
    const BatchClass& c = classes[i];
    BatchMeta cm = m;
    cm.order = m.order + c.first;
    cm.count = c.count;
    int* counter = counters + i;
    void* cs = c.scratch ? sp : nullptr;
    if (c.scratch) sp += (size_t)c.grid * kScratchElems * elem_size(p->dtype);
    void* args[] = {&cm, &a, &b, &piv, &info, &counter, &cs};
    const int q = (int)(i % kBatchStreams);
    e = cudaLaunchKernel(batch_kernel(p->dtype, p->mode, c.ni, c.scratch, c.lone), dim3(c.grid), dim3(c.threads), args, c.smem,
                         q == 0 ? stream : p->branch[q - 1]);
  }
  for (int q = 0; q < nb; ++q) {  // the join, also after an error
    cudaError_t j = cudaEventRecord(p->joined[q], p->branch[q]);
    if (j == cudaSuccess) j = cudaStreamWaitEvent(stream, p->joined[q], 0);
    if (e == cudaSuccess) e = j;
  }
  return e;
}

static size_t scratch_ctas(const std::vector<BatchClass>& classes) {
  size_t n = 0;
  for (const auto& c : classes)
    if (c.scratch) n += c.grid;
  return n;
}

static int upload_meta(luhot_batch* p) {
  luhot_ctx* ctx = p->ctx;
  const size_t c = (size_t)p->count;
  build_classes(ctx, p->dtype, p->mode, p->tune, p->smem_n, p->count <= ctx->num_sms, p->sizes, p->order, p->classes);
  if ((int)p->classes.size() > kMaxBatchClasses) return set_error(ctx, LUHOT_ERR_UNSUPPORTED, "batch: too many size classes");
  int rc = make_branches(p, p->classes);
  if (rc) return rc;
  const size_t need = scratch_ctas(p->classes);
  if (need > p->scratch_ctas) {
    if (p->d_scratch) cudaFree(p->d_scratch);
    p->d_scratch = nullptr;
    p->scratch_ctas = 0;
    LUHOT_CUDA_TRY(ctx, cudaMalloc(&p->d_scratch, need * kScratchElems * elem_size(p->dtype)));
    p->scratch_ctas = need;
  }
  const size_t bytes = c * (sizeof(int) + 2 * sizeof(int64_t) + sizeof(int)) + 256;
  if (!p->d_meta) {
    LUHOT_CUDA_TRY(ctx, cudaMalloc(&p->d_meta, bytes));
    LUHOT_CUDA_TRY(ctx, cudaMalloc(&p->d_counter, 256));
  }
  char* base = static_cast<char*>(p->d_meta);
  int64_t* aoff = reinterpret_cast<int64_t*>(base);
  int64_t* boff = aoff + c;
  int* sizes = reinterpret_cast<int*>(boff + c);
  int* order = sizes + c;
  // On the context's stream and waited for: a copy on the default stream can return
  // before its data has arrived, and orders nothing for streams that do not block on it.
  auto up = [&](void* dst, const void* src, size_t bytes) {
    return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream);
  };
  LUHOT_CUDA_TRY(ctx, up(aoff, p->aoff.data(), c * sizeof(int64_t)));
  LUHOT_CUDA_TRY(ctx, up(boff, p->boff.data(), c * sizeof(int64_t)));
  LUHOT_CUDA_TRY(ctx, up(sizes, p->sizes.data(), c * sizeof(int)));
  LUHOT_CUDA_TRY(ctx, up(order, p->order.data(), c * sizeof(int)));
  LUHOT_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  p->meta.sizes = sizes;
  p->meta.aoff = aoff;
  p->meta.boff = boff;
  p->meta.order = order;
  p->meta.count = (int)p->count;
  return LUHOT_OK;
}

static void drop_graph(luhot_batch* p) {
  if (p->exec) cudaGraphExecDestroy(p->exec);
  if (p->graph) cudaGraphDestroy(p->graph);
  p->exec = nullptr;
  p->graph = nullptr;
  for (auto& q : p->g_ptrs) q = nullptr;
}

}  // namespace luhot

using namespace luhot;

extern "C" {

int luhot_batch_create(luhot_ctx* ctx, int64_t count, const int32_t* sizes, int dtype, int mode, luhot_batch** out) {
  LUHOT_NVTX_FN();
  if (!ctx || !out) return LUHOT_ERR_INVALID_ARG;
  CtxGuard g(ctx);
  *out = nullptr;
  if (count < 0 || count >= INT32_MAX || (count > 0 && !sizes) || (dtype != 0 && dtype != 1) ||
      (mode != LUHOT_MODE_FAST && mode != LUHOT_MODE_EXACT))
    return set_error(ctx, LUHOT_ERR_INVALID_ARG, "batch: invalid arguments");
  for (int64_t i = 0; i < count; ++i)
    if (sizes[i] < 1 || sizes[i] > kBatchMaxN)
      return set_error(ctx, LUHOT_ERR_UNSUPPORTED, "batch: system sizes must be in [1, 256]");
  luhot_batch* p = new (std::nothrow) luhot_batch();
  if (!p) return LUHOT_ERR_ALLOC;
  p->ctx = ctx;
  p->dtype = dtype;
  p->mode = mode;
  p->count = count;
  p->sizes.assign(sizes, sizes + count);
  p->aoff.resize(count);
  p->boff.resize(count);
  int64_t ao = 0, bo = 0;
  for (int64_t i = 0; i < count; ++i) {
    p->aoff[i] = ao;
    p->boff[i] = bo;
    ao += (int64_t)sizes[i] * sizes[i];
    bo += sizes[i];
  }
  p->a_elems = ao;
  p->b_elems = bo;
  p->smem_n = smem_n_for(dtype, kBatchSmem);
  // Untuned: shared memory where it fits for FP32; FP64 up to 96, where three
  // CTAs or more share an SM (its pipe idles while one CTA's panel runs).
  for (int bk = 0; bk < kBuckets; ++bk) p->tune[bk] = dtype == 0 && bk > 3 ? batch_width(dtype) : 0;
  int rc = count > 0 ? upload_meta(p) : LUHOT_OK;
  if (rc) {
    luhot_batch_destroy(p);
    return rc;
  }
  *out = p;
  return LUHOT_OK;
}

void luhot_batch_destroy(luhot_batch* p) {
  if (!p) return;
  cudaSetDevice(p->ctx->device);
  drop_graph(p);
  if (p->d_meta) cudaFree(p->d_meta);
  if (p->d_counter) cudaFree(p->d_counter);
  if (p->d_scratch) cudaFree(p->d_scratch);
  for (auto& s : p->branch)
    if (s) cudaStreamDestroy(s);
  for (auto& e : p->joined)
    if (e) cudaEventDestroy(e);
  if (p->fork) cudaEventDestroy(p->fork);
  delete p;
}

int luhot_batch_layout(const luhot_batch* p, int64_t* a_elems, int64_t* b_elems) {
  if (!p) return LUHOT_ERR_INVALID_ARG;
  if (a_elems) *a_elems = p->a_elems;
  if (b_elems) *b_elems = p->b_elems;
  return LUHOT_OK;
}

int luhot_batch_tuning(const luhot_batch* p, int32_t* nb_per_bucket, int32_t* smem_n) {
  if (!p) return LUHOT_ERR_INVALID_ARG;
  if (nb_per_bucket)
    for (int i = 0; i < kBuckets; ++i) nb_per_bucket[i] = p->tune[i];
  if (smem_n) *smem_n = p->smem_n;
  return LUHOT_OK;
}

int luhot_selftest_batch_form(luhot_batch* p, int form) {
  if (!p || form < 0 || form > 1) return LUHOT_ERR_INVALID_ARG;
  CtxGuard g(p->ctx);
  for (int& t : p->tune) t = form ? batch_width(p->dtype) : 0;
  drop_graph(p);
  return p->count > 0 ? upload_meta(p) : LUHOT_OK;
}

int luhot_batch_solve(luhot_batch* p, void* d_a, void* d_b, int32_t* d_piv, int32_t* d_info) {
  LUHOT_NVTX_FN();
  if (!p) return LUHOT_ERR_INVALID_ARG;
  luhot_ctx* ctx = p->ctx;
  CtxGuard g(ctx);
  if (p->count == 0) return LUHOT_OK;
  if (!d_a || !d_b || !d_piv || !d_info) return set_error(ctx, LUHOT_ERR_INVALID_ARG, "batch: null pointer");
  void* ptrs[4] = {d_a, d_b, d_piv, d_info};
  if (!p->exec || memcmp(ptrs, p->g_ptrs, sizeof(ptrs)) != 0) {
    drop_graph(p);
    // Capture [counter reset, the classes' launches] once for these buffers.
    LUHOT_CUDA_TRY(ctx, cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
    cudaError_t e = launch_classes(p, p->classes, p->meta, p->d_scratch, d_a, d_b, d_piv, d_info, p->d_counter,
                                   ctx->stream);
    cudaGraph_t graph = nullptr;
    cudaError_t e2 = cudaStreamEndCapture(ctx->stream, &graph);
    if (e != cudaSuccess || e2 != cudaSuccess) {
      if (graph) cudaGraphDestroy(graph);
      cudaGetLastError();
      return set_error(ctx, LUHOT_ERR_CUDA, std::string("batch: graph capture failed: ") +
                                                cudaGetErrorString(e != cudaSuccess ? e : e2));
    }
    p->graph = graph;
    LUHOT_CUDA_TRY(ctx, cudaGraphInstantiate(&p->exec, p->graph, 0));
    memcpy(p->g_ptrs, ptrs, sizeof(ptrs));
  }
  prof_begin(ctx, kProfOther);
  LUHOT_CUDA_TRY(ctx, cudaGraphLaunch(p->exec, ctx->stream));
  double fl = 0.0;
  for (int n : p->sizes) fl += 2.0 / 3.0 * n * (double)n * n + 2.0 * n * (double)n;
  prof_end(ctx, kProfOther, fl, (double)(p->a_elems + p->b_elems) * 2 * elem_size(p->dtype));
  LUHOT_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return LUHOT_OK;
}

// Time both forms (shared memory where it fits, scratch) per size bucket on up
// to 304 sample systems of that bucket (two per SM, so that it is throughput and
// not one system's latency that is compared), copied from the caller's data into
// scratch before each run, and keep the faster.
constexpr size_t kTuneSample = 2 * kNumSmsGB300;
int luhot_batch_autotune(luhot_batch* p, const void* d_a, const void* d_b) {
  LUHOT_NVTX_FN();
  if (!p) return LUHOT_ERR_INVALID_ARG;
  luhot_ctx* ctx = p->ctx;
  CtxGuard g(ctx);
  if (p->count == 0) return LUHOT_OK;
  if (!d_a || !d_b) return set_error(ctx, LUHOT_ERR_INVALID_ARG, "batch: null pointer");
  const size_t es = elem_size(p->dtype);
  std::vector<std::vector<int>> members(kBuckets);
  for (int64_t i = 0; i < p->count; ++i) {
    auto& v = members[batch_bucket(p->sizes[i])];
    if (v.size() < kTuneSample) v.push_back((int)i);
  }
  // Scratch: sample matrices + rhs, and a pristine copy to restore from.
  int64_t sa = 0, sb = 0;
  for (auto& v : members)
    for (int i : v) {
      sa += (int64_t)p->sizes[i] * p->sizes[i];
      sb += p->sizes[i];
    }
  const size_t scratch = (size_t)(2 * sa + 2 * sb) * es + (size_t)sb * sizeof(int) + (size_t)p->count * sizeof(int) +
                         8 * 256;
  int rc = ensure_buf(ctx, ctx->work[1], scratch);
  if (rc) return rc;
  char* base = static_cast<char*>(ctx->work[1].ptr);
  char* wa = base;
  char* wb = wa + sa * es;
  char* pa = wb + sb * es;
  char* pb = pa + sa * es;
  int* spiv = reinterpret_cast<int*>(pb + sb * es);
  int* sinfo = spiv + sb;
  // Per-bucket sample metadata in the plan's layout style.
  std::vector<int> s_sizes, s_sys;
  std::vector<int64_t> s_aoff, s_boff;
  std::vector<int> bucket_first(kBuckets + 1, 0);
  int64_t ao = 0, bo = 0;
  for (int bk = 0; bk < kBuckets; ++bk) {
    bucket_first[bk] = (int)s_sizes.size();
    for (int i : members[bk]) {
      const int n = p->sizes[i];
      s_sizes.push_back(n);
      s_sys.push_back(i);
      s_aoff.push_back(ao);
      s_boff.push_back(bo);
      ao += (int64_t)n * n;
      bo += n;
    }
  }
  bucket_first[kBuckets] = (int)s_sizes.size();
  const int ns = (int)s_sizes.size();
  DevBuf meta_buf, mat_buf;
  rc = ensure_buf(ctx, meta_buf, (size_t)ns * (2 * sizeof(int64_t) + 2 * sizeof(int)) + kMaxBatchClasses * sizeof(int) + 512);
  if (rc) return rc;
  int64_t* m_aoff = static_cast<int64_t*>(meta_buf.ptr);
  int64_t* m_boff = m_aoff + ns;
  int* m_sizes = reinterpret_cast<int*>(m_boff + ns);
  int* m_order = m_sizes + ns;
  int* m_counter = m_order + ns;
  cudaMemcpyAsync(m_aoff, s_aoff.data(), ns * sizeof(int64_t), cudaMemcpyHostToDevice, ctx->stream);
  cudaMemcpyAsync(m_boff, s_boff.data(), ns * sizeof(int64_t), cudaMemcpyHostToDevice, ctx->stream);
  cudaMemcpyAsync(m_sizes, s_sizes.data(), ns * sizeof(int), cudaMemcpyHostToDevice, ctx->stream);
  cudaMemcpyAsync(m_order, s_sys.data(), ns * sizeof(int), cudaMemcpyHostToDevice, ctx->stream);
  if (es == 8)
    gather_samples_kernel<unsigned long long><<<ns, 256, 0, ctx->stream>>>(
        static_cast<const unsigned long long*>(d_a), static_cast<const unsigned long long*>(d_b), m_order, m_sizes,
        p->meta.aoff, p->meta.boff, m_aoff, m_boff, reinterpret_cast<unsigned long long*>(pa),
        reinterpret_cast<unsigned long long*>(pb));
  else
    gather_samples_kernel<unsigned><<<ns, 256, 0, ctx->stream>>>(
        static_cast<const unsigned*>(d_a), static_cast<const unsigned*>(d_b), m_order, m_sizes, p->meta.aoff,
        p->meta.boff, m_aoff, m_boff, reinterpret_cast<unsigned*>(pa), reinterpret_cast<unsigned*>(pb));
  count_launch(ctx);
  if (cudaError_t e = cudaGetLastError(); e != cudaSuccess || (e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) {
    cudaFree(meta_buf.ptr);
    return set_error(ctx, LUHOT_ERR_CUDA, std::string("batch autotune: ") + cudaGetErrorString(e));
  }
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaError_t err = cudaSuccess;
  for (int bk = 0; bk < kBuckets && !rc; ++bk) {
    const int first = bucket_first[bk], cnt = bucket_first[bk + 1] - first;
    if (cnt == 0) continue;
    const std::vector<int> b_sizes(s_sizes.begin() + first, s_sizes.begin() + first + cnt);
    if (*std::min_element(b_sizes.begin(), b_sizes.end()) > p->smem_n) {
      p->tune[bk] = batch_width(p->dtype);  // nothing of it fits in shared memory
      continue;
    }
    float best = 1e30f;
    int best_form = p->tune[bk];
    for (const int form : {0, batch_width(p->dtype)}) {
      int tune_all[kBuckets];
      for (int q = 0; q < kBuckets; ++q) tune_all[q] = form;
      std::vector<int> order;
      std::vector<BatchClass> classes;
      build_classes(ctx, p->dtype, p->mode, tune_all, p->smem_n, p->count <= ctx->num_sms, b_sizes, order, classes);
      rc = make_branches(p, classes);
      if (rc) break;
      for (auto& q : order) q += first;
      rc = ensure_buf(ctx, mat_buf, scratch_ctas(classes) * kScratchElems * es);
      if (rc) break;
      cudaMemcpyAsync(m_order, order.data(), cnt * sizeof(int), cudaMemcpyHostToDevice, ctx->stream);
      BatchMeta m{m_sizes, m_aoff, m_boff, m_order, cnt};
      float ms = 0.f;
      for (int rep = 0; rep < 2 && err == cudaSuccess; ++rep) {
        const int64_t a0 = s_aoff[first], a1 = first + cnt < ns ? s_aoff[first + cnt] : sa;
        cudaMemcpyAsync(wa + a0 * es, pa + a0 * es, (a1 - a0) * es, cudaMemcpyDeviceToDevice, ctx->stream);
        cudaMemcpyAsync(wb, pb, sb * es, cudaMemcpyDeviceToDevice, ctx->stream);
        cudaEventRecord(e0, ctx->stream);
        err = launch_classes(p, classes, m, mat_buf.ptr, wa, wb, spiv, sinfo, m_counter, ctx->stream);
        cudaEventRecord(e1, ctx->stream);
        if (err == cudaSuccess) err = cudaEventSynchronize(e1);
        cudaEventElapsedTime(&ms, e0, e1);
      }
      if (err != cudaSuccess) {
        rc = set_error(ctx, LUHOT_ERR_CUDA, std::string("batch autotune: ") + cudaGetErrorString(err));
        break;
      }
      count_launch(ctx, 2 * (int64_t)classes.size());
      if (ms < best) {
        best = ms;
        best_form = form;
      }
    }
    p->tune[bk] = best_form;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(meta_buf.ptr);
  if (mat_buf.ptr) cudaFree(mat_buf.ptr);
  if (rc) return rc;
  drop_graph(p);
  return upload_meta(p);
}

// Host-buffer form: packed host arrays in the plan's layout, staged in and out.
int luhot_batch_solve_host(luhot_batch* p, void* a, void* b, int32_t* piv, int32_t* info) {
  LUHOT_NVTX_FN();
  if (!p) return LUHOT_ERR_INVALID_ARG;
  luhot_ctx* ctx = p->ctx;
  if (p->count == 0) return LUHOT_OK;
  if (!a || !b || !piv || !info) return set_error(ctx, LUHOT_ERR_INVALID_ARG, "batch: null pointer");
  const size_t es = elem_size(p->dtype);
  void *d_a, *d_b;
  int *d_piv, *d_info;
  {
    CtxGuard g(ctx);
    int rc = ensure_buf(ctx, ctx->work[0], (size_t)p->a_elems * es);
    if (!rc) rc = ensure_buf(ctx, ctx->work[2], (size_t)p->b_elems * (es + sizeof(int)) + (size_t)p->count * sizeof(int) + 256);
    if (rc) return rc;
    d_a = ctx->work[0].ptr;
    d_b = ctx->work[2].ptr;
    d_piv = reinterpret_cast<int*>(static_cast<char*>(d_b) + (size_t)p->b_elems * es);
    d_info = d_piv + p->b_elems;
    LUHOT_CUDA_TRY(ctx, cudaMemcpyAsync(d_a, a, (size_t)p->a_elems * es, cudaMemcpyHostToDevice, ctx->stream));
    LUHOT_CUDA_TRY(ctx, cudaMemcpyAsync(d_b, b, (size_t)p->b_elems * es, cudaMemcpyHostToDevice, ctx->stream));
  }
  int rc = luhot_batch_solve(p, d_a, d_b, d_piv, d_info);
  if (rc) return rc;
  CtxGuard g(ctx);
  LUHOT_CUDA_TRY(ctx, cudaMemcpyAsync(a, d_a, (size_t)p->a_elems * es, cudaMemcpyDeviceToHost, ctx->stream));
  LUHOT_CUDA_TRY(ctx, cudaMemcpyAsync(b, d_b, (size_t)p->b_elems * es, cudaMemcpyDeviceToHost, ctx->stream));
  LUHOT_CUDA_TRY(ctx, cudaMemcpyAsync(piv, d_piv, (size_t)p->b_elems * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  LUHOT_CUDA_TRY(ctx, cudaMemcpyAsync(info, d_info, (size_t)p->count * sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  LUHOT_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->stream));
  return LUHOT_OK;
}

}  // extern "C"
