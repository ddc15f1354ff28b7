// FP64 Schur update on the FP16 tensor cores (Ozaki scheme).
//
//   C (M x N, FP64, row-major, ldc)  -=  L (M x K) U (K x N),   K <= 128
//
// This part runs FP64 at about 2 FMA per clock per SM and FP16 tensor-core
// products at 4096 per clock, so fast-mode FP64 trailing updates are computed
// as exact integer products on the tensor cores:
//
// Split (oz_split_rows_kernel for L, oz_split_cols_kernel for U).  Row i of L
//   gets the exponent ea[i] with max_k |L(i,k)| < 2^ea[i], column j of U the
//   exponent eb[j] (K > 64: one for both halves of 64, unless they lie apart, see
//   kOzApart).  Each element x of a row (column) with exponent e is
//   rounded to the 56-bit integer N = round(|x| 2^(56-e)) and written as seven
//   balanced base-256 digits, most significant first:
//       x = sign(x) 2^e sum_{p=0..6} d_p 2^(-8(p+1))    (error <= 2^(e-57)),
//   d_0 in [-256, 256], d_1..d_6 in [-128, 128], every digit exact in FP16.
//   The digits of L are stored K-major per slice, As[p][i][k], those of U
//   transposed, Bs[p][j][k] (one 128-byte row per i or j: one TMA box row).
// Products (oz_gemm_kernel).  With A_p, B_q the digit matrices,
//       L U = 2^(ea+eb) sum_G T_G 2^(-8(G+2)),   T_G = sum_{p+q=G} A_p B_q^T,
//   kept for G = 0..6 (28 slice products of the 49).  Every partial sum of
//   T_G is an integer of magnitude below 9 * 2^20 for K <= 64, and at most 2^24
//   for K <= 128 but for group 6, whose two K halves have an accumulator each, so
//   the FP32 accumulation in TMEM is exact.  The dropped groups (G >= 7) weigh at
//   most 2^-49.4 of 2^(ea+eb) for K = 64, 2^-48.4 for K = 128 (typically 2^-55),
//   the element roundings 2^-57 of each operand's scale.  That is relative to the
//   largest elements of the row and the column, not to |L||U|: on rows and columns of
//   one scale well inside FP64's own bound for a K-term dot product (measured on
//   N(0,1) factors: 1.1e-16 of |C| + |L||U| against 4.7e-16 for the FP64 tensor
//   cores), but more where a row's large elements meet a column's small ones.
// Combine (epilogue).  R = floor(sum_G T_G 2^(38-8G)), a 64-bit integer (|R| < 2^62),
//   then C = C - R 2^(ea+eb-54): one rounding of R to 53 bits (built with integer
//   operations) and one of the subtraction.  Rows or columns holding Inf or NaN
//   give NaN in the elements they touch.
//
// oz_gemm_kernel: persistent, one CTA per SM, tiles of 128 columns x 64 rows of C,
// a contiguous range per CTA in row-block order.  What bounds it is the epilogue's
// arithmetic, 64 cycles of an SM quarter's FP64 pipe a warp's subtraction and about
// as many for the rest, so that a product is worth doing over K = 128 (two "halves"
// of 64): one epilogue instead of two.  A 128 x 64 tile leaves TMEM room for all
// eight accumulators at once, and the MMAs of a piece of U against stacked pieces
// of L are then single products with N up to 256 on neighbouring accumulators:
// 10 a k-step in place of 28, the tensor pipe's full rate (3700 cycles a half).  The
// MMAs compute C^T: TMEM lanes are C's columns, so a warp's accesses to one row of C
// are 32 consecutive doubles.  Cycles a tile, K = 64 / 128: MMAs 5300 / 10100 (U's
// pieces come from L2 at 23 bytes a cycle and SM), folds 3500 / 4000, C and
// subtraction 7200; together 11800 / 14400 (a 128 x 128 tile with three
// accumulators, a fold per group on 64-bit words: 29000 for K = 64).  n = 16384's
// updates: 142 ms before, 114 in steps of K = 64, 74 with K = 128.  Eighteen warps:
//   warp 0      TMA producer: the L pieces (a slice's 64 rows x 64 k, 8 KB) of the
//               CTA's row block, reloaded when the row block changes, and the
//               seven U pieces (128 columns, 16 KB) of each tile and half, one
//               barrier pair per piece, in the order the MMAs free them (6 .. 0);
//               3-D tensor maps (k, row, slice), 128-byte swizzle, rows past M or
//               N zero-filled;
//   warp 1      TMEM owner (512 columns) and MMA issuer: per tile and half, U pieces
//               6 .. 0 against L pieces 0 .. 6 - q, 4 k-steps of K = 16 each, then
//               a commit to that piece's empty barrier; a commit to the tile's full
//               barrier at its end;
//   warps 2-17  epilogue: per group the accumulator is read and released, so that
//               the next tile's first MMAs overlap the folds and the rest of them
//               the work on C; C is prefetched into L2 at the tile's start.
// All mbarrier waits are bounded by the context's wait limit; on expiry a role
// records the error and raises the CTA's abort flag, the others stop at their
// next wait, and before exit the CTA waits (bounded) for its copies and MMAs
// in flight and frees TMEM.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <string>
#include <type_traits>

#include "common.cuh"
#include "luhot_internal.h"
#include "ozaki.cuh"
#include "ozaki_split.cuh"
#include "tcgen05.cuh"

namespace luhot {

constexpr int kOzBN = 128;     // columns of C of a tile (TMEM lanes)
constexpr int kOzBM = 64;      // rows of C of a tile (TMEM columns of an accumulator)
constexpr int kOzMaxHalves = 2;  // K = 64 or 128
constexpr int kOzFrac = 38;    // fractional bits of the fixed-point combine
constexpr int kOzEpiWarps = 16;
constexpr int kOzThreads = 64 + 32 * kOzEpiWarps;
constexpr int kOzRows = kOzBM / 4;              // rows of C of an epilogue thread
constexpr int kOzUBytes = kOzBN * kOzK * 2;     // a U piece: one slice, one K half, 128 columns
constexpr int kOzLBytes = kOzBM * kOzK * 2;     // an L piece: 64 rows
constexpr size_t kOzSmem = 1024 + (size_t)kOzSlices * kOzUBytes + (size_t)kOzMaxHalves * kOzSlices * kOzLBytes;
constexpr int kOzAccs = kOzGroups + 1;  // accumulators: groups 0 .. 6 and group 6 of the second K half
static_assert(kOzAccs * kOzBM <= 512, "the accumulators fit in TMEM");

// ---------------------------------------------------------------------------
// Split (digits: ozaki_split.cuh).
// ---------------------------------------------------------------------------

// Two K halves share their exponents unless the halves of some row of L and those of
// some column of U lie more than kOzApart bits apart (a zero half lies apart from
// any other).  A shared exponent costs an element of C the smaller of its row's and
// its column's distance at most, where the larger half of one meets the smaller half
// of the other: without such a row, or without such a column, kOzApart bits.  With
// both the operands are split again (oz_resplit_kernel), an exponent a half, and the
// product is bit for bit that of two products of K = 64.  Halves of 64 normally
// distributed elements hardly ever lie more than two bits apart; the columns of U do
// while its rows grow (in the first pairs of an N(0,1) matrix), the rows of L do not.
constexpr int kOzApart = 2;
enum { kOzRowsApart = 0, kOzColsApart = 1 };  // flags

// Exponents of the halves; true if they lie apart.  !own: the larger one for both.
template <int kH>
__device__ __forceinline__ bool oz_half_exponents(const double (&x)[2 * kH], bool own, int (&e)[kH]) {
#pragma unroll
  for (int h = 0; h < kH; ++h) e[h] = oz_warp_max(max(oz_exponent(x[2 * h]), oz_exponent(x[2 * h + 1])));
  const bool apart = kH == 2 && abs(e[0] - e[kH - 1]) > kOzApart;
  if (kH == 2 && !own) e[0] = e[kH - 1] = max(e[0], e[kH - 1]);
  return apart;
}

// Row i of M rows of L (row: its w <= 64 kH elements): As[p][i][k] (zero for k >= w),
// ea[h M + i].  One warp.
template <int kH>
__device__ __forceinline__ bool oz_split_row(const double* __restrict__ row, int i, int M, int w, bool own,
                                             __half* __restrict__ as, int* __restrict__ ea, int lane) {
  double x[2 * kH];
  int e[kH];
#pragma unroll
  for (int q = 0; q < 2 * kH; ++q) x[q] = lane + 32 * q < w ? row[lane + 32 * q] : 0.0;
  const bool apart = oz_half_exponents<kH>(x, own, e);
#pragma unroll
  for (int h = 0; h < kH; ++h) {
    oz_emit_row(x[2 * h], x[2 * h + 1], e[h], as + ((int64_t)i * kH + h) * kOzK, (int64_t)M * kH * kOzK, lane);
    if (lane == 0) ea[(int64_t)h * M + i] = e[h] == kOzZero ? 0 : e[h];
  }
  return apart;
}
// Columns j0 .. j0 + 31 of N columns of U (w <= 64 kH rows of a): Bs[p][j][k] (the
// transpose; zero for k >= w), eb[h N + j].  A CTA of 256 threads stages 64 kH x 32
// elements through shared memory (coalesced reads along the rows), then each warp
// splits four columns.
template <int kH>
__device__ __forceinline__ bool oz_split_cols(double (&tile)[kH * kOzK][33], const double* __restrict__ a, int64_t lda,
                                              int w, int j0, int N, bool own, __half* __restrict__ bs,
                                              int* __restrict__ eb) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 8
  for (int k = warp; k < kH * kOzK; k += 8) {
    const int j = j0 + lane;
    tile[k][lane] = (k < w && j < N) ? a[(int64_t)k * lda + j] : 0.0;
  }
  __syncthreads();
  bool apart = false;
  for (int jj = warp; jj < 32; jj += 8) {
    const int j = j0 + jj;
    if (j >= N) break;
    double x[2 * kH];
    int e[kH];
#pragma unroll
    for (int q = 0; q < 2 * kH; ++q) x[q] = tile[lane + 32 * q][jj];
    apart |= oz_half_exponents<kH>(x, own, e);
#pragma unroll
    for (int h = 0; h < kH; ++h) {
      oz_emit_row(x[2 * h], x[2 * h + 1], e[h], bs + ((int64_t)j * kH + h) * kOzK, (int64_t)N * kH * kOzK, lane);
      if (lane == 0) eb[(int64_t)h * N + j] = e[h] == kOzZero ? 0 : e[h];
    }
  }
  return apart;
}

// kH = 2: raise the flags (cleared before).
template <int kH>
__global__ void __launch_bounds__(256) oz_split_rows_kernel(const double* __restrict__ l, int64_t ldl, int M, int w,
                                                            __half* __restrict__ as, int* __restrict__ ea,
                                                            int* flags) {
  const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (i >= M) return;
  if (oz_split_row<kH>(l + (int64_t)i * ldl, i, M, w, false, as, ea, lane) && lane == 0) flags[kOzRowsApart] = 1;
}
template <int kH>
__global__ void __launch_bounds__(256) oz_split_cols_kernel(const double* __restrict__ u, int64_t ldu, int w, int N,
                                                            __half* __restrict__ bs, int* __restrict__ eb,
                                                            int* flags) {
  __shared__ double tile[kH * kOzK][33];
  if (oz_split_cols<kH>(tile, u, ldu, w, blockIdx.x * 32, N, false, bs, eb) && (threadIdx.x & 31) == 0)
    flags[kOzColsApart] = 1;
}
// Both operands of K = 128 again, an exponent a half, if both flags are up.
__global__ void __launch_bounds__(256) oz_resplit_kernel(const double* __restrict__ l, int64_t ldl, int M,
                                                         const double* __restrict__ u, int64_t ldu, int N, int w,
                                                         __half* __restrict__ as, int* __restrict__ ea,
                                                         __half* __restrict__ bs, int* __restrict__ eb,
                                                         const int* __restrict__ flags) {
  __shared__ double tile[2 * kOzK][33];
  if (flags[kOzRowsApart] == 0 || flags[kOzColsApart] == 0) return;
  for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < M; i += gridDim.x * 8)
    oz_split_row<2>(l + (int64_t)i * ldl, i, M, w, true, as, ea, threadIdx.x & 31);
  for (int j0 = blockIdx.x * 32; j0 < N; j0 += gridDim.x * 32) {
    __syncthreads();  // the tile's last readers
    oz_split_cols<2>(tile, u, ldu, w, j0, N, true, bs, eb);
  }
}

// ---------------------------------------------------------------------------
// Products and combine.
// ---------------------------------------------------------------------------

__device__ __forceinline__ void oz_abort(DeviceStatus* st, int* s_abort) {
  atomicCAS(&st->error, kDevOk, kDevBarrierTimeout);
  atomicExch(&st->abort, 1);
  atomicExch(s_abort, 1);
}

// Bounded mbarrier wait that also gives up once the CTA's abort flag is up.  The
// timer is read only when the first try fails: the read takes longer than the try.
__device__ __forceinline__ bool oz_try(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(bar), "r"(parity)
      : "memory");
  return done != 0u;
}
__device__ __noinline__ bool oz_wait_long(unsigned bar, unsigned parity, unsigned long long limit_ns,
                                          const int* s_abort) {
  const unsigned long long t0 = global_timer_ns();
  for (unsigned spins = 0;; ++spins) {
    if (oz_try(bar, parity)) return true;
    if ((spins & 15u) == 15u) {
      if (*reinterpret_cast<const volatile int*>(s_abort)) return false;
      if (global_timer_ns() - t0 > limit_ns) return false;
    }
  }
}
__device__ __forceinline__ bool oz_wait(unsigned bar, unsigned parity, unsigned long long limit_ns,
                                        const int* s_abort) {
  return oz_try(bar, parity) || oz_wait_long(bar, parity, limit_ns, s_abort);
}

__device__ __forceinline__ void oz_tma3d(unsigned dst, const CUtensorMap* map, int x, int y, int z, unsigned bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar)
      : "memory");
}

// TMEM load of one warp: its 32 lanes, 16 consecutive 32-bit columns from taddr
// (lane field in bits 16+).
__device__ __forceinline__ void tmem_ld16(unsigned taddr, unsigned (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
// One M = 128, K = 16 MMA on K-major operands in 128-byte swizzled rows; the
// descriptors' low words (address and leading offset) vary, the high word (8-row
// groups 1024 bytes apart, version, swizzle) does not.
__device__ __forceinline__ void oz_mma(unsigned acc, unsigned a_lo, unsigned b_lo, unsigned idesc, unsigned accumulate) {
  constexpr unsigned hi = (1024u >> 4) | (1u << 14) | (2u << 29);
  asm volatile(
      "{\n .reg .pred p;\n .reg .b64 da, db;\n mov.b64 da, {%1, %5};\n mov.b64 db, {%2, %5};\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}\n" ::"r"(acc),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(hi));
}

// Instruction descriptor: D FP32 (bit 4), A and B FP16 (format 0), both K-major,
// M = 128, N = 64 per piece.
__device__ __forceinline__ constexpr unsigned oz_idesc(int pieces) {
  return (1u << 4) | ((unsigned)(pieces * kOzBM >> 3) << 17) | ((unsigned)(kOzBN >> 4) << 24);
}
// One k-step of a U piece against `pieces` stacked L pieces, added to as many
// accumulators from `acc` on (N = 256 at most in one MMA).
__device__ __forceinline__ void oz_mma_range(unsigned acc, unsigned a_lo, unsigned b_lo, int pieces) {
  if (pieces > 4) {
    oz_mma(acc, a_lo, b_lo, oz_idesc(4), 1u);
    oz_mma(acc + 4 * kOzBM, a_lo, b_lo + 4 * (kOzLBytes >> 4), oz_idesc(pieces - 4), 1u);
  } else {
    oz_mma(acc, a_lo, b_lo, oz_idesc(pieces), 1u);
  }
}

__device__ __forceinline__ void oz_commit(unsigned bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// The products of one K half of a tile, q = 6 .. 0: piece q adds to the groups from
// q up, so each step needs one more accumulator, in the order the epilogue frees
// them.  Called by the whole MMA warp; one lane issues.  Unrolled: what a product
// costs the warp besides the instruction itself has to stay below the tensor
// pipe's 128 cycles, so that descriptors and addresses are constants off a base.
template <int kHalf>
__device__ __forceinline__ bool oz_mma_half(unsigned tmem, unsigned u_lo, unsigned l_lo, bool leader, unsigned acc_empty,
                                            unsigned u_full, unsigned u_empty, unsigned acc_parity, unsigned u_parity,
                                            unsigned long long limit, const int* s_abort) {
  const unsigned db = l_lo + (unsigned)(kHalf * kOzSlices * (kOzLBytes >> 4));
#pragma unroll
  for (int q = kOzSlices - 1; q >= 0; --q) {
    if (kHalf == 0 || q == kOzSlices - 1) {
      if (!__all_sync(0xffffffffu, oz_wait(acc_empty + 8u * (unsigned)(kHalf == 0 ? q : kOzGroups), acc_parity, limit, s_abort)))
        return false;
    }
    if (!__all_sync(0xffffffffu, oz_wait(u_full + 8u * (unsigned)q, u_parity, limit, s_abort))) return false;
    asm volatile("tcgen05.fence::after_thread_sync;");
    const unsigned da = u_lo + (unsigned)(q * (kOzUBytes >> 4));
    const unsigned acc = tmem + (unsigned)(q * kOzBM);
    if (leader) {
#pragma unroll
      for (int ks = 0; ks < kOzK / 16; ++ks) {
        if (kHalf == 0) {
          // Group q's accumulator starts here (its first k-step alone).
          if (ks == 0) {
            oz_mma(acc, da, db, oz_idesc(1), 0u);
            if (q < kOzSlices - 1) oz_mma_range(acc + kOzBM, da, db + (kOzLBytes >> 4), kOzSlices - 1 - q);
          } else {
            oz_mma_range(acc, da + 2 * ks, db + 2 * ks, kOzSlices - q);
          }
        } else {
          // Second half: group 6 has an accumulator of its own (its sum over both
          // halves could pass 2^24).
          if (q < kOzSlices - 1) oz_mma_range(acc, da + 2 * ks, db + 2 * ks, kOzSlices - 1 - q);
          oz_mma(tmem + (unsigned)(kOzGroups * kOzBM), da + 2 * ks,
                 db + 2 * ks + (unsigned)((kOzSlices - 1 - q) * (kOzLBytes >> 4)), oz_idesc(1),
                 q == kOzSlices - 1 && ks == 0 ? 0u : 1u);
        }
      }
      oz_commit(u_empty + 8u * (unsigned)q);
    }
  }
  return true;
}

// C - R 2^s for the fixed-point R = hi 2^32 + lo (s = ea + eb - 54); NaN
// when a row or column held Inf or NaN.  R 2^s is rounded to 53 bits (to
// nearest, ties to even, as a conversion of R would).  oz_combine_fast
// assembles it with 32-bit integer operations whenever it is a normal number
// and |R| >= 2^32, so the FP64 pipe runs one subtraction per element; the
// rest (zeros, small sums, subnormal and overflowing products, non-finite
// rows or columns) go through oz_combine, rarely.
__device__ __noinline__ double oz_combine_rare(long long R, int s, double c) {
  const unsigned long long neg = R < 0 ? (1ull << 63) : 0ull;
  const unsigned long long u = R < 0 ? 0ull - (unsigned long long)R : (unsigned long long)R;
  if (u == 0) return __dsub_rn(c, 0.0);
  const int lz = __clzll((long long)u);
  const unsigned long long un = u << lz;
  unsigned long long m = un >> 11;
  const unsigned rem = (unsigned)(un & 0x7FF);
  int t = 63 - lz;
  m += (rem > 0x400u || (rem == 0x400u && (m & 1))) ? 1ull : 0ull;
  if (m >> 53) {
    m >>= 1;
    ++t;
  }
  const int E = t + s + 1023;
  const unsigned long long frac = m & 0xFFFFFFFFFFFFFull;
  if (E >= 1 && E <= 2046)
    return __dsub_rn(c, __longlong_as_double((long long)(neg | ((unsigned long long)E << 52) | frac)));
  if (E > 2046) return __dsub_rn(c, __longlong_as_double((long long)(neg | 0x7FF0000000000000ull)));
  // Below the normal range: the 53-bit value at exponent -1000 (exact), then
  // one multiplication by 2^d rounds it once, to the subnormal grid.
  const int d = E - 23;  // the value is (that number) x 2^d, d < -22
  if (d < -1074) return __dsub_rn(c, __longlong_as_double((long long)neg));
  const double mid = __longlong_as_double((long long)(neg | (23ull << 52) | frac));
  const double p2 = d >= -1022 ? __longlong_as_double((long long)(d + 1023) << 52)
                               : __longlong_as_double((long long)(1ull << (d + 1074)));
  return __dsub_rn(c, __dmul_rn(mid, p2));
}

// The common case of oz_combine: |R| >= 2^32, and an s for which every such R gives
// a normal number (kOzMinScale .. kOzMaxScale); s20 = s 2^20 (mod 2^32).  The
// words of R 2^s are |R| normalised to 53 bits with the leading one left in
// place: it adds one to the exponent field below it, and a rounding that carries
// out of the 53 bits adds another, so the rounding is one addition with carry.
// Returns false, leaving c alone, when the element needs oz_combine.
constexpr int kOzMinScale = 1 - 1023 - 32, kOzMaxScale = 2046 - 1023 - 64;
__device__ __forceinline__ bool oz_combine_fast(unsigned hi, unsigned lo, unsigned s20, double& c) {
  const unsigned sgn = (unsigned)((int)hi >> 31);  // 0 or ~0
  unsigned ul, uh;                                 // |R| < 2^62
  asm("{\n sub.cc.u32 %0, %2, %4;\n subc.u32 %1, %3, %4;\n}\n" : "=&r"(ul), "=r"(uh) : "r"(lo ^ sgn), "r"(hi ^ sgn), "r"(sgn));
  const int lz = __clz((int)uh);
  const unsigned nh = __funnelshift_l(ul, uh, lz);  // leading one at bit 31 (when uh != 0)
  const unsigned nl = ul << lz;
  const unsigned ml = __funnelshift_r(nl, nh, 11);
  // Round to nearest even: the 11 bits below, plus the last bit kept, above one half.
  const unsigned x = (nl & 0x7FFu) + (ml & 1u);
  const unsigned eh = s20 + ((unsigned)(62 + 1023) << 20) - ((unsigned)lz << 20) + (nh >> 11);
  unsigned t, dl, dh;
  asm("{\n add.cc.u32 %0, %3, 0xfffffbff;\n addc.cc.u32 %1, %4, 0;\n addc.u32 %2, %5, 0;\n}\n"
      : "=&r"(t), "=&r"(dl), "=r"(dh)
      : "r"(x), "r"(ml), "r"(eh));
  if (uh == 0u) return false;
  c = __dsub_rn(c, __hiloint2double((int)(dh | (sgn & 0x80000000u)), (int)dl));
  return true;
}

// Splitting an exact integer x, |x| < 2^30 in FP32, at its low 8 bits: returns the
// multiple of 256 nearest to x; lo = the rest, -128 .. 128.
__device__ __forceinline__ float oz_carry(float x, float& lo) {
  const float q = __fsub_rn(__fadd_rn(x, 3221225472.0f), 3221225472.0f);  // 1.5 2^31: an ulp of 256
  lo = __fsub_rn(x, q);
  return q;
}
// x 2^0 as the low bits of an integer (0x4B400000 + x), |x| < 2^22.
__device__ __forceinline__ unsigned oz_int_bits(float x) { return __float_as_uint(__fadd_rn(x, 12582912.0f)); }

__device__ __forceinline__ double oz_combine(unsigned hi, unsigned lo, int ea_i, int eb_j, double c) {
  if (ea_i >= kOzNonFinite || eb_j >= kOzNonFinite) return __longlong_as_double(0x7ff8000000000000ll);
  return oz_combine_rare((long long)(((unsigned long long)hi << 32) | lo), ea_i + eb_j - (kOzFrac + 16), c);
}

__global__ void __launch_bounds__(kOzThreads, 1)
    oz_gemm_kernel(const __grid_constant__ CUtensorMap tmL, const __grid_constant__ CUtensorMap tmU, int halves,
                   double* __restrict__ c, int64_t ldc, int M, int N, const int* __restrict__ ea,
                   const int* __restrict__ eb, const int* __restrict__ flags, DeviceStatus* st) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sU = base;                                  // streamed: the U pieces of each tile and K half
  unsigned char* sL = base + (size_t)kOzSlices * kOzUBytes;  // resident: the L pieces of the row block
  __shared__ __align__(8) unsigned long long l_full, l_empty, u_full[kOzSlices], u_empty[kOzSlices],
      acc_full, acc_empty[kOzAccs], mma_done;
  __shared__ unsigned tmem_base;
  __shared__ int s_abort, s_l_issued, s_l_consumed, s_u_issued;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned long long limit = st->timeout_ns;
  // Two halves on exponents of their own: each tile in two passes of K = 64.
  const int passes = halves == 2 && flags[kOzRowsApart] != 0 && flags[kOzColsApart] != 0 ? 2 : 1;
  const bool joint = halves == 2 && passes == 1;
  const int tiles_j = (N + kOzBN - 1) / kOzBN;
  const int tiles = tiles_j * ((M + kOzBM - 1) / kOzBM);
  const int t_begin = (int)((int64_t)blockIdx.x * tiles / gridDim.x);
  const int t_end = (int)((int64_t)(blockIdx.x + 1) * tiles / gridDim.x);

  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&l_full)));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&l_empty)));
    for (int p = 0; p < kOzSlices; ++p) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&u_full[p])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&u_empty[p])));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&acc_full)));
    for (int g = 0; g < kOzAccs; ++g)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&acc_empty[g])), "r"(kOzEpiWarps));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mma_done)));
    s_abort = 0;
    s_l_issued = s_l_consumed = s_u_issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;");
    asm volatile("fence.proxy.async.shared::cta;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const unsigned tmem = tmem_base;

  if (warp == 0) {
    if (lane == 0) {
      // Producer.  U pieces go in the order the MMAs free them (6 .. 0).
      int cur_ib = -1, nl = 0, use = 0;
      bool ok = true;
      for (int t = t_begin; t < t_end && ok; ++t) {
        if (*reinterpret_cast<volatile int*>(&s_abort)) break;
        const int ib = t / tiles_j, jb = t - ib * tiles_j;
        if (ib != cur_ib) {
          // The previous row block's pieces are free once its last MMAs end.
          if (nl > 0 && !oz_wait(smem_u32(&l_empty), (unsigned)((nl - 1) & 1), limit, &s_abort)) {
            ok = false;
            break;
          }
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&l_full)),
                       "r"((unsigned)(halves * kOzSlices * kOzLBytes))
                       : "memory");
          for (int h = 0; h < halves; ++h)
            for (int p = kOzSlices - 1; p >= 0; --p)
              oz_tma3d(smem_u32(sL + (h * kOzSlices + p) * kOzLBytes), &tmL, h * kOzK, ib * kOzBM, p,
                       smem_u32(&l_full));
          s_l_issued = ++nl;
          cur_ib = ib;
        }
        for (int h = 0; h < halves && ok; ++h, ++use) {
          for (int q = kOzSlices - 1; q >= 0; --q) {
            if (!oz_wait(smem_u32(&u_empty[q]), (unsigned)(use & 1) ^ 1u, limit, &s_abort)) {
              ok = false;
              break;
            }
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&u_full[q])),
                         "r"((unsigned)kOzUBytes)
                         : "memory");
            oz_tma3d(smem_u32(sU + q * kOzUBytes), &tmU, h * kOzK, jb * kOzBN, q, smem_u32(&u_full[q]));
            ++s_u_issued;
          }
        }
      }
      if (!ok) oz_abort(st, &s_abort);
    }
  } else if (warp == 1) {
    // MMA issuer: D[j][i] += sum_k U^T_q[j][k] L_p[i][k]: TMEM lanes are columns of C.
    // The whole warp runs the loop, so its addresses and descriptors stay in
    // uniform registers, which the MMAs take them from; one lane issues.
    // U piece q against the stacked L pieces 0, 1, .. is one product with N = 64 a
    // piece whose columns are the accumulators of groups q, q + 1, ..: 10 MMAs a
    // k-step instead of 28, each of them long enough for the pipe (an MMA of N = 64
    // takes as long as one of N = 128: 128 cycles with its operands from shared
    // memory).
    const bool leader = lane == 0;
    const unsigned u_lo = (smem_u32(sU) >> 4) | (1u << 16), l_lo = (smem_u32(sL) >> 4) | (1u << 16);
    int cur_ib = -1, nl = 0, tc = 0, use = 0;
    bool ok = true;
    // The passes as a constant: with a count read from memory a factorization of n =
    // 16384 takes 145.2 ms instead of 141.6.
    auto tiles_of = [&](auto passes_constant) {
      constexpr int kPasses = decltype(passes_constant)::value;
      for (int t = t_begin; t < t_end && ok; ++t) {
        const int ib = t / tiles_j;
        if (ib != cur_ib) {
          ok = __all_sync(0xffffffffu, oz_wait(smem_u32(&l_full), (unsigned)(nl & 1), limit, &s_abort));
          if (!ok) break;
          ++nl;
          if (leader) s_l_consumed = nl;
          cur_ib = ib;
        }
        for (int h = 0; h < kPasses; ++h, ++tc) {
          ok = oz_mma_half<0>(tmem, u_lo, l_lo + (unsigned)(h * kOzSlices * (kOzLBytes >> 4)), leader,
                              smem_u32(acc_empty), smem_u32(u_full), smem_u32(u_empty), (unsigned)(tc & 1) ^ 1u,
                              (unsigned)(use & 1), limit, &s_abort);
          ++use;
          if (ok && kPasses == 1 && halves == 2) {
            ok = oz_mma_half<1>(tmem, u_lo, l_lo, leader, smem_u32(acc_empty), smem_u32(u_full), smem_u32(u_empty),
                                (unsigned)(tc & 1) ^ 1u, (unsigned)(use & 1), limit, &s_abort);
            ++use;
          }
          if (!ok) break;
          if (leader) {
            oz_commit(smem_u32(&acc_full));
            const bool block_ends = (t + 1 >= t_end) || ((t + 1) / tiles_j != ib);
            if (block_ends && h + 1 == kPasses) oz_commit(smem_u32(&l_empty));
          }
          __syncwarp();
        }
      }
    };
    if (passes == 1)
      tiles_of(std::integral_constant<int, 1>());
    else
      tiles_of(std::integral_constant<int, 2>());
    if (leader) {
      if (!ok) oz_abort(st, &s_abort);
      // Arrives once every MMA issued above has completed.
      oz_commit(smem_u32(&mma_done));
      mbar_wait(smem_u32(&mma_done), 0u, limit);
    }
    __syncwarp();
  } else {
    // Epilogue: warp w owns TMEM lanes 32 (w % 4) .. + 31 (32 columns of the
    // tile) and 16 of its 64 rows, (w - 2) / 4.  Its thread keeps its column's
    // 16 sums in two registers each.
    // Fold.  R = floor(sum_G T_G 2^(38-8G)), exactly.  Converting each T_G and
    // shifting 64-bit sums costs a conversion (8 cycles of a quarter's unit) and
    // three integer instructions (2 cycles each) a group; FP32 additions run at full
    // rate and are exact here, so the groups' low 8 bits are split off in FP32 and
    // the rest carried to the next group: with q_G the carry out of group G, and
    // lo_G its digit (-128 .. 128),
    //   x_G = T_G + q_(G+1) / 256 = q_G + lo_G,
    //   R = T_0 2^38 + x_1 2^30 + lo_2 2^22 + lo_3 2^14 + floor((lo_4 2^16 + lo_5 2^8 + lo_6) / 2^10),
    // three conversions in all.  |T_G| < 2^24 - 2^20 for G <= 4, so that x_G is
    // exact; T_5 can come within 2^15 of 2^24 (K = 128) and is split before it
    // takes the carry, as are the two sums of group 6.
    const int quarter = warp & 3, rq = (warp - 2) >> 2;
    const unsigned lane_base = tmem + ((unsigned)(quarter * 32) << 16) + (unsigned)(rq * kOzRows);
    for (int tc = 0; tc < (t_end - t_begin) * passes; ++tc) {
      const int t = t_begin + (tc >> (passes - 1)), h = tc & (passes - 1);
      const int ib = t / tiles_j, jb = t - ib * tiles_j;
      const int col = jb * kOzBN + quarter * 32 + lane;
      const int row0 = ib * kOzBM + rq * kOzRows;
      const bool col_ok = col < N;
      {
        // Bring this warp's 16 rows x 32 columns of C into L2 while the tile's
        // products run (lane r: half of row r % 16, 128 bytes).
        const int c0 = jb * kOzBN + quarter * 32 + (lane >> 4) * 16, rr = row0 + (lane & 15);
        if (c0 < N && rr < M) asm volatile("prefetch.global.L2 [%0];" ::"l"(c + (int64_t)rr * ldc + c0));
      }
      const bool got = oz_wait(smem_u32(&acc_full), (unsigned)(tc & 1), limit, &s_abort);
      if (!__all_sync(0xffffffffu, got)) {
        if (lane == 0) oz_abort(st, &s_abort);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      float xq[kOzRows], lo[kOzRows];
      unsigned rh[kOzRows], rl[kOzRows];
      auto load = [&](int acc, unsigned (&tv)[kOzRows]) {
        tmem_ld16(lane_base + (unsigned)(acc * kOzBM), tv);
        asm volatile("tcgen05.wait::ld.sync.aligned;");
        // This warp has read the accumulator: the MMA warp may reuse it.
        asm volatile("tcgen05.fence::before_thread_sync;");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&acc_empty[acc]));
      };
      {
        unsigned tv[kOzRows];
        load(6, tv);
#pragma unroll
        for (int r = 0; r < kOzRows; ++r) xq[r] = oz_carry(__uint_as_float(tv[r]), lo[r]);
      }
      if (joint) {
        unsigned tv[kOzRows];
        load(kOzGroups, tv);
#pragma unroll
        for (int r = 0; r < kOzRows; ++r) {
          float lo2;
          xq[r] = __fadd_rn(xq[r], oz_carry(__uint_as_float(tv[r]), lo2));
          lo[r] = __fadd_rn(lo[r], lo2);
        }
      }
      {
        unsigned tv[kOzRows];
        load(5, tv);
#pragma unroll
        for (int r = 0; r < kOzRows; ++r) {
          float d, e;
          const float qa = oz_carry(__uint_as_float(tv[r]), d);
          const float qb = oz_carry(__fmaf_rn(xq[r], 0.00390625f, d), e);
          xq[r] = __fadd_rn(qa, qb);
          lo[r] = __fmaf_rn(e, 256.0f, lo[r]);
        }
      }
      {
        unsigned tv[kOzRows];
        load(4, tv);
#pragma unroll
        for (int r = 0; r < kOzRows; ++r) {
          float d;
          xq[r] = oz_carry(__fmaf_rn(xq[r], 0.00390625f, __uint_as_float(tv[r])), d);
          rl[r] = (unsigned)(__float2int_rn(__fmaf_rn(d, 65536.0f, lo[r])) >> 10);
        }
      }
#pragma unroll
      for (int g = 3; g >= 2; --g) {
        unsigned tv[kOzRows];
        load(g, tv);
#pragma unroll
        for (int r = 0; r < kOzRows; ++r) {
          float d;
          xq[r] = oz_carry(__fmaf_rn(xq[r], 0.00390625f, __uint_as_float(tv[r])), d);
          rl[r] += oz_int_bits(d) << (kOzFrac - 8 * g);  // the bias is shifted out
        }
      }
      {
        unsigned tv[kOzRows];
        load(1, tv);
#pragma unroll
        for (int r = 0; r < kOzRows; ++r) {
          const int x1 = __float2int_rn(__fmaf_rn(xq[r], 0.00390625f, __uint_as_float(tv[r])));
          const unsigned h = (unsigned)((x1 >> 2) + ((int)rl[r] >> 31));
          asm("{\n add.cc.u32 %0, %2, %3;\n addc.u32 %1, %4, 0;\n}\n"
              : "=&r"(rl[r]), "=r"(rh[r])
              : "r"(rl[r]), "r"((unsigned)x1 << 30), "r"(h));
        }
      }
      {
        unsigned tv[kOzRows];
        load(0, tv);
#pragma unroll
        for (int r = 0; r < kOzRows; ++r)
          rh[r] += (unsigned)__float2int_rn(__uint_as_float(tv[r])) << (kOzFrac - 32);
      }
      // C -= the sums: thread = one column of C, its rows in chunks of 4;
      // a warp's loads and stores of one row are 32 consecutive doubles.
      // Lane r holds the exponent of row r.  Elements the fast path declines
      // (rare) are redone, warp-uniformly, by the general path.
      const int eb_j = col_ok ? eb[(int64_t)h * N + col] : 0;
      const int my_ea = lane < kOzRows && row0 + lane < M ? ea[(int64_t)h * M + row0 + lane] : 0;
      const int s_col = eb_j >= kOzNonFinite ? (1 << 24) : eb_j - (kOzFrac + 16);
      const int s_row = my_ea >= kOzNonFinite ? (1 << 24) : my_ea;
      const bool in_range =
          __reduce_min_sync(0xffffffffu, s_col) + __reduce_min_sync(0xffffffffu, s_row) >= kOzMinScale &&
          __reduce_max_sync(0xffffffffu, s_col) + __reduce_max_sync(0xffffffffu, s_row) <= kOzMaxScale;
      const bool whole = (jb * kOzBN + quarter * 32 + 32 <= N) && (row0 + kOzRows <= M);  // warp-uniform
      double* cptr = c + (int64_t)row0 * ldc + (col_ok ? col : 0);
      constexpr int kC = 4;
#pragma unroll
      for (int cc = 0; cc < kOzRows / kC; ++cc) {
        double cv[kC];
#pragma unroll
        for (int r = 0; r < kC; ++r)
          cv[r] = (whole || (col_ok && row0 + kC * cc + r < M)) ? __ldcs(cptr + (int64_t)r * ldc) : 0.0;
        unsigned declined = in_range ? 0u : (1u << kC) - 1u;
        if (in_range) {
#pragma unroll
          for (int r = 0; r < kC; ++r) {
            const int k = kC * cc + r;
            const unsigned s20 = (unsigned)(s_col + __shfl_sync(0xffffffffu, s_row, k)) << 20;
            if (!oz_combine_fast(rh[k], rl[k], s20, cv[r])) declined |= 1u << r;
          }
        }
        if (__any_sync(0xffffffffu, declined != 0u)) {
#pragma unroll
          for (int r = 0; r < kC; ++r) {
            const int k = kC * cc + r;
            const int ea_i = __shfl_sync(0xffffffffu, my_ea, k);
            if (declined & (1u << r)) cv[r] = oz_combine(rh[k], rl[k], ea_i, eb_j, cv[r]);
          }
        }
#pragma unroll
        for (int r = 0; r < kC; ++r)
          if (whole || (col_ok && row0 + kC * cc + r < M)) __stcs(cptr + (int64_t)r * ldc, cv[r]);
        cptr += kC * ldc;
        asm volatile("" ::: "memory");  // keep the chunks' loads from being hoisted together
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0 && s_abort) {
    // Copies issued but never consumed must land before the CTA exits.
    if (s_l_issued > s_l_consumed) mbar_wait(smem_u32(&l_full), (unsigned)((s_l_issued - 1) & 1), limit);
    // U pieces: every issued piece's barrier completes once its bytes land
    // (issue order 6 .. 0 per tile and half).
    for (int p = 0; p < kOzSlices; ++p) {
      const int uses = s_u_issued / kOzSlices + (kOzSlices - 1 - p < s_u_issued % kOzSlices ? 1 : 0);
      if (uses > 0) mbar_wait(smem_u32(&u_full[p]), (unsigned)((uses - 1) & 1), limit);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
static size_t oz_round(size_t b) { return (b + 1023) / 1024 * 1024; }

// Workspace layout for an M x N product over K = 64 * halves: A slices
// [7][M][K], B slices [7][N][K], exponents ea[halves][M], eb[halves][N], two flags.
struct OzWs {
  __half* as;
  __half* bs;
  int* ea;
  int* eb;
  int* flags;
};
static OzWs oz_layout(void* ws, int M, int N, int halves = 1) {
  const size_t kb = (size_t)kOzSlices * kOzK * 2 * halves;
  char* p = static_cast<char*>(ws);
  OzWs w;
  w.as = reinterpret_cast<__half*>(p);
  p += oz_round(kb * M);
  w.bs = reinterpret_cast<__half*>(p);
  p += oz_round(kb * N);
  w.ea = reinterpret_cast<int*>(p);
  p += oz_round((size_t)M * halves * 4);
  w.eb = reinterpret_cast<int*>(p);
  p += oz_round((size_t)N * halves * 4);
  w.flags = reinterpret_cast<int*>(p);
  return w;
}

size_t ozaki_workspace_bytes(int m, int n) {
  const size_t kb = (size_t)kOzSlices * kOzK * 2 * kOzMaxHalves;
  return oz_round(kb * m) + oz_round(kb * n) + oz_round((size_t)m * kOzMaxHalves * 4) +
         oz_round((size_t)n * kOzMaxHalves * 4) + oz_round(2 * sizeof(int));
}

bool ozaki_available(luhot_ctx* ctx) { return kOzSmem <= (size_t)ctx->max_smem_optin && encode_fn() != nullptr; }

// Slices [7][rows][K] FP16, K = 64 * halves, as a 3-D tensor map (k, row, slice)
// with boxes of 64 x box_rows x 1 (128-byte rows, 128-byte swizzle); rows past
// `rows` read as zero.
static int make_slice_map(luhot_ctx* ctx, CUtensorMap* map, void* ptr, int rows, int box_rows, int halves) {
  EncodeTiledFn enc = encode_fn();
  if (!enc) return set_error(ctx, LUHOT_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is unavailable");
  const cuuint64_t kk = (cuuint64_t)kOzK * halves;
  cuuint64_t dims[3] = {kk, (cuuint64_t)rows, (cuuint64_t)kOzSlices};
  cuuint64_t strides[2] = {kk * 2, (cuuint64_t)rows * kk * 2};
  cuuint32_t box[3] = {(cuuint32_t)kOzK, (cuuint32_t)box_rows, 1};
  cuuint32_t estr[3] = {1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, ptr, dims, strides, box, estr,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return set_error(ctx, LUHOT_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string((int)r));
  return LUHOT_OK;
}

// C (M x N, ldc) -= the product of the slices in `w`; one persistent launch.
static int oz_launch_gemm(luhot_ctx* ctx, const OzWs& w, int halves, double* c, int64_t ldc, int M, int N,
                          cudaStream_t stream) {
  CUtensorMap tmL, tmU;
  int rc = make_slice_map(ctx, &tmL, w.as, M, kOzBM, halves);
  if (!rc) rc = make_slice_map(ctx, &tmU, w.bs, N, kOzBN, halves);
  if (rc) return rc;
  const int tiles = ((M + kOzBM - 1) / kOzBM) * ((N + kOzBN - 1) / kOzBN);
  LUHOT_CUDA_TRY(ctx, allow_max_dynamic_smem(oz_gemm_kernel));
  const int cap = ctx->tc_grid_cap > 0 ? ctx->tc_grid_cap : ctx->num_sms;
  oz_gemm_kernel<<<std::min(tiles, cap), kOzThreads, kOzSmem, stream>>>(tmL, tmU, halves, c, ldc, M, N, w.ea, w.eb,
                                                                      w.flags, ctx->d_status);
  LUHOT_CUDA_TRY(ctx, cudaGetLastError());
  return LUHOT_OK;
}

SplitOut ozaki_split_out(void* ws, int r1, int M, int N) {
  const OzWs lay = oz_layout(ws, M, N);
  SplitOut s;
  s.as = lay.as;
  s.ea = lay.ea;
  s.r1 = r1;
  s.M = M;
  s.bs = lay.bs;
  s.eb = lay.eb;
  return s;
}

int ozaki_update_split(luhot_ctx* ctx, double* a, int64_t lda, int w, int r1, int m, int c1, int n, void* ws,
                       cudaStream_t stream) {
  const int M = m - r1, N = n - c1;
  const OzWs lay = oz_layout(ws, M, N);
  prof_begin(ctx, kProfGemm);
  int rc = oz_launch_gemm(ctx, lay, 1, a + (int64_t)r1 * lda + c1, lda, M, N, stream);
  // algorithmic work: 2MNK FP64 flops; bytes: C read + written, the slices read once
  prof_end(ctx, kProfGemm, 2.0 * M * N * w,
           (double)M * N * 16 + (double)(M + N) * kOzK * kOzSlices * 2 + (double)(M + N) * 4);
  return rc;
}

int ozaki_product(luhot_ctx* ctx, const double* l, int64_t ldl, const double* u, int64_t ldu, int w, double* c,
                  int64_t ldc, int M, int N, void* ws, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || w <= 0) return LUHOT_OK;
  if (w > kOzMaxHalves * kOzK) return set_error(ctx, LUHOT_ERR_INVALID_ARG, "ozaki_product: more than 128 columns");
  const int halves = w > kOzK ? 2 : 1;
  const OzWs lay = oz_layout(ws, M, N, halves);
  const double slice_bytes = (double)halves * kOzK * kOzSlices * 2;
  if (halves == 2) LUHOT_CUDA_TRY(ctx, cudaMemsetAsync(lay.flags, 0, 2 * sizeof(int), stream));
  prof_begin(ctx, kProfOther);
  if (halves == 2)
    oz_split_rows_kernel<2><<<(M + 7) / 8, 256, 0, stream>>>(l, ldl, M, w, lay.as, lay.ea, lay.flags);
  else
    oz_split_rows_kernel<1><<<(M + 7) / 8, 256, 0, stream>>>(l, ldl, M, w, lay.as, lay.ea, nullptr);
  prof_end(ctx, kProfOther, 0.0, M * (w * 8.0 + slice_bytes));
  prof_begin(ctx, kProfOther);
  if (halves == 2)
    oz_split_cols_kernel<2><<<(N + 31) / 32, 256, 0, stream>>>(u, ldu, w, N, lay.bs, lay.eb, lay.flags);
  else
    oz_split_cols_kernel<1><<<(N + 31) / 32, 256, 0, stream>>>(u, ldu, w, N, lay.bs, lay.eb, nullptr);
  prof_end(ctx, kProfOther, 0.0, N * (w * 8.0 + slice_bytes));
  if (halves == 2) {
    prof_begin(ctx, kProfOther);
    oz_resplit_kernel<<<ctx->num_sms, 256, 0, stream>>>(l, ldl, M, u, ldu, N, w, lay.as, lay.ea, lay.bs, lay.eb,
                                                        lay.flags);
    prof_end(ctx, kProfOther, 0.0, 0.0);
  }
  LUHOT_CUDA_TRY(ctx, cudaGetLastError());
  prof_begin(ctx, kProfGemm);
  int rc = oz_launch_gemm(ctx, lay, halves, c, ldc, M, N, stream);
  // algorithmic work: 2MNK FP64 flops; bytes: C read + written, the slices read once
  prof_end(ctx, kProfGemm, 2.0 * M * N * w, (double)M * N * 16 + (M + N) * (slice_bytes + 4.0));
  return rc;
}

int ozaki_update(luhot_ctx* ctx, double* a, int64_t lda, int k0, int w, int r1, int m, int c1, int n, void* ws,
                 cudaStream_t stream) {
  return ozaki_product(ctx, a + (int64_t)r1 * lda + k0, lda, a + (int64_t)k0 * lda + c1, lda, w,
                       a + (int64_t)r1 * lda + c1, lda, m - r1, n - c1, ws, stream);
}

}  // namespace luhot
