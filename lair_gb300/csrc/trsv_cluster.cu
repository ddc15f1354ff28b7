// Triangular sweep with given diagonal inverses: a cluster of four CTAs a block.
//
// op(A) x = b with op(A) triangular (A or A^T of a row-major LU factor), kNR
// right-hand sides a chain, in place.  The rows are cut into 64-row blocks; a
// cluster takes a (chain, block) by ticket in the order the sweep needs them, as
// in trsv.cu, so that it only waits for clusters that are already running.
//
// What bounds a sweep with few right-hand sides is its chain, the way from x(I-1)
// to x(I): the last off-diagonal tile and the diagonal inverse, two 64 x 64
// products of FP64, 2000 cycles each on one SM, and the publication of x(I).
//   - Each of the four CTAs has 16 of the block's rows, a quarter of that work.
//     The sums of the rows are exchanged through distributed shared memory
//     (cluster.cuh) between the two products.
//   - x(I) is published as words that carry the launch's epoch (two an FP64
//     value), which the readers poll themselves: no flag, no fence, and one trip to
//     L2 instead of two.
// Thread (row, right-hand side, part): 16 rows, 8 parts of 8 columns (4 of 16 for
// wide chains), one sum a thread, reduced over the parts at the end.  The next
// tile's elements and words are requested while the current tile is used.
// Every wait is bounded by the context's wait limit (LUHOT_ERR_TIMEOUT).
#include <algorithm>

#include "cluster.cuh"
#include "common.cuh"
#include "luhot_internal.h"
#include "trsv.cuh"

namespace luhot {

constexpr int kTB = 64;         // block rows (the diagonal-inverse blocks)
constexpr int kTCtas = 4;       // CTAs of a cluster
constexpr int kTRows = 16;      // rows of a CTA
constexpr int kTAhead = 3;      // tiles from memory to L2 ahead of their use

template <int kNR>
__host__ __device__ constexpr int tc_parts() {
  return kNR >= 4 ? 4 : 8;
}
template <int kNR>
__host__ __device__ constexpr int tc_threads() {
  return kTRows * kNR * tc_parts<kNR>();
}

// A published value: one (FP32) or two (FP64) words of 32 bits below the epoch.
template <typename T>
struct TcWord;
template <>
struct TcWord<double> {
  static constexpr int kWords = 2;
  __device__ static void load(const unsigned long long* p, unsigned long long (&v)[2]) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "l"(p) : "memory");
  }
  __device__ static bool ok(const unsigned long long (&v)[2], unsigned epoch) {
    return (unsigned)(v[0] >> 32) == epoch && (unsigned)(v[1] >> 32) == epoch;
  }
  __device__ static double value(const unsigned long long (&v)[2]) {
    return __hiloint2double((int)(unsigned)v[0], (int)(unsigned)v[1]);
  }
  __device__ static void store(unsigned long long* p, double x, unsigned epoch) {
    const unsigned long long tag = (unsigned long long)epoch << 32;
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(tag | (unsigned)__double2hiint(x)),
                 "l"(tag | (unsigned)__double2loint(x))
                 : "memory");
  }
  __device__ static unsigned long long bits(double x) { return (unsigned long long)__double_as_longlong(x); }
  __device__ static double from(unsigned long long b) { return __longlong_as_double((long long)b); }
};
template <>
struct TcWord<float> {
  static constexpr int kWords = 1;
  __device__ static void load(const unsigned long long* p, unsigned long long (&v)[1]) {
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v[0]) : "l"(p) : "memory");
  }
  __device__ static bool ok(const unsigned long long (&v)[1], unsigned epoch) { return (unsigned)(v[0] >> 32) == epoch; }
  __device__ static float value(const unsigned long long (&v)[1]) { return __uint_as_float((unsigned)v[0]); }
  __device__ static void store(unsigned long long* p, float x, unsigned epoch) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p),
                 "l"(((unsigned long long)epoch << 32) | __float_as_uint(x))
                 : "memory");
  }
  __device__ static unsigned long long bits(float x) { return __float_as_uint(x); }
  __device__ static float from(unsigned long long b) { return __uint_as_float((unsigned)b); }
};

template <typename T, typename TA, bool kLower, bool kTrans, int kNR>
__global__ void __launch_bounds__(tc_threads<kNR>())
    trsv_cluster_kernel(const TA* __restrict__ a, int64_t lda, T* x, int64_t ldx, int n, int nrhs, int nchain,
                        const T* __restrict__ dinv, unsigned long long* xt, unsigned epoch, int* ticket,
                        DeviceStatus* st) {
  using Word = TcWord<T>;
  constexpr int kParts = tc_parts<kNR>(), kLen = kTB / kParts, kW = Word::kWords;
  constexpr int kVals = kTB * kNR;  // values of a block
  static_assert(kVals <= tc_threads<kNR>(), "a thread polls one value at most");
  constexpr unsigned kFull = 0xffffffffu;
  __shared__ T xs[2][kVals];                   // x(J), [k][c]
  __shared__ unsigned long long sums[kVals];   // the block's sums, [row][c]
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int s_ticket;
  const int tid = threadIdx.x;
  const int rank = blockIdx.x & (kTCtas - 1);  // one-dimensional grid and clusters
  const int nblk = (n + kTB - 1) / kTB;
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cl_smem(&bar)));
    asm volatile("fence.mbarrier_init.release.cluster;");
    cl_expect(cl_smem(&bar), (unsigned)kVals * 8u);
    if (rank == 0) {
      const int t = atomicAdd(ticket, 1);
      for (int r = 0; r < kTCtas; ++r)
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cl_peer(cl_smem(&s_ticket), r)), "r"(t) : "memory");
    }
  }
  cl_sync();
  const int chain = s_ticket % nchain, t = s_ticket / nchain;
  x += chain * kNR;
  nrhs = min(kNR, nrhs - chain * kNR);
  xt += (size_t)chain * nblk * kVals * kW;
  const int I = kLower ? t : nblk - 1 - t;
  const int i0 = I * kTB;

  const int part = tid % kParts, c = tid / kParts % kNR, r = rank * kTRows + tid / (kParts * kNR);
  const int row = i0 + r;
  const bool on = row < n && c < nrhs;
  const int nupd = kLower ? I : nblk - 1 - I;  // blocks before I in sweep order
  auto block = [&](int s) { return kLower ? s : nblk - 1 - s; };
  auto load_tile = [&](int J, T(&v)[kLen]) {
#pragma unroll
    for (int e = 0; e < kLen; ++e) {
      const int k = J * kTB + part + kParts * e;
      v[e] = row < n && k < n ? static_cast<T>(kTrans ? a[(int64_t)k * lda + row] : a[(int64_t)row * lda + k]) : T(0);
    }
  };
  // This thread's value of x(J): index tid of the block's (beyond n or nrhs: zero).
  const bool polls = tid < kVals && tid % kNR < nrhs;
  auto word = [&](int J) { return xt + ((size_t)J * kVals + tid) * kW; };

  T d[kLen];  // this thread's part of the diagonal inverse's row
#pragma unroll
  for (int e = 0; e < kLen; ++e) {
    const int k = part + kParts * e;
    d[e] = dinv[(size_t)I * kTB * kTB + (kTrans ? k * kTB + r : r * kTB + k)];
  }
  T acc = on && part == 0 ? x[(int64_t)row * ldx + c] : T(0);
  T v[kLen];
  unsigned long long w[kW];
  bool ok = true;
  if (nupd > 0) {
    load_tile(block(0), v);
    if (polls) Word::load(word(block(0)), w);
  }
  for (int s = 0; s < nupd; ++s) {
    const int J = block(s);
    T xv = T(0);
    if (polls && J * kTB + tid / kNR < n) {
      unsigned long long t0 = 0;
      unsigned spins = 0;
      while (!Word::ok(w, epoch)) {
        Word::load(word(J), w);
        if ((++spins & 31u) == 0) {
          const unsigned long long now = global_timer_ns();
          if (t0 == 0) t0 = now;
          const bool late = now - t0 > st->timeout_ns;
          if (late) {
            atomicCAS(&st->error, kDevOk, kDevBarrierTimeout);
            atomicExch(&st->timeout_where, (unsigned long long)J);
            atomicExch(&st->abort, 1);
          }
          if (late || ld_relaxed_i32(&st->abort)) {
            ok = false;
            break;
          }
        }
      }
      xv = Word::value(w);
    }
    if (tid < kVals) xs[s & 1][tid] = xv;
    T nv[kLen];
    if (s + 1 < nupd) {
      load_tile(block(s + 1), nv);
      if (polls) Word::load(word(block(s + 1)), w);
    }
    if (kNR == 1 && s + kTAhead < nupd) {
      // A later tile's lines from memory to L2 (n = 16384, 1 rhs 1725 -> 1544 us; chains
      // of four, whose steps are longer, lose by it: 2206 -> 2277).
      const int Jp = block(s + kTAhead) * kTB;
      if (kTrans) {
        const int k = Jp + tid / 2;
        if (tid % 2 == 0 && k < n && i0 + rank * kTRows < n)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(a + (int64_t)k * lda + i0 + rank * kTRows));
      } else if (part < kTB * (int)sizeof(TA) / 128 && row < n && Jp + part * (128 / (int)sizeof(TA)) < n) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(a + (int64_t)row * lda + Jp + part * (128 / (int)sizeof(TA))));
      }
    }
    ok = __syncthreads_or(!ok) == 0;
    if (!ok) break;
#pragma unroll
    for (int e = 0; e < kLen; ++e) acc = fma(-v[e], xs[s & 1][(part + kParts * e) * kNR + c], acc);
    if (s + 1 < nupd) {
#pragma unroll
      for (int e = 0; e < kLen; ++e) v[e] = nv[e];
    }
  }
  if (ok) {
    // The row's sum, to all four CTAs (a lane each).
#pragma unroll
    for (int off = 1; off < kParts; off <<= 1) acc += __shfl_xor_sync(kFull, acc, off);
    if (part < kTCtas)
      cl_push8(cl_peer(cl_smem(&sums[r * kNR + c]), part), cl_peer(cl_smem(&bar), part), Word::bits(on ? acc : T(0)));
    ok = cl_wait(cl_smem(&bar), 0u, st, I);
    if (ok) {
      T y = T(0);
#pragma unroll
      for (int e = 0; e < kLen; ++e) y = fma(d[e], Word::from(sums[(part + kParts * e) * kNR + c]), y);
#pragma unroll
      for (int off = 1; off < kParts; off <<= 1) y += __shfl_xor_sync(kFull, y, off);
      if (on && part == 0) {
        Word::store(xt + ((size_t)I * kVals + r * kNR + c) * kW, y, epoch);
        x[(int64_t)row * ldx + c] = y;
      }
    }
  }
  cl_sync();  // every push has been issued; those to this CTA have landed if it waited for them
  if (!ok) cl_drain();
}

// Wide chains of transposed FP32 sweeps (four right-hand sides).  A row of a tile is a
// column of memory there, so that a load takes a line for every column of the tile
// among its lanes; a thread has all four right-hand sides of its row, a quarter of the
// loads: 16 rows x 16 parts of 4 columns, a warp on 16 rows and two columns (64 bytes
// of two lines a load), sums over the parts by shuffle and over the warps in shared
// memory.  Otherwise as above.  Two sweeps with 16 right-hand sides, us, one CTA a
// block with flags / a sum a thread / so: n = 4097 535 / 388 / 260, 8000 1400 / 1343 / 581,
// 16384 3413 / 4829 / 1700.
template <bool kLower>
__global__ void __launch_bounds__(256)
    trsv_cluster_wide_kernel(const float* __restrict__ a, int64_t lda, float* x, int64_t ldx, int n, int nrhs,
                             int nchain, const float* __restrict__ dinv, unsigned long long* xt, unsigned epoch,
                             int* ticket, DeviceStatus* st) {
  using Word = TcWord<float>;
  constexpr int kNR = 4, kThreads = 256, kParts = kThreads / kTRows, kLen = kTB / kParts;
  constexpr int kVals = kTB * kNR, kOut = kTRows * kNR;  // values of a block, of a CTA
  static_assert(kVals == kThreads && kOut * kTCtas == kThreads, "a thread polls a value and sends one to a peer");
  constexpr unsigned kFull = 0xffffffffu;
  __shared__ __align__(16) float xs[2][kVals];                     // x(J), [k][c]
  __shared__ __align__(16) float red[2][kThreads / 32][kOut];      // the warps' sums, of both products
  __shared__ unsigned long long sums[kVals];                       // the block's sums, [row][c]
  __shared__ __align__(8) unsigned long long bar;
  __shared__ int s_ticket;
  const int tid = threadIdx.x;
  const int rank = blockIdx.x & (kTCtas - 1);
  const int nblk = (n + kTB - 1) / kTB;
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cl_smem(&bar)));
    asm volatile("fence.mbarrier_init.release.cluster;");
    cl_expect(cl_smem(&bar), (unsigned)kVals * 8u);
    if (rank == 0) {
      const int t = atomicAdd(ticket, 1);
      for (int r = 0; r < kTCtas; ++r)
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cl_peer(cl_smem(&s_ticket), r)), "r"(t) : "memory");
    }
  }
  cl_sync();
  const int chain = s_ticket % nchain, t = s_ticket / nchain;
  x += chain * kNR;
  nrhs = min(kNR, nrhs - chain * kNR);
  xt += (size_t)chain * nblk * kVals;
  const int I = kLower ? t : nblk - 1 - t;
  const int part = tid / kTRows, r = rank * kTRows + tid % kTRows;
  const int row = I * kTB + r;
  const int nupd = kLower ? I : nblk - 1 - I;  // blocks before I in sweep order
  auto block = [&](int s) { return kLower ? s : nblk - 1 - s; };
  auto load_tile = [&](int J, float(&v)[kLen]) {
#pragma unroll
    for (int e = 0; e < kLen; ++e) {
      const int k = J * kTB + part + kParts * e;
      v[e] = row < n && k < n ? a[(int64_t)k * lda + row] : 0.0f;
    }
  };
  const bool polls = tid % kNR < nrhs;
  auto word = [&](int J) { return xt + (size_t)J * kVals + tid; };
  float d[kLen], v[kLen], acc[kNR];
#pragma unroll
  for (int e = 0; e < kLen; ++e) d[e] = dinv[(size_t)I * kTB * kTB + (part + kParts * e) * kTB + r];
#pragma unroll
  for (int c = 0; c < kNR; ++c) acc[c] = part == 0 && row < n && c < nrhs ? x[(int64_t)row * ldx + c] : 0.0f;
  unsigned long long w[1];
  bool ok = true;
  if (nupd > 0) {
    load_tile(block(0), v);
    if (polls) Word::load(word(block(0)), w);
  }
  for (int s = 0; s < nupd; ++s) {
    const int J = block(s);
    float xv = 0.0f;
    if (polls && J * kTB + tid / kNR < n) {
      unsigned long long t0 = 0;
      unsigned spins = 0;
      while (!Word::ok(w, epoch)) {
        Word::load(word(J), w);
        if ((++spins & 31u) == 0) {
          const unsigned long long now = global_timer_ns();
          if (t0 == 0) t0 = now;
          const bool late = now - t0 > st->timeout_ns;
          if (late) {
            atomicCAS(&st->error, kDevOk, kDevBarrierTimeout);
            atomicExch(&st->timeout_where, (unsigned long long)J);
            atomicExch(&st->abort, 1);
          }
          if (late || ld_relaxed_i32(&st->abort)) {
            ok = false;
            break;
          }
        }
      }
      xv = Word::value(w);
    }
    xs[s & 1][tid] = xv;
    float nv[kLen];
    if (s + 1 < nupd) {
      load_tile(block(s + 1), nv);
      if (polls) Word::load(word(block(s + 1)), w);
    }
    ok = __syncthreads_or(!ok) == 0;
    if (!ok) break;
#pragma unroll
    for (int e = 0; e < kLen; ++e) {
      const float4 xk = *reinterpret_cast<const float4*>(&xs[s & 1][(part + kParts * e) * kNR]);
      acc[0] = fmaf(-v[e], xk.x, acc[0]);
      acc[1] = fmaf(-v[e], xk.y, acc[1]);
      acc[2] = fmaf(-v[e], xk.z, acc[2]);
      acc[3] = fmaf(-v[e], xk.w, acc[3]);
    }
    if (s + 1 < nupd) {
#pragma unroll
      for (int e = 0; e < kLen; ++e) v[e] = nv[e];
    }
  }
  if (ok) {
    // Sums over the parts, to thread t for value t % kOut of the CTA and peer t / kOut.
    auto over_parts = [&](float(&sum)[kNR], int buf) {
#pragma unroll
      for (int c = 0; c < kNR; ++c) sum[c] += __shfl_xor_sync(kFull, sum[c], kTRows);
      if ((tid & 31) < kTRows)
        *reinterpret_cast<float4*>(&red[buf][tid >> 5][(tid & 31) * kNR]) = make_float4(sum[0], sum[1], sum[2], sum[3]);
      __syncthreads();
      float total = 0.0f;
#pragma unroll
      for (int q = 0; q < kThreads / 32; ++q) total += red[buf][q][tid % kOut];
      return total;
    };
    const int vr = rank * kTRows + tid % kOut / kNR, vc = tid % kNR, peer = tid / kOut, vrow = I * kTB + vr;
    const bool on = vrow < n && vc < nrhs;
    const float sum = over_parts(acc, 0);
    cl_push8(cl_peer(cl_smem(&sums[vr * kNR + vc]), peer), cl_peer(cl_smem(&bar), peer), Word::bits(on ? sum : 0.0f));
    // All warps alike: there is a barrier ahead.
    ok = __syncthreads_and(cl_wait(cl_smem(&bar), 0u, st, I)) != 0;
    if (ok) {
      float y[kNR] = {};
#pragma unroll
      for (int e = 0; e < kLen; ++e)
#pragma unroll
        for (int c = 0; c < kNR; ++c) y[c] = fmaf(d[e], Word::from(sums[(part + kParts * e) * kNR + c]), y[c]);
      const float out = over_parts(y, 1);
      if (on && peer == 0) {
        Word::store(xt + (size_t)I * kVals + vr * kNR + vc, out, epoch);
        x[(int64_t)vrow * ldx + vc] = out;
      }
    }
  }
  cl_sync();  // as above
  if (!ok) cl_drain();
}

// Right-hand sides of one chain (at most 16 chains run in a launch).  FP64 sweeps
// run every right-hand side as a chain of its own: they are bound by the chain or,
// with many, by the FP64 pipes, whatever the width.  FP32 sweeps of much work read
// the factor fewer times in chains of four.  Two sweeps with their inverses in us,
// chains of 1 / 4: FP64 n = 2048, 8 rhs 212 / 288, n = 4097, 16 rhs 737 / 900, n =
// 16384, 16 rhs 8098 / 9863; FP32 n = 2048, 16 rhs 110 / 101, n = 4097, 8 rhs 227 / 181,
// 16 rhs 323 / 227, n = 16384, 4 rhs 1217 / 920.  (One CTA a block, flags and fences:
// FP64 n = 1000, 1 rhs 174, now 98; 2048, 8 rhs 354, now 208; 4097, 16 rhs 1079, now
// 712; 16384, 16 rhs 10145, now 8003; FP32 n = 2048, 16 rhs 210, 4097, 8 rhs 375.)
template <typename T>
static int tc_width(int n, int nc) {
  return sizeof(T) == 4 && nc > 2 && (int64_t)n * nc > 30000 ? 4 : 1;
}

size_t trsv_cluster_tag_words(int n, int nrhs, size_t elem) {
  return (size_t)trsv_syncfree_blocks(n) * kTB * ((std::min(nrhs, kTrsvMaxChains) + 3) / 4 * 4) * (elem / 4);
}

template <typename T, typename TA, bool LO, bool TR, int NR>
static cudaError_t launch_nr(cudaStream_t stream, const TA* a, int64_t lda, T* x, int64_t ldx, int n, int nc,
                             const T* dinv, unsigned long long* xt, unsigned epoch, int* ticket, DeviceStatus* st) {
  const int nchain = (nc + NR - 1) / NR;
  cudaLaunchAttribute attr;
  cudaLaunchConfig_t cfg = cl_config(kTCtas, tc_threads<NR>(), 0, stream, &attr);
  cfg.gridDim = dim3(kTCtas * trsv_syncfree_blocks(n) * nchain);
  return cudaLaunchKernelEx(&cfg, trsv_cluster_kernel<T, TA, LO, TR, NR>, a, lda, x, ldx, n, nc, nchain, dinv, xt,
                            epoch, ticket, st);
}

template <typename T, typename TA, bool LO, bool TR>
static cudaError_t launch_dir(cudaStream_t stream, const TA* a, int64_t lda, T* x, int64_t ldx, int n, int nc,
                              const T* dinv, unsigned long long* xt, unsigned epoch, int* ticket, DeviceStatus* st) {
  if constexpr (sizeof(T) == 4) {
    if (tc_width<T>(n, nc) == 4) {
      if constexpr (TR) {
        const int nchain = (nc + 3) / 4;
        cudaLaunchAttribute attr;
        cudaLaunchConfig_t cfg = cl_config(kTCtas, 256, 0, stream, &attr);
        cfg.gridDim = dim3(kTCtas * trsv_syncfree_blocks(n) * nchain);
        return cudaLaunchKernelEx(&cfg, trsv_cluster_wide_kernel<LO>, a, lda, x, ldx, n, nc, nchain, dinv, xt, epoch,
                                  ticket, st);
      } else {
        return launch_nr<T, TA, LO, TR, 4>(stream, a, lda, x, ldx, n, nc, dinv, xt, epoch, ticket, st);
      }
    }
  }
  return launch_nr<T, TA, LO, TR, 1>(stream, a, lda, x, ldx, n, nc, dinv, xt, epoch, ticket, st);
}

template <typename T, typename TA>
cudaError_t launch_trsv_cluster(cudaStream_t stream, const TA* a, int64_t lda, T* x, int64_t ldx, int n, int nc,
                                bool lower, bool trans, const T* dinv, unsigned long long* xt, unsigned epoch,
                                int* ticket, DeviceStatus* st) {
  cudaError_t e = cudaMemsetAsync(ticket, 0, sizeof(int), stream);
  if (e != cudaSuccess) return e;
  if (lower && !trans) return launch_dir<T, TA, true, false>(stream, a, lda, x, ldx, n, nc, dinv, xt, epoch, ticket, st);
  if (lower) return launch_dir<T, TA, true, true>(stream, a, lda, x, ldx, n, nc, dinv, xt, epoch, ticket, st);
  if (!trans) return launch_dir<T, TA, false, false>(stream, a, lda, x, ldx, n, nc, dinv, xt, epoch, ticket, st);
  return launch_dir<T, TA, false, true>(stream, a, lda, x, ldx, n, nc, dinv, xt, epoch, ticket, st);
}

#define LUHOT_TRSV_CLUSTER(T, TA)                                                                                  \
  template cudaError_t launch_trsv_cluster<T, TA>(cudaStream_t, const TA*, int64_t, T*, int64_t, int, int, bool, bool, \
                                                  const T*, unsigned long long*, unsigned, int*, DeviceStatus*);
LUHOT_TRSV_CLUSTER(double, double)
LUHOT_TRSV_CLUSTER(float, float)
LUHOT_TRSV_CLUSTER(double, float)
#undef LUHOT_TRSV_CLUSTER

}  // namespace luhot
