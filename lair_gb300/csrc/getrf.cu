// Blocked right-looking LU with partial pivoting on one GB300 (sm_103a).
//
// Matrix layout in HBM: row-major, leading dimension lda >= n (elements).
// Pivots: int32 on the device, LAPACK-style sequential interchanges
// (step i swapped row i with row piv[i]), the convention of lair's
// src/lapack/getrf.rs:12-27.
//
// One block step k0 (panel width w) runs three kernels:
//   1. panel_kernel   cooperative; factors rows [k0, m) x cols [k0, k0+w) held
//                     in shared memory across all CTAs; per column one
//                     exchange of step-tagged candidates through L2 (integer
//                     pivot keys, redux.sync reduce, deterministic order; the
//                     winner's row segment follows by cp.async off the
//                     critical path), row interchanges as id swaps, and the
//                     update of the previous step overlapping the exchange.
//                     Panels whose rows fit in one thread-block cluster run
//                     there (panel_cluster.cu): 1.1 us a column instead of 2.5.
//   2. swap_solve_kernel (swap_solve.cu): the panel's interchanges on the
//                     columns left and right of it (a gather of the at most 2w
//                     rows that moved), U12 <- L11^-1 A12, and the operand slices
//                     of a tensor-core update.
//   3. gemm_*_kernel  A22 <- A22 - L21 U12 (the Schur complement).
//
// Two arithmetic modes:
//   exact: every update is a separately rounded multiply then subtract, in
//          increasing elimination-step order, which is exactly the sequence
//          of lair's getrf_row_major (src/lapack/getrf.rs:76-89).  Blocking
//          only moves data, so results are bit-identical to lair.
//   fast:  the FP64 Schur update runs as integer slice products on the FP16 tensor
//          cores (ozaki.cu) for trailing blocks of at least 256 x 256, else on the
//          FP64 tensor cores (DMMA, mma.sync m8n8k4); the other kernels use FMA.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "luhot_internal.h"
#include "ozaki.cuh"
#include "panel.cuh"
#include "swap_solve.cuh"
#include "tc_gemm.cuh"

namespace luhot {

// ---------------------------------------------------------------------------
// 1. Panel factorization.
// ---------------------------------------------------------------------------
// Exchange words: payload in the low 32 bits, the step tag in the high 32 (headers:
// 48 bits and 16).
// A reader accepts a word only when its tag is the step it waits for, so no
// fence or counter orders the writers and readers: each 8-byte word is
// written and read whole.  Tags are step + 1 and the slots are zeroed before
// each factorization, so a stale word never carries a live tag.
// Reuse: the slots alternate by step parity, and a CTA rewrites its slot of
// parity j & 1 at step j + 2 only after it has seen every CTA's step j + 1
// header.  Each CTA publishes that header only after all its reads of step j
// have returned their values (the poll consumes them; the segment copy is
// waited for and its tags checked).  So no read of step j can observe a
// step j + 2 word; the order comes from the data dependencies, not from a
// fence.
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_word(unsigned long long* p, unsigned int bits, unsigned int tag) {
  const unsigned long long v = ((unsigned long long)tag << 32) | bits;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ bool word_ok(unsigned long long v, unsigned int tag) {
  return (unsigned int)(v >> 32) == tag;
}
// A whole header (FP64 32 bytes, FP32 16) in one load or store; each 8-byte
// element is read and written whole.  p aligned to the header.
__device__ __forceinline__ void ld_head(const unsigned long long* p, unsigned long long (&v)[4]) {
  asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
               : "=l"(v[0]), "=l"(v[1]), "=l"(v[2]), "=l"(v[3])
               : "l"(p)
               : "memory");
}
__device__ __forceinline__ void ld_head(const unsigned long long* p, unsigned long long (&v)[2]) {
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v[0]), "=l"(v[1]) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_head(unsigned long long* p, const unsigned long long (&v)[4]) {
  asm volatile("st.relaxed.gpu.global.v4.u64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(v[0]), "l"(v[1]), "l"(v[2]), "l"(v[3])
               : "memory");
}
__device__ __forceinline__ void st_head(unsigned long long* p, const unsigned long long (&v)[2]) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(v[0]), "l"(v[1]) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// 16 bytes global -> shared through L2 (cp.async.cg), completed by
// cp_async_wait_all; no register holds the data in between.
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const unsigned int d = (unsigned int)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(gmem_src) : "memory");
}

// Segment values as one (FP32) or two (FP64) tagged words.  The header of a
// CTA holds its candidate's key with the pivot's sign in the top bit (so the key
// also gives the pivot value), the row id and the candidate's column j+1 value,
// 96 (FP32) or 160 bits, in kHead words of 48 bits over a 16-bit tag (the step's
// low bits; a header is rewritten at every second step, so that an old tag is
// never 65536 steps old).  The headers lie 64 bytes apart, ahead of all segments: a
// warp's poll of 64 CTAs reads 32 lines of 128 bytes and has every load in flight at
// once, an L2 latency (some 850 cycles across the dies) a poll.  (Packed, FP32 headers
// share a line with seven others that are being written: 205 / 192 us a 64-column panel
// of 20000 rows, 254 / 241 of 40000; FP64, two to a line or four, the same.)
template <typename T>
struct Tagged;
template <>
struct Tagged<float> {
  using K = unsigned int;
  static constexpr int kWords = 1, kHead = 2;
  static constexpr K kSign = 0x80000000u;
  __device__ static void put(unsigned long long* p, float v, unsigned int tag) { st_word(p, __float_as_uint(v), tag); }
  __device__ static float value(const unsigned long long* w) { return __uint_as_float((unsigned int)w[0]); }
  __device__ static bool ok(const unsigned long long* w, unsigned int tag) { return word_ok(w[0], tag); }
  __device__ static void pack(K key, int id, float u1, unsigned int tag, unsigned long long (&h)[2]) {
    const unsigned int u = __float_as_uint(u1), t = tag & 0xffffu;
    h[0] = ((unsigned long long)key << 32) | (u & 0xffff0000u) | t;
    h[1] = ((unsigned long long)(unsigned int)id << 32) | (u << 16) | t;
  }
  __device__ static bool head_ok(const unsigned long long (&h)[2], unsigned int tag) {
    return (((h[0] ^ tag) | (h[1] ^ tag)) & 0xffffu) == 0;
  }
  __device__ static K key(const unsigned long long (&h)[2]) { return (K)(h[0] >> 32); }
  __device__ static int id(const unsigned long long (&h)[2]) { return (int)(h[1] >> 32); }
  __device__ static float u1(const unsigned long long (&h)[2]) {
    return __uint_as_float(((unsigned int)h[0] & 0xffff0000u) | ((unsigned int)h[1] >> 16));
  }
};
template <>
struct Tagged<double> {
  using K = unsigned long long;
  static constexpr int kWords = 2, kHead = 4;
  static constexpr K kSign = 0x8000000000000000ull;
  __device__ static void put(unsigned long long* p, double v, unsigned int tag) {
    const K k = (K)__double_as_longlong(v);
    st_word(p, (unsigned int)(k >> 32), tag);
    st_word(p + 1, (unsigned int)k, tag);
  }
  __device__ static double value(const unsigned long long* w) {
    return __longlong_as_double((long long)(((K)(unsigned int)w[0] << 32) | (unsigned int)w[1]));
  }
  __device__ static bool ok(const unsigned long long* w, unsigned int tag) {
    return word_ok(w[0], tag) && word_ok(w[1], tag);
  }
  __device__ static void pack(K key, int id, double u1, unsigned int tag, unsigned long long (&h)[4]) {
    const K u = (K)__double_as_longlong(u1), t = tag & 0xffffu;
    h[0] = (key & ~(K)0xffff) | t;
    h[1] = (key << 48) | ((K)(unsigned int)id << 16) | t;
    h[2] = (u & ~(K)0xffff) | t;
    h[3] = (u << 48) | t;
  }
  __device__ static bool head_ok(const unsigned long long (&h)[4], unsigned int tag) {
    return (((h[0] ^ tag) | (h[1] ^ tag) | (h[2] ^ tag) | (h[3] ^ tag)) & 0xffffu) == 0;
  }
  __device__ static K key(const unsigned long long (&h)[4]) { return (h[0] & ~(K)0xffff) | (h[1] >> 48); }
  __device__ static int id(const unsigned long long (&h)[4]) { return (int)(unsigned int)(h[1] >> 16); }
  __device__ static double u1(const unsigned long long (&h)[4]) {
    return __longlong_as_double((long long)((h[2] & ~(K)0xffff) | (h[3] >> 48)));
  }
};

// Give up a wait: record the step, raise abort so every other wait of the
// launch returns at once.  Called by one lane.
__device__ __forceinline__ void panel_give_up(DeviceStatus* st, int step) {
  atomicCAS(&st->error, kDevOk, kDevBarrierTimeout);
  atomicExch(&st->timeout_where, (unsigned long long)step);
  atomicExch(&st->abort, 1);
}
// Warp-uniform test of the wait limit and of another CTA's abort.
__device__ __forceinline__ bool panel_wait_over(DeviceStatus* st, unsigned long long t0) {
  const int late = (global_timer_ns() - t0 > st->timeout_ns) ? 1 : 0;
  return __shfl_sync(0xffffffffu, late, 0) != 0 || __any_sync(0xffffffffu, ld_relaxed_i32(&st->abort) != 0);
}

// FP32 rows in 16-byte chunks: lane (sub, ch) of a warp takes columns
// [4ch, 4ch+4) of row sub of the warp's current row group (W/4 chunks a row,
// 32/(W/4) rows a warp instruction); two row groups per pass with all loads
// first.  Columns left of c0 in the first chunk keep their value (the same
// single update per element as the scalar form, so exact mode is unchanged);
// chunks at or beyond the padded width are not touched.  Needs rows and u
// 16-byte aligned (lds and the row base multiples of 4 floats).
template <int W, bool kExact>
__device__ __forceinline__ void panel_update_f32x4(float* S, int lds, int r0, int nloc, int skip, int jj, int c0,
                                                   int w, const float* u, int t, int nt) {
  constexpr int CH = W / 4, RPW = 32 / CH, kR = 2;
  const int lane = t & 31, wi = t >> 5, nw = nt >> 5;
  const int ch = lane % CH, sub = lane / CH;
  const int c = ch * 4;
  if (c + 4 <= c0 || c >= w || r0 >= nloc) return;
  const float4 uv = *reinterpret_cast<const float4*>(u + c);
  const int G = nw * RPW;
  for (int rb = r0 + wi * RPW + sub; rb < nloc; rb += kR * G) {
    float l[kR];
    float4 x[kR];
#pragma unroll
    for (int e = 0; e < kR; ++e) {
      const float* row = S + (rb + e * G < nloc ? rb + e * G : rb) * lds;
      l[e] = row[jj];
      x[e] = *reinterpret_cast<const float4*>(row + c);
    }
#pragma unroll
    for (int e = 0; e < kR; ++e) {
      const int r = rb + e * G;
      if (r < nloc && r != skip) {
        float4 y = x[e];
        if (c + 0 >= c0) y.x = upd<kExact>(y.x, l[e], uv.x);
        if (c + 1 >= c0) y.y = upd<kExact>(y.y, l[e], uv.y);
        if (c + 2 >= c0) y.z = upd<kExact>(y.z, l[e], uv.z);
        if (c + 3 >= c0) y.w = upd<kExact>(y.w, l[e], uv.w);
        *reinterpret_cast<float4*>(S + r * lds + c) = y;
      }
    }
  }
}
// A[r][c] -= A[r][jj] * u[c] for the rows [r0, nloc) other than `skip` and
// the columns [c0, w), by threads t of nt (a multiple of 32).  FP64 flattens
// (row, column) pairs so every lane is busy (the FP64 pipe bounds it); FP32
// gives each warp whole rows, lanes along the columns (no index arithmetic
// per element; shared-memory latency bounds it, hence the batched loads).
template <typename T, bool kExact>
__device__ __forceinline__ void panel_update(T* S, int lds, int r0, int nloc, int skip, int jj, int c0, int w,
                                             const T* u, int t, int nt) {
  const int wc = w - c0;
  if (wc <= 0 || r0 >= nloc) return;
  if constexpr (sizeof(T) == 8) {
    const int total = (nloc - r0) * wc;
    const int step_r = nt / wc, step_c = nt - step_r * wc;
    int r = r0 + t / wc, c = t - (t / wc) * wc;
    for (int idx = t; idx < total; idx += 2 * nt) {
      const int ra = r, ca = c;
      r += step_r;
      c += step_c;
      if (c >= wc) {
        c -= wc;
        ++r;
      }
      const int rb = r, cb = c;
      const bool on_b = idx + nt < total;
      r += step_r;
      c += step_c;
      if (c >= wc) {
        c -= wc;
        ++r;
      }
      T xa = T(0), la = T(0), ua = T(0), xb = T(0), lb = T(0), ub = T(0);
      const bool do_a = ra != skip, do_b = on_b && rb != skip;
      if (do_a) {
        xa = S[ra * lds + c0 + ca];
        la = S[ra * lds + jj];
        ua = u[c0 + ca];
      }
      if (do_b) {
        xb = S[rb * lds + c0 + cb];
        lb = S[rb * lds + jj];
        ub = u[c0 + cb];
      }
      if (do_a) S[ra * lds + c0 + ca] = upd<kExact>(xa, la, ua);
      if (do_b) S[rb * lds + c0 + cb] = upd<kExact>(xb, lb, ub);
    }
  } else {
    if (w <= 64)
      panel_update_f32x4<64, kExact>(S, lds, r0, nloc, skip, jj, c0, w, u, t, nt);
    else
      panel_update_f32x4<128, kExact>(S, lds, r0, nloc, skip, jj, c0, w, u, t, nt);
  }
}

// Cooperative panel factorization: rows [k0, m) x columns [k0, k0 + w) are
// spread over P CTAs (rows_per each) and held in shared memory for the whole
// panel.  Rows are never moved between CTAs during the panel: each CTA keeps
// the global row index (id) of every row it holds, and an interchange of rows
// ul and pr only swaps two ids.  The row that receives id ul is the pivot
// row; its CTA moves it into its block of retired rows [0, r0) (a local move).
// At the end every row is written to the global row its id names.
//
// Per column j (elimination step ul = k0 + j), with the update of step j-1
// to columns j+1.. still pending for all rows but this CTA's candidate row:
//   warp 0:     publish the candidate's header (key = |pivot| bits with the
//               pivot's sign on top, row id, column j+1 value after the
//               pending update) in one store; poll the P headers until all
//               carry this step's tag, folding them into the winner (the
//               pivot and its column j+1 value come with its header); pass the
//               winner to warp 1 and form the reciprocal;
//   warp 1:     meanwhile, the candidate row's pending update (columns
//               j+2..) and the publication of its segment j+2..; once the winner
//               is known, start the copy of its segment into shared memory
//               (cp.async) and relabel the ids of rows ul and pr;
//   warps 1-:   the pending update of step j-1 of the other rows (columns
//               j+1..), which thus overlaps the exchange.
//   barrier;    the pivot row's CTA retires it; the warps but 1 scale column j,
//               update column j+1 only and find its candidates while warp 1
//               checks the copied segment's tags and keeps it for the next
//               step's updates; barrier.
// What bounds it is that chain: some 2200 of a column's 5000 cycles are the header's
// way through L2 and its polls, 500 an FP64 division, 800 the scaling and search.
// us a 64-column panel (a getrf call), with 40- or 64-byte slots polled one after the
// other / now: FP64 218 / 230 at 4000 rows (polls of two headers a lane), 243 / 230 at 4500,
// 242 / 230 at 6000, 287 / 258 at 16000; FP32 200 / 180 at 8000, 208 / 192 at 20000, 239 / 241
// at 40000, 283 / 256 at 80000.
// The arithmetic and its order per element are those of lair's
// getrf_row_major (src/lapack/getrf.rs:56-89): 1/p rounded, l = a*(1/p)
// rounded, a - l*u (separately rounded in exact mode), steps in order.
template <typename T, bool kExact>
__global__ void __launch_bounds__(512, 1) panel_kernel(PanelArgs<T> p) {
  using K = typename PivotKey<T>::K;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* S = reinterpret_cast<T*>(smem_raw);                        // [rows_per][lds]
  T* segb = S + (size_t)p.rows_per * p.lds;                     // [2][kMaxPanelWidth] pivot rows
  int* ids = reinterpret_cast<int*>(segb + 2 * kMaxPanelWidth);  // [rows_per] global row of each slot
  int* orig = ids + p.rows_per;  // [rows_per] the row each slot's content started in
  __shared__ K red_k[16];
  __shared__ int red_i[16], red_s[16];
  __shared__ int ulslot[kMaxPanelWidth];  // slot holding row id k0 + jj in this CTA, or -1
  __shared__ __align__(16) unsigned long long stage[2 * kMaxPanelWidth];  // the winner's segment words
  __shared__ int s_ok, s_r0, s_pivoted, s_ret;
  __shared__ T s_recip, s_u1;
  __shared__ int s_pr, s_win;  // the step's pivot row and its CTA (-1: no pivot)

  constexpr unsigned kFull = 0xffffffffu;
  const int kWarps = blockDim.x >> 5;
  constexpr int kW = Tagged<T>::kWords;
  const int P = gridDim.x;
  const int b = blockIdx.x;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int r_begin = p.k0 + b * p.rows_per;
  const int nloc = max(0, min(p.m, r_begin + p.rows_per) - r_begin);
  const int w = p.w;
  const int lds = p.lds;

  for (int idx = tid; idx < nloc * w; idx += blockDim.x) {
    const int r = idx / w, c = idx - r * w;
    S[r * lds + c] = p.a[(int64_t)(r_begin + r) * p.lda + p.k0 + c];
  }
  for (int r = tid; r < nloc; r += blockDim.x) ids[r] = orig[r] = r_begin + r;
  for (int jj = tid; jj < w; jj += blockDim.x) {
    const int s = p.k0 + jj - r_begin;
    ulslot[jj] = (s >= 0 && s < nloc) ? s : -1;
  }
  if (tid == 0) {
    s_r0 = 0;
    s_ok = 1;
  }
  __syncthreads();
  {
    // Column 0 candidates.
    K bk = 0;
    int bi = INT_MAX, bs = -1;
    for (int r = tid; r < nloc; r += blockDim.x) key_combine(bk, bi, bs, PivotKey<T>::of(S[r * lds]), ids[r], r);
    key_reduce_redux(bk, bi, bs);
    if (lane == 0) {
      red_k[warp] = bk;
      red_i[warp] = bi;
      red_s[warp] = bs;
    }
  }
  __syncthreads();

  const int nq = (P + 31) / 32;  // candidate CTAs per lane in the poll
  int dj = -1;                   // step whose update of columns dj+2.. is pending
  int dr0 = 0;                   // first active row of that step
  for (int j = 0; j < w; ++j) {
    const int ul = p.k0 + j;
    const unsigned int tag = (unsigned int)ul + 1u;
    unsigned long long* slots = p.slots + (size_t)(j & 1) * kMaxPanelCtas * kPanelSlotWords;
    T* seg = segb + (j & 1) * kMaxPanelWidth;
    // The CTA's candidate for column j (lanes below kWarps hold the warps').
    K ck = lane < kWarps ? red_k[lane] : K(0);
    int ci = lane < kWarps ? red_i[lane] : INT_MAX;
    int cs = lane < kWarps ? red_s[lane] : -1;
    const int csrc = warp_best(ck, ci);
    ck = PivotKey<T>::shfl(ck, csrc);
    ci = __shfl_sync(kFull, ci, csrc);
    cs = __shfl_sync(kFull, cs, csrc);
    bool seg_live = false;  // warp 1: the winner's segment j+2.. is being copied into stage
    const unsigned long long* wseg = nullptr;
    if (warp == 0) {
      const unsigned long long* heads = p.heads + (size_t)(j & 1) * kMaxPanelCtas * kPanelHeaderWords;
      const T* up = segb + (dj & 1) * kMaxPanelWidth;  // step dj's pivot row
      // The header only (warp 1 publishes the segment): the column j+1 value
      // after the pending update (kept in the row), the row id and the key
      // with the pivot's sign.
      {
        K sgn = 0;
        T u1 = T(0);
        if (cs >= 0) {
          const T* row = S + cs * lds;
          if (j + 1 < w) {
            u1 = row[j + 1];
            if (dj >= 0) u1 = upd<kExact>(u1, row[dj], up[j + 1]);
          }
          if (signbit(row[j])) sgn = Tagged<T>::kSign;
        }
        __syncwarp();
        if (lane == 0) {
          unsigned long long h[Tagged<T>::kHead];
          Tagged<T>::pack(ck | sgn, ci, u1, tag, h);
          st_head(const_cast<unsigned long long*>(heads) + b * kPanelHeaderWords, h);
          if (cs >= 0 && j + 1 < w && dj >= 0) S[cs * lds + j + 1] = u1;
        }
      }
      // Poll every CTA's header; fold each one in as soon as it is current.
      K k = 0, kraw = 0;
      int i = INT_MAX, win = -1;
      T u1b = T(0);
      unsigned pending = 0;
      for (int q = 0; q < nq; ++q)
        if (lane + 32 * q < P) pending |= 1u << q;
      unsigned long long t0 = 0;
      unsigned int spins = 0;
      int ok = 1;
      while (true) {
        constexpr int kB = 3;  // loads in flight (96 CTAs)
        for (int q0 = 0; q0 < nq; q0 += kB) {
          unsigned long long h[kB][Tagged<T>::kHead];
#pragma unroll
          for (int e = 0; e < kB; ++e)
            if (pending & (1u << (q0 + e))) ld_head(heads + (lane + 32 * (q0 + e)) * kPanelHeaderWords, h[e]);
#pragma unroll
          for (int e = 0; e < kB; ++e) {
            if (!(pending & (1u << (q0 + e))) || !Tagged<T>::head_ok(h[e], tag)) continue;
            const K hraw = Tagged<T>::key(h[e]);
            const K hk = hraw & ~Tagged<T>::kSign;
            const int hid = Tagged<T>::id(h[e]);
            if (hk > k || (hk == k && hid < i)) {
              k = hk;
              i = hid;
              win = lane + 32 * (q0 + e);
              kraw = hraw;
              u1b = Tagged<T>::u1(h[e]);
            }
            pending &= ~(1u << (q0 + e));
          }
        }
        if (__all_sync(kFull, pending == 0)) break;
        if ((++spins & 15u) == 0) {
          if (spins == 16u) t0 = global_timer_ns();
          if (panel_wait_over(p.st, t0)) {
            if (lane == 0 && !ld_relaxed_i32(&p.st->abort)) panel_give_up(p.st, ul);
            ok = 0;
            break;
          }
        }
      }
      const int src = warp_best(k, i);
      const K praw = PivotKey<T>::shfl(kraw, src);
      const bool pos = (praw & ~Tagged<T>::kSign) != 0;
      if (lane == src) {
        s_win = ok && pos ? win : -1;
        s_pr = pos ? i : ul;
        s_u1 = u1b;
        s_pivoted = pos ? 1 : 0;
        s_ok = ok;
      }
      __syncwarp();
      asm volatile("bar.arrive 1, 64;" ::: "memory");
      if (lane == 0 && ok) {
        if (pos)
          s_recip = T(1) / PivotKey<T>::value(praw);
        else if (b == 0)
          // lair: max == 0 -> the step is singular, no swap, no update
          // (src/lapack/getrf.rs:72-73).  The last such step wins.
          atomicMax(&p.st->singular, ul);
      }
    } else {
      unsigned long long* slots = p.slots + (size_t)(j & 1) * kMaxPanelCtas * kPanelSlotWords;
      if (warp == 1 && cs >= 0) {
        // The candidate row's pending update of columns j+2.. (warp 0 did
        // column j+1), then its segment j+2.., while warp 0 polls.
        unsigned long long* mine = slots + (size_t)b * kPanelSlotWords;
        if (dj >= 0) {
          const T* up = segb + (dj & 1) * kMaxPanelWidth;
          const T l = S[cs * lds + dj];
          for (int c = dj + 3 + lane; c < w; c += 32) S[cs * lds + c] = upd<kExact>(S[cs * lds + c], l, up[c]);
          __syncwarp();
        }
        for (int c = j + 2 + lane; c < w; c += 32) Tagged<T>::put(mine + c * kW, S[cs * lds + c], tag);
      }
      if (dj >= 0)
        panel_update<T, kExact>(S, lds, dr0, nloc, cs, dj, dj + 2, w, segb + (dj & 1) * kMaxPanelWidth, tid - 32,
                                blockDim.x - 32);
      if (warp == 1) {
        asm volatile("bar.sync 1, 64;" ::: "memory");  // warp 0 has the winner
        const int win = s_win, pr = s_pr;
        if (win >= 0) {
          // Start the copy of the winner's segment j+2.. (whole 16-byte pairs of
          // its slot's words) into stage; it completes while the step goes on.
          wseg = slots + (size_t)win * kPanelSlotWords;
          const int o0 = ((j + 2) * kW) & ~1, o1 = (w * kW + 1) & ~1;
          seg_live = o1 > o0;
          for (int o = o0 + 2 * lane; o < o1; o += 64) cp_async16(stage + o, wseg + o);
          cp_async_commit();
        }
        // Relabel: the row with id ul takes id pr and the row with id pr
        // takes id ul; the latter (the pivot row) retires after the barrier.
        // Row pr is the winning CTA's candidate (slot cs); row ul's slot
        // comes from the map of the panel's pending row ids.
        if (s_ok && lane == 0) {
          const int s_ul = ulslot[j];
          int ret = s_ul;
          if (pr != ul) {
            const int s_pr_slot = (win == b) ? cs : -1;
            if (s_ul >= 0) ids[s_ul] = pr;
            if (s_pr_slot >= 0) ids[s_pr_slot] = ul;
            if (pr < p.k0 + w) ulslot[pr - p.k0] = s_ul;
            ret = s_pr_slot;
          }
          if (b == 0) p.piv[ul] = pr;
          s_ret = ret;
        }
      }
    }
    __syncthreads();
    if (!s_ok) return;
    // Retire the pivot row into slot r0.
    int r0 = s_r0;
    const int ret = s_ret;
    if (ret >= 0) {
      if (warp == 0 && ret != r0) {
        for (int c = lane; c < w; c += 32) {
          const T x = S[ret * lds + c];
          S[ret * lds + c] = S[r0 * lds + c];
          S[r0 * lds + c] = x;
        }
        if (lane == 0) {
          const int t = ids[ret];
          const int moved = ids[r0];  // this row now lives in slot ret
          if (moved > ul && moved < p.k0 + w) ulslot[moved - p.k0] = ret;
          ids[ret] = moved;
          ids[r0] = t;
          const int o = orig[ret];
          orig[ret] = orig[r0];
          orig[r0] = o;
        }
      }
      ++r0;
      __syncthreads();
      if (tid == 0) s_r0 = r0;
    }

    // Warps 0, 2-: scale column j, update column j+1 only, find its candidates.
    // Warp 1 meanwhile keeps the winner's segment for the next step.
    K bk = 0;
    int bi = INT_MAX, bs = -1;
    const int pivoted = s_pivoted;
    if (warp != 1) {
      const int t1 = warp == 0 ? tid : tid - 32, n1 = blockDim.x - 32;
      if (pivoted) {
        const T recip = s_recip, u1 = s_u1;
        const bool more = j + 1 < w;
        for (int r = r0 + t1; r < nloc; r += n1) {
          T* row = S + r * lds;
          const T l = mul_rn(row[j], recip);
          row[j] = l;
          if (more) {
            const T v = upd<kExact>(row[j + 1], l, u1);
            row[j + 1] = v;
            key_combine(bk, bi, bs, PivotKey<T>::of(v), ids[r], r);
          }
        }
      } else if (j + 1 < w) {
        for (int r = r0 + t1; r < nloc; r += n1)
          key_combine(bk, bi, bs, PivotKey<T>::of(S[r * lds + j + 1]), ids[r], r);
      }
      const int bsrc = warp_best(bk, bi);
      bk = PivotKey<T>::shfl(bk, bsrc);
      bi = __shfl_sync(kFull, bi, bsrc);
      bs = __shfl_sync(kFull, bs, bsrc);
    } else if (seg_live) {
      // The winner's segment from stage into the pivot-row buffer; a word
      // whose tag is not yet this step's (relaxed stores land in any order)
      // is read again.
      cp_async_wait_all();
      __syncwarp();
      bool got = true;
      unsigned long long t0 = 0;
      while (got) {
        for (int c = j + 2 + lane; c < w; c += 32) {
          unsigned long long* sw = stage + c * kW;
          if (Tagged<T>::ok(sw, tag)) {
            seg[c] = Tagged<T>::value(sw);
          } else {
#pragma unroll
            for (int e = 0; e < kW; ++e) sw[e] = ld_word(wseg + c * kW + e);
            got = false;
          }
        }
        if (__all_sync(kFull, got)) break;
        got = true;
        if (t0 == 0) t0 = global_timer_ns();
        if (panel_wait_over(p.st, t0)) got = false;
      }
      if (!got && lane == 0) {
        if (!ld_relaxed_i32(&p.st->abort)) panel_give_up(p.st, ul);
        s_ok = 0;
      }
    }
    if (lane == 0) {
      red_k[warp] = bk;
      red_i[warp] = bi;
      red_s[warp] = bs;
    }
    dj = pivoted ? j : -1;
    dr0 = r0;
    __syncthreads();
    if (!s_ok) return;
  }
  for (int idx = tid; idx < nloc * w; idx += blockDim.x) {
    const int r = idx / w, c = idx - r * w;
    p.a[(int64_t)ids[r] * p.lda + p.k0 + c] = S[r * lds + c];
  }
  // The rows that changed place, for the interchanges outside the panel.
  for (int r = tid; r < nloc; r += blockDim.x) {
    if (ids[r] != orig[r]) {
      const int e = atomicAdd(p.move_count, 1);
      if (e < 2 * kMaxPanelWidth) {  // at most 2w rows move; the bound guards the list
        p.moves[2 * e] = ids[r];
        p.moves[2 * e + 1] = orig[r];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// 2. Row interchanges outside the panel, from the panel's list of moved rows
//    (the composition of its w interchanges: at most 2w rows, each row's
//    final content comes from one source row).  A CTA takes 32 columns: it
//    loads every moved row's source values into shared memory, then stores
//    them at the destinations -- all loads independent, 256-byte row
//    segments.  Pure data movement, so exact mode is unaffected.
template <typename T>
__global__ void __launch_bounds__(256) laswp_moves_kernel(T* a, int64_t lda, const int* moves,
                                                          const int* move_count, int capacity, int c_left_begin,
                                                          int c_left_end, int c_right_begin, int n) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* vals = reinterpret_cast<T*>(smem_raw);  // [capacity][32]
  __shared__ int mv[4 * kMaxPanelWidth];      // the (destination, source) pairs
  const int count = min(min(*move_count, capacity), 2 * kMaxPanelWidth);
  const int tid = threadIdx.y * 32 + threadIdx.x;
  for (int i = tid; i < 2 * count; i += blockDim.x * blockDim.y) mv[i] = moves[i];
  __syncthreads();
  const int nleft = max(0, c_left_end - c_left_begin);
  const int t = blockIdx.x * 32 + threadIdx.x;
  const int nright = max(0, n - c_right_begin);
  const bool on = t < nleft + nright;
  const int c = (t < nleft) ? (c_left_begin + t) : (c_right_begin + t - nleft);
  // Eight source rows per thread in flight before any is stored.
  constexpr int kB = 8;
  for (int e0 = threadIdx.y; e0 < count; e0 += blockDim.y * kB) {
    T v[kB];
#pragma unroll
    for (int q = 0; q < kB; ++q) {
      const int e = e0 + q * blockDim.y;
      v[q] = (on && e < count) ? a[(int64_t)mv[2 * e + 1] * lda + c] : T(0);
    }
#pragma unroll
    for (int q = 0; q < kB; ++q) {
      const int e = e0 + q * blockDim.y;
      if (on && e < count) vals[e * 32 + threadIdx.x] = v[q];
    }
  }
  __syncthreads();
  for (int e = threadIdx.y; e < count; e += blockDim.y)
    if (on) a[(int64_t)mv[2 * e] * lda + c] = vals[e * 32 + threadIdx.x];
}


// ---------------------------------------------------------------------------
// 3a. Schur update on the CUDA cores (exact mode and FP32): C -= A B with a
//     kTile x kTile tile per CTA, a quarter of kTile / 4 squared elements a
//     thread, K staged in shared memory.  Each C entry starts from its old value
//     and takes the K updates one at a time in increasing k, which is lair's
//     order.  The tile is 64 where that makes two CTAs per SM, else smaller: FP64
//     arithmetic on one SM takes 150 us for a 64 x 64 tile (K = 64, a product and
//     a subtraction), 10 us for a 16 x 16 one.
// ---------------------------------------------------------------------------
constexpr int kGemmKC = 32;  // K chunk staged per pass (static smem stays < 48 KB)

template <typename T, bool kExact, int kTile>
__global__ void __launch_bounds__(256) gemm_cuda_kernel(T* a, int64_t lda, int r0, int c0, int kk0,
                                                        int K, int M, int N) {
  constexpr int kE = kTile / 16;  // elements of a thread in each direction
  __shared__ T As[kGemmKC][kTile + 1];  // As[k][i] = L21[i][k]
  __shared__ T Bs[kGemmKC][kTile];      // Bs[k][j] = U12[k][j]
  const int tile_r = r0 + blockIdx.y * kTile;
  const int tile_c = c0 + blockIdx.x * kTile;
  const int tid = threadIdx.x;
  const int tr = (tid / 16) * kE, tc = (tid % 16);
  T acc[kE][kE];
#pragma unroll
  for (int i = 0; i < kE; ++i)
#pragma unroll
    for (int jj = 0; jj < kE; ++jj) {
      const int r = tile_r + tr + i, c = tile_c + tc + 16 * jj;
      acc[i][jj] = (r < r0 + M && c < c0 + N) ? a[(int64_t)r * lda + c] : T(0);
    }
  for (int kb = 0; kb < K; kb += kGemmKC) {
    const int kc = min(kGemmKC, K - kb);
    __syncthreads();
    for (int idx = tid; idx < kc * kTile; idx += 256) {
      const int i = idx / kc, k = idx - i * kc;
      const int r = tile_r + i;
      As[k][i] = (r < r0 + M) ? a[(int64_t)r * lda + kk0 + kb + k] : T(0);
    }
    for (int idx = tid; idx < kc * kTile; idx += 256) {
      const int k = idx / kTile, j = idx - k * kTile;
      const int c = tile_c + j;
      Bs[k][j] = (c < c0 + N) ? a[(int64_t)(kk0 + kb + k) * lda + c] : T(0);
    }
    __syncthreads();
    for (int k = 0; k < kc; ++k) {
      T av[kE], bv[kE];
#pragma unroll
      for (int i = 0; i < kE; ++i) av[i] = As[k][tr + i];
#pragma unroll
      for (int jj = 0; jj < kE; ++jj) bv[jj] = Bs[k][tc + 16 * jj];
#pragma unroll
      for (int i = 0; i < kE; ++i)
#pragma unroll
        for (int jj = 0; jj < kE; ++jj) acc[i][jj] = upd<kExact>(acc[i][jj], av[i], bv[jj]);
    }
  }
#pragma unroll
  for (int i = 0; i < kE; ++i)
#pragma unroll
    for (int jj = 0; jj < kE; ++jj) {
      const int r = tile_r + tr + i, c = tile_c + tc + 16 * jj;
      if (r < r0 + M && c < c0 + N) a[(int64_t)r * lda + c] = acc[i][jj];
    }
}

// ---------------------------------------------------------------------------
// 3b. Schur update on the FP64 tensor cores: mma.sync.m8n8k4 (DMMA).
//     CTA tile 128x128, 8 warps as 4 (rows) x 2 (cols), warp tile 32x64 =
//     4 x 8 MMA tiles.  L21/U12 slices (K <= 64) are staged in shared memory
//     once; C is read, updated and written once.
// ---------------------------------------------------------------------------
constexpr int kDmmaBM = 128, kDmmaBN = 128;

__device__ __forceinline__ void dmma_8x8x4(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

__global__ void __launch_bounds__(256) gemm_dmma_kernel(double* a, int64_t lda, int r0, int c0,
                                                        int kk0, int K, int M, int N) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  // As: [kDmmaBM][Kp] (row i, col k), Kp = Kpad + 4 keeps the fragment loads
  // free of bank conflicts; Bs: [Kpad][kDmmaBN + 4] likewise.
  const int Kpad = (K + 15) & ~15;
  const int Kp = Kpad + 4;
  double* As = reinterpret_cast<double*>(smem_raw);
  double* Bs = As + kDmmaBM * Kp;
  const int ldb = kDmmaBN + 4;
  const int tile_r = r0 + blockIdx.y * kDmmaBM;
  const int tile_c = c0 + blockIdx.x * kDmmaBN;
  const int tid = threadIdx.x;
  for (int idx = tid; idx < kDmmaBM * Kpad; idx += 256) {
    const int i = idx / Kpad, k = idx - i * Kpad;
    const int r = tile_r + i;
    As[i * Kp + k] = (r < r0 + M && k < K) ? a[(int64_t)r * lda + kk0 + k] : 0.0;
  }
  for (int idx = tid; idx < Kpad * kDmmaBN; idx += 256) {
    const int k = idx / kDmmaBN, j = idx - k * kDmmaBN;
    const int c = tile_c + j;
    Bs[k * ldb + j] = (c < c0 + N && k < K) ? a[(int64_t)(kk0 + k) * lda + c] : 0.0;
  }
  __syncthreads();
  const int lane = tid & 31, warp = tid >> 5;
  const int wr = (warp >> 1) * 32;  // warp row offset in tile
  const int wc = (warp & 1) * 64;   // warp col offset in tile
  const int g = lane >> 2, t4 = lane & 3;
  double acc[4][8][2];
#pragma unroll
  for (int mi = 0; mi < 4; ++mi)
#pragma unroll
    for (int ni = 0; ni < 8; ++ni)
#pragma unroll
      for (int e = 0; e < 2; ++e) acc[mi][ni][e] = 0.0;
  const int Kmma = (K + 3) & ~3;
  for (int k = 0; k < Kmma; k += 4) {
    double af[4], bf[8];
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) af[mi] = As[(wr + mi * 8 + g) * Kp + k + t4];
#pragma unroll
    for (int ni = 0; ni < 8; ++ni) bf[ni] = Bs[(k + t4) * ldb + wc + ni * 8 + g];
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
      for (int ni = 0; ni < 8; ++ni) dmma_8x8x4(acc[mi][ni][0], acc[mi][ni][1], af[mi], bf[ni]);
  }
#pragma unroll
  for (int mi = 0; mi < 4; ++mi) {
    const int r = tile_r + wr + mi * 8 + g;
    if (r >= r0 + M) continue;
#pragma unroll
    for (int ni = 0; ni < 8; ++ni) {
      const int c = tile_c + wc + ni * 8 + t4 * 2;
      double* dst = a + (int64_t)r * lda + c;
      if (c + 1 < c0 + N && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
        double2 v = *reinterpret_cast<double2*>(dst);
        v.x -= acc[mi][ni][0];
        v.y -= acc[mi][ni][1];
        *reinterpret_cast<double2*>(dst) = v;
      } else {
        if (c < c0 + N) dst[0] -= acc[mi][ni][0];
        if (c + 1 < c0 + N) dst[1] -= acc[mi][ni][1];
      }
    }
  }
}

// Persistent form of the same update for aligned operands: one CTA per SM
// walks a contiguous range of 128 x 128 tiles in row-block order, so the
// L21 block (A) changes only when the range crosses a row block.  The next
// tile's U12 block (B) is copied into a second buffer by cp.async while the
// current tile runs on the FP64 pipe, and the C tile is prefetched into L2
// before its read-modify-write.  The FP64 pipe therefore stays busy across
// tile boundaries instead of idling through each tile's loads and stores.
// Needs 16-byte aligned rows and panel columns (even lda, kk0 and c0 and a
// 16-byte aligned base); the launcher falls back to gemm_dmma_kernel.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, int src_bytes) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(src_bytes) : "memory");
}

__global__ void __launch_bounds__(256, 1) gemm_dmma_persistent_kernel(double* a, int64_t lda, int r0, int c0,
                                                                      int kk0, int K, int M, int N) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Kpad = (K + 15) & ~15;
  const int Kp = Kpad + 4;
  const int ldb = kDmmaBN + 4;
  double* As = reinterpret_cast<double*>(smem_raw);  // [128][Kp]
  double* Bs0 = As + kDmmaBM * Kp;                   // [2][Kpad][ldb]
  const int tiles_n = (N + kDmmaBN - 1) / kDmmaBN;
  const int tiles = ((M + kDmmaBM - 1) / kDmmaBM) * tiles_n;
  const int G = gridDim.x;
  const int t_begin = (int)((int64_t)blockIdx.x * tiles / G);
  const int t_end = (int)((int64_t)(blockIdx.x + 1) * tiles / G);
  if (t_begin >= t_end) return;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  const int wr = (warp >> 1) * 32, wc = (warp & 1) * 64;
  const int g = lane >> 2, t4 = lane & 3;
  const int kchunks = Kpad / 2;  // 16-byte chunks per A row

  auto load_a = [&](int tm) {
    const int tile_r = r0 + tm * kDmmaBM;
    for (int idx = tid; idx < kDmmaBM * kchunks; idx += 256) {
      const int i = idx / kchunks, k = (idx - i * kchunks) * 2;
      const int r = tile_r + i;
      const int valid = (r < r0 + M) ? max(0, min(2, K - k)) : 0;
      const double* src = valid ? a + (int64_t)r * lda + kk0 + k : a;
      cp_async16(As + i * Kp + k, src, valid * 8);
    }
  };
  auto load_b = [&](int tn, double* Bs) {
    const int tile_c = c0 + tn * kDmmaBN;
    for (int idx = tid; idx < Kpad * (kDmmaBN / 2); idx += 256) {
      const int k = idx / (kDmmaBN / 2), j = (idx - k * (kDmmaBN / 2)) * 2;
      const int c = tile_c + j;
      const int valid = (k < K) ? max(0, min(2, c0 + N - c)) : 0;
      const double* src = valid ? a + (int64_t)(kk0 + k) * lda + c : a;
      cp_async16(Bs + k * ldb + j, src, valid * 8);
    }
  };

  int tm = t_begin / tiles_n, tn = t_begin - tm * tiles_n;
  load_a(tm);
  load_b(tn, Bs0);
  cp_async_commit();
  for (int t = t_begin; t < t_end; ++t) {
    double* Bs = Bs0 + (size_t)((t - t_begin) & 1) * Kpad * ldb;
    cp_async_wait_all();
    __syncthreads();
    const int tile_r = r0 + tm * kDmmaBM, tile_c = c0 + tn * kDmmaBN;
    // Next tile: its B block now (other buffer, last read two tiles ago).
    int tm_n = tm, tn_n = tn + 1;
    if (tn_n == tiles_n) {
      tn_n = 0;
      ++tm_n;
    }
    const bool more = t + 1 < t_end;
    if (more) {
      load_b(tn_n, Bs0 + (size_t)((t + 1 - t_begin) & 1) * Kpad * ldb);
      cp_async_commit();
    }
    // C tile into L2 ahead of its read-modify-write: 128 rows x 1 KB.
    for (int idx = tid; idx < kDmmaBM * 8; idx += 256) {
      const int i = idx >> 3, part = idx & 7;
      const int r = tile_r + i, c = tile_c + part * 16;
      if (r < r0 + M && c < c0 + N) asm volatile("prefetch.global.L2 [%0];" ::"l"(a + (int64_t)r * lda + c));
    }
    double acc[4][8][2];
#pragma unroll
    for (int mi = 0; mi < 4; ++mi)
#pragma unroll
      for (int ni = 0; ni < 8; ++ni) acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
    const int Kmma = (K + 3) & ~3;
    for (int k = 0; k < Kmma; k += 4) {
      double af[4], bf[8];
#pragma unroll
      for (int mi = 0; mi < 4; ++mi) af[mi] = As[(wr + mi * 8 + g) * Kp + k + t4];
#pragma unroll
      for (int ni = 0; ni < 8; ++ni) bf[ni] = Bs[(k + t4) * ldb + wc + ni * 8 + g];
#pragma unroll
      for (int mi = 0; mi < 4; ++mi)
#pragma unroll
        for (int ni = 0; ni < 8; ++ni) dmma_8x8x4(acc[mi][ni][0], acc[mi][ni][1], af[mi], bf[ni]);
    }
    if (more && tm_n != tm) {
      // The range crosses into the next row block: reload A once every warp
      // is done with it.
      __syncthreads();
      load_a(tm_n);
      cp_async_commit();
    }
#pragma unroll
    for (int mi = 0; mi < 4; ++mi) {
      const int r = tile_r + wr + mi * 8 + g;
      if (r >= r0 + M) continue;
#pragma unroll
      for (int ni = 0; ni < 8; ++ni) {
        const int c = tile_c + wc + ni * 8 + t4 * 2;
        double* dst = a + (int64_t)r * lda + c;
        if (c + 1 < c0 + N) {
          double2 v = *reinterpret_cast<double2*>(dst);
          v.x -= acc[mi][ni][0];
          v.y -= acc[mi][ni][1];
          *reinterpret_cast<double2*>(dst) = v;
        } else if (c < c0 + N) {
          dst[0] -= acc[mi][ni][0];
        }
      }
    }
    tm = tm_n;
    tn = tn_n;
  }
}

// The same product for small blocks: a 16 x 32 tile per CTA, four warps of 8 x 16
// (two MMA tiles each).  One SM's FP64 pipes take 300 us for a 128 x 128 tile at
// K = 64, so blocks of fewer such tiles than SMs are cut finer: a 200 x 200 block
// 302 -> 12 us, 400 x 400 308 -> 24 us.  Any alignment.
constexpr int kSmallBM = 16, kSmallBN = 32;

__global__ void __launch_bounds__(128) gemm_dmma_small_kernel(double* a, int64_t lda, int r0, int c0, int kk0, int K,
                                                              int M, int N) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Kpad = (K + 3) & ~3;
  const int Kp = Kpad + 4;
  constexpr int ldb = kSmallBN + 4;
  double* As = reinterpret_cast<double*>(smem_raw);  // [16][Kp]
  double* Bs = As + kSmallBM * Kp;                   // [Kpad][ldb]
  const int tile_r = r0 + blockIdx.y * kSmallBM, tile_c = c0 + blockIdx.x * kSmallBN;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wr = (warp >> 1) * 8, wc = (warp & 1) * 16;
  const int g = lane >> 2, t4 = lane & 3;
  // C first: its loads overlap those of the operands.
  double cv[2][2];
  const int r = tile_r + wr + g;
#pragma unroll
  for (int ni = 0; ni < 2; ++ni)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int c = tile_c + wc + ni * 8 + t4 * 2 + e;
      cv[ni][e] = (r < r0 + M && c < c0 + N) ? a[(int64_t)r * lda + c] : 0.0;
    }
  for (int idx = tid; idx < kSmallBM * Kpad; idx += 128) {
    const int i = idx / Kpad, k = idx - i * Kpad;
    As[i * Kp + k] = (tile_r + i < r0 + M && k < K) ? a[(int64_t)(tile_r + i) * lda + kk0 + k] : 0.0;
  }
  for (int idx = tid; idx < Kpad * kSmallBN; idx += 128) {
    const int k = idx / kSmallBN, j = idx - k * kSmallBN;
    Bs[k * ldb + j] = (tile_c + j < c0 + N && k < K) ? a[(int64_t)(kk0 + k) * lda + tile_c + j] : 0.0;
  }
  __syncthreads();
  double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
  for (int k = 0; k < Kpad; k += 4) {
    const double af = As[(wr + g) * Kp + k + t4];
#pragma unroll
    for (int ni = 0; ni < 2; ++ni)
      dmma_8x8x4(acc[ni][0], acc[ni][1], af, Bs[(k + t4) * ldb + wc + ni * 8 + g]);
  }
#pragma unroll
  for (int ni = 0; ni < 2; ++ni)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int c = tile_c + wc + ni * 8 + t4 * 2 + e;
      if (r < r0 + M && c < c0 + N) a[(int64_t)r * lda + c] = cv[ni][e] - acc[ni][e];
    }
}

// ---------------------------------------------------------------------------
// Host driver.
// ---------------------------------------------------------------------------
// Shared-memory row stride of the panel: FP64 w + 1 (conflict-free column
// access); FP32 rows padded to a multiple of 4 floats plus 4, so every row
// starts on 16 bytes for the float4 look-ahead (column access then has
// 4-way bank conflicts, a small cost on two columns a step).
template <typename T>
static int panel_lds(int w) {
  return sizeof(T) == 4 ? ((w + 3) & ~3) + 4 : w + 1;
}
// Threads of a panel CTA: 16 warps hide the look-ahead's shared-memory latency
// (FP64, 8 warps against 16: 207 / 200 us at 8192 rows, 270 / 229 at 16384).
constexpr int kPanelThreads = 512;
template <typename T>
static size_t panel_smem_bytes(int rows_per, int w) {
  return ((size_t)rows_per * panel_lds<T>(w) + 2 * kMaxPanelWidth) * sizeof(T) + 2 * (size_t)rows_per * sizeof(int);
}

// (Exact FP64: 64 / 40 rows a CTA at least, 242 / 230 us at 2500 and 4000 rows.)
template <typename T>
static int panel_ctas(luhot_ctx* ctx, int rows, bool exact = false) {
  const int pmax = std::min(ctx->num_sms, sizeof(T) == 4 ? 64 : 96);
  const int min_rows = sizeof(T) == 4 ? 32 : exact ? 40 : 64;
  return std::min(pmax, std::max(1, (rows + min_rows - 1) / min_rows));
}

// Where a panel reports its moved rows unless told otherwise.
static int* live_moves(luhot_ctx* ctx) {
  return reinterpret_cast<int*>(static_cast<char*>(ctx->panel_scratch) + kPanelSlotBytes);
}

template <typename T, bool kExact>
static int launch_panel(luhot_ctx* ctx, T* a, int64_t lda, int m, int k0, int w, int* piv, cudaStream_t stream,
                        int* moves = nullptr) {
  const int rows = m - k0;
  if (!moves) moves = live_moves(ctx);
  if (panel_cluster_fits<T, kExact>(ctx, rows, w))
    return launch_panel_cluster<T, kExact>(ctx, a, lda, m, k0, w, piv, moves, stream);
  auto kern = panel_kernel<T, kExact>;
  cudaFuncAttributes fa;
  LUHOT_CUDA_TRY(ctx, cudaFuncGetAttributes(&fa, kern));
  const int max_smem = ctx->max_smem_optin - (int)fa.sharedSizeBytes;  // less the static exchange buffers
  // CTAs: FP32 panels (light update work) run fastest on 64 CTAs with >= 32
  // rows each; FP64 panels, whose look-ahead update needs FP64 pipes, on 96
  // CTAs with >= 64 rows each (measured at n = 16384 against 64 .. 152 CTAs:
  // fewer CTAs shorten the per-column exchange, more share the update).  The
  // count is raised, up to the SM count, when the rows of one CTA would not
  // fit in shared memory.
  int P = panel_ctas<T>(ctx, rows, kExact);
  int rows_per = (rows + P - 1) / P;
  while (panel_smem_bytes<T>(rows_per, w) > (size_t)max_smem && P < ctx->num_sms) {
    P = std::min(ctx->num_sms, P * 2);
    rows_per = (rows + P - 1) / P;
  }
  if (panel_smem_bytes<T>(rows_per, w) > (size_t)max_smem)
    return set_error(ctx, LUHOT_ERR_UNSUPPORTED, "panel does not fit in shared memory");
  const size_t smem = panel_smem_bytes<T>(rows_per, w);
  LUHOT_CUDA_TRY(ctx, allow_max_dynamic_smem(kern));
  int per_sm = 0;
  LUHOT_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kPanelThreads, smem));
  if (per_sm * ctx->num_sms < P)
    return set_error(ctx, LUHOT_ERR_UNSUPPORTED, "panel grid cannot be co-resident");
  PanelArgs<T> args;
  args.a = a;
  args.lda = lda;
  args.m = m;
  args.k0 = k0;
  args.w = w;
  args.rows_per = rows_per;
  args.lds = panel_lds<T>(w);
  args.piv = piv;
  args.heads = static_cast<unsigned long long*>(ctx->panel_scratch);
  args.slots = args.heads + 2 * (size_t)kMaxPanelCtas * kPanelHeaderWords;
  args.moves = moves;
  args.move_count = args.moves + 4 * kMaxPanelWidth;
  args.st = ctx->d_status;
  LUHOT_CUDA_TRY(ctx, cudaMemsetAsync(args.move_count, 0, sizeof(int), stream));
  void* kargs[] = {&args};
  prof_begin(ctx, kProfPanel);
  LUHOT_CUDA_TRY(ctx, cudaLaunchCooperativeKernel((void*)kern, dim3(P), dim3(kPanelThreads), kargs, smem,
                                                  stream));
  // panel flops: sum over steps of (rows below) * (1 + 2 * cols right)
  double fl = 0.0;
  for (int j = 0; j < w; ++j) fl += (double)(rows - j - 1) * (1.0 + 2.0 * (w - j - 1));
  prof_end(ctx, kProfPanel, fl, 2.0 * rows * w * sizeof(T));
  return LUHOT_OK;
}

template <typename T, bool kExact>
static int launch_gemm(luhot_ctx* ctx, T* a, int64_t lda, int r0, int c0, int kk0, int K, int M,
                       int N, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return LUHOT_OK;
  if constexpr (std::is_same<T, double>::value && !kExact) {
    const int Kpad = (K + 15) & ~15;
    const size_t smem = ((size_t)kDmmaBM * (Kpad + 4) + (size_t)Kpad * (kDmmaBN + 4)) * sizeof(double);
    const size_t smem_p = smem + (size_t)Kpad * (kDmmaBN + 4) * sizeof(double);
    const int tiles = ((N + kDmmaBN - 1) / kDmmaBN) * ((M + kDmmaBM - 1) / kDmmaBM);
    if (tiles < ctx->num_sms) {
      const int Kq = (K + 3) & ~3;
      const size_t smem_s = ((size_t)kSmallBM * (Kq + 4) + (size_t)Kq * (kSmallBN + 4)) * sizeof(double);
      LUHOT_CUDA_TRY(ctx, allow_max_dynamic_smem(gemm_dmma_small_kernel));
      dim3 grid((N + kSmallBN - 1) / kSmallBN, (M + kSmallBM - 1) / kSmallBM);
      prof_begin(ctx, kProfGemm);
      gemm_dmma_small_kernel<<<grid, 128, smem_s, stream>>>(a, lda, r0, c0, kk0, K, M, N);
      prof_end(ctx, kProfGemm, 2.0 * M * N * K, ((double)2 * M * N + (double)M * K + (double)K * N) * sizeof(T));
      LUHOT_CUDA_TRY(ctx, cudaGetLastError());
      return LUHOT_OK;
    }
    const bool aligned = (lda % 2 == 0) && (kk0 % 2 == 0) && (c0 % 2 == 0) &&
                         (reinterpret_cast<uintptr_t>(a) % 16 == 0);
    if (aligned && smem_p <= (size_t)ctx->max_smem_optin) {
      LUHOT_CUDA_TRY(ctx, allow_max_dynamic_smem(gemm_dmma_persistent_kernel));
      prof_begin(ctx, kProfGemm);
      gemm_dmma_persistent_kernel<<<std::min(tiles, ctx->tc_grid_cap > 0 ? ctx->tc_grid_cap : ctx->num_sms), 256, smem_p, stream>>>(a, lda, r0, c0, kk0, K,
                                                                                          M, N);
    } else {
      LUHOT_CUDA_TRY(ctx, allow_max_dynamic_smem(gemm_dmma_kernel));
      dim3 grid((N + kDmmaBN - 1) / kDmmaBN, (M + kDmmaBM - 1) / kDmmaBM);
      prof_begin(ctx, kProfGemm);
      gemm_dmma_kernel<<<grid, 256, smem, stream>>>(a, lda, r0, c0, kk0, K, M, N);
    }
  } else {
    auto ctas = [&](int t) { return (int64_t)((N + t - 1) / t) * ((M + t - 1) / t); };
    const int tile = ctas(64) >= 2 * ctx->num_sms ? 64 : (ctas(32) >= 2 * ctx->num_sms || sizeof(T) == 4) ? 32 : 16;
    dim3 grid((N + tile - 1) / tile, (M + tile - 1) / tile);
    prof_begin(ctx, kProfGemm);
    if (tile == 64)
      gemm_cuda_kernel<T, kExact, 64><<<grid, 256, 0, stream>>>(a, lda, r0, c0, kk0, K, M, N);
    else if (tile == 32)
      gemm_cuda_kernel<T, kExact, 32><<<grid, 256, 0, stream>>>(a, lda, r0, c0, kk0, K, M, N);
    else
      gemm_cuda_kernel<T, kExact, 16><<<grid, 256, 0, stream>>>(a, lda, r0, c0, kk0, K, M, N);
  }
  // algorithmic work: 2MNK flops; bytes: C read + written, L21 and U12 read once
  prof_end(ctx, kProfGemm, 2.0 * M * N * K,
           ((double)2 * M * N + (double)M * K + (double)K * N) * sizeof(T));
  LUHOT_CUDA_TRY(ctx, cudaGetLastError());
  return LUHOT_OK;
}

// Row interchanges of a panel of width w, from the list of moved rows it
// reported (`moves`: kPanelMovesBytes, the layout of the panel scratch), on
// the columns [cl0, cl1) and [cr0, cr1).
template <typename T>
static int launch_laswp_cols(luhot_ctx* ctx, T* a, int64_t lda, const int* moves, int w, int cl0, int cl1, int cr0,
                             int cr1, cudaStream_t stream) {
  const int ncols_swap = std::max(0, cl1 - cl0) + std::max(0, cr1 - cr0);
  if (ncols_swap <= 0) return LUHOT_OK;
  prof_begin(ctx, kProfLaswp);
  const size_t lsm = (size_t)2 * w * 32 * sizeof(T);
  LUHOT_CUDA_TRY(ctx, allow_max_dynamic_smem(laswp_moves_kernel<T>));
  laswp_moves_kernel<T><<<(ncols_swap + 31) / 32, dim3(32, 8), lsm, stream>>>(
      a, lda, moves, moves + 4 * kMaxPanelWidth, 2 * w, cl0, std::max(cl0, cl1), cr0, std::max(cr0, cr1));
  prof_end(ctx, kProfLaswp, 0.0, 4.0 * w * ncols_swap * sizeof(T));
  LUHOT_CUDA_TRY(ctx, cudaGetLastError());
  return LUHOT_OK;
}

// Whether the update of a trailing block of M rows and N columns runs on the FP16
// tensor cores as slice products (ozaki.cu).  M and N are those of the whole block
// behind a panel, whatever part of it a launch takes: an element's digits come from
// its row of L21 and its column of U12 alone, so that every part gives the same bits.
// AUTO takes blocks of at least 256 x 256.  Smaller ones would gain a little (one
// product takes some 8 us for up to a tile of 64 x 128 per SM, FP64 arithmetic 9 us
// for the tile of 16 x 32 that each SM takes at 128 000 elements; factorizations of
// n = 500 0.745 against 0.780 ms with the line at 25 000 / 200 000 elements, 1000
// 1.685 / 1.715), but slices hold the elements relative to the largest of their row or
// column, where FP64 arithmetic holds each to its own 53 bits.
static bool update_on_slices(const void* oz_ws, int engine, int M, int N) {
  if (!oz_ws || engine == LUHOT_UPDATE_DMMA) return false;
  return engine == LUHOT_UPDATE_OZAKI ? M >= 128 && N >= 64 : M >= 256 && N >= 256;
}

// Workspace of the tensor-core FP64 update for an m x n factorization
// (nullptr: the engine setting or the device rules it out).
static int ozaki_workspace(luhot_ctx* ctx, int m, int n, int engine, void** ws, int n2 = 0, void** ws2 = nullptr) {
  *ws = nullptr;
  if (engine == LUHOT_UPDATE_DMMA || !ozaki_available(ctx)) return LUHOT_OK;
  const size_t bytes = (ozaki_workspace_bytes(m, n) + 1023) / 1024 * 1024;
  int rc = ensure_buf(ctx, ctx->oz_buf, bytes + (n2 > 0 ? ozaki_workspace_bytes(m, n2) : 0));
  if (rc != LUHOT_OK) return rc;
  *ws = ctx->oz_buf.ptr;
  if (ws2) *ws2 = static_cast<char*>(ctx->oz_buf.ptr) + bytes;
  return LUHOT_OK;
}

int fp64_schur_update(luhot_ctx* ctx, double* a, int64_t lda, int k, int m, int n, int engine) {
  void* ws = nullptr;
  int rc = ozaki_workspace(ctx, m, n, engine, &ws);
  if (rc) return rc;
  if (update_on_slices(ws, engine, m - k, n - k)) return ozaki_update(ctx, a, lda, 0, k, k, m, k, n, ws, ctx->stream);
  return launch_gemm<double, false>(ctx, a, lda, k, k, 0, k, m - k, n - k, ctx->stream);
}

// Two panels [k0, k0 + 64), [k0 + 64, k0 + 128) of fast-mode FP64 and one trailing
// update with K = 128: a slice product's time is its epilogue's, which a pair pays
// once.  In between, the second panel's columns and the second panel's rows of U
// take K = 64 products of their own and the interchanges two launches, some 40 us
// in all, so that the pair pays from about 4000 x 4000 on (kPairElems: the block
// behind the pair).  n = 16384: updates 114 -> 75 ms, 193 -> 159 ms in all; n = 4097
// (31 pairs smaller than the rule's limit): 15.65 ms without, 15.59 with pairs from
// 3000 x 3000 on, 15.8 from 2000 x 2000 on.
constexpr int64_t kPairElems = 16000000;

static int fp64_panel_pair(luhot_ctx* ctx, double* a, int64_t lda, int m, int n, int k0, int* piv, void* oz_ws,
                           cudaStream_t stream) {
  constexpr int w = kDefaultPanelWidth;
  const int k1 = k0 + w, r1 = k1 + w, N = n - r1;
  int rc = ensure_buf(ctx, ctx->la_moves, 4 * kPanelMovesBytes);
  if (rc) return rc;
  int* mv = static_cast<int*>(ctx->la_moves.ptr);
  double* const ab = a + (int64_t)k1 * lda;  // row k1
  // The first panel's interchanges on the other columns come after the second's
  // columns are done: its list is kept apart.
  rc = launch_panel<double, false>(ctx, a, lda, m, k0, w, piv, stream, mv);
  if (rc) return rc;
  const SplitOut split = ozaki_split_out(oz_ws, k1, m - k1, w);
  rc = launch_swap_solve<double, false>(ctx, a, lda, mv, k0, w, 0, 0, k1, r1, &split, stream);
  if (!rc) rc = ozaki_update_split(ctx, a, lda, w, k1, m, k1, r1, oz_ws, stream);
  if (!rc) rc = launch_panel<double, false>(ctx, a, lda, m, k1, w, piv, stream);
  if (!rc) rc = launch_swap_solve<double, false>(ctx, a, lda, mv, k0, w, 0, k0, r1, n, nullptr, stream);
  if (!rc) rc = launch_laswp_cols<double>(ctx, a, lda, live_moves(ctx), w, 0, k1, r1, n, stream);
  if (!rc) rc = ozaki_product(ctx, ab + k0, lda, a + (int64_t)k0 * lda + r1, lda, w, ab + r1, lda, w, N, oz_ws, stream);
  if (!rc) rc = launch_swap_solve<double, false>(ctx, a, lda, nullptr, k1, w, 0, 0, r1, n, nullptr, stream);
  if (!rc) rc = ozaki_update(ctx, a, lda, k0, 2 * w, r1, m, r1, n, oz_ws, stream);
  return rc;
}

static int* la_saved_moves(luhot_ctx* ctx, int parity, int half) {
  return reinterpret_cast<int*>(static_cast<char*>(ctx->la_moves.ptr) + (size_t)(2 * parity + half) * kPanelMovesBytes);
}

// Launches between its construction and destruction go to `s` (the
// profile's events are recorded on the context's stream).
struct OnStream {
  luhot_ctx* ctx;
  cudaStream_t old;
  OnStream(luhot_ctx* c, cudaStream_t s) : ctx(c), old(c->stream) { c->stream = s; }
  ~OnStream() { ctx->stream = old; }
};

static int la_setup(luhot_ctx* ctx) {
  if (!ctx->la_hi) {
    int least = 0, greatest = 0;
    LUHOT_CUDA_TRY(ctx, cudaDeviceGetStreamPriorityRange(&least, &greatest));
    LUHOT_CUDA_TRY(ctx, cudaStreamCreateWithPriority(&ctx->la_lo, cudaStreamNonBlocking, least));
    LUHOT_CUDA_TRY(ctx, cudaStreamCreateWithPriority(&ctx->la_hi, cudaStreamNonBlocking, greatest));
  }
  for (auto& e : ctx->la_ev)
    if (!e) LUHOT_CUDA_TRY(ctx, cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  return ensure_buf(ctx, ctx->la_moves, 4 * kPanelMovesBytes);
}

// Look-ahead: panel k + 1 beside the rest of step k.  A high-priority stream (hs)
// factors the panels and brings each next panel's columns up to date; a
// low-priority one (ls) does the rest of the step (interchanges, rows of U, update
// of the columns behind the next panel) on the SMs that the next panel leaves.
// hs waits for the rest of step k - 1 before it touches step k + 1's columns,
// so that at most two steps are under way; their lists of moved rows alternate.
// Takes the steps from k0 on while la_pays; returns the first one it left in k0.
// The price is two launches more a step on the panels' way, some 40 us, so that it
// pays while the block behind the next panel is large.  FP64 updates are persistent
// kernels on the SMs that the panel leaves, so that it pays, besides, while rest +
// panel in turn take longer than the rest on those alone (rest P <= panel (SMs - P)):
// not beside a panel on many SMs when the update is long (n = 16384, DMMA updates:
// 2.9 s in turn, 7.5 s beside 96-CTA panels).  us: a panel as measured; an element of
// an update by slices 5.0e-6, by DMMA 1.16e-4.  FP32 updates are many short CTAs, which
// take what is free (n = 16384: 171 ms in turn until panels are a cluster's, 162 beside).
// ms, FP64 / FP32, step by step against with look-ahead: n = 1000 1.69 -> 1.69 (1.71 with
// a limit of 500000) / 1.25 -> 1.25, 2000 4.29 -> 4.17 / 3.07 -> 2.86, 3000 8.07 -> 7.41 /
// 5.36 -> 4.56.
template <typename T>
static bool la_pays(luhot_ctx* ctx, const void* oz_ws, int m, int n, int k0, int nb) {
  const int64_t M = m - k0 - 2 * nb, N = n - k0 - 2 * nb;
  if (M <= 0 || N <= 0) return false;
  if (sizeof(T) == 4) return M * N >= 500000;
  if (M * N < 1000000) return false;
  const int rows = m - k0 - nb;
  const bool cluster = panel_cluster_fits<T, false>(ctx, rows, nb);
  const int P = cluster ? ctx->panel_cluster : panel_ctas<T>(ctx, rows);
  const bool slices = update_on_slices(oz_ws, ctx->fp64_update, rows, n - k0 - nb);
  const double rest = (double)M * N * (slices ? 5.0e-6 : 1.16e-4) * nb / 64;
  return rest * P <= (cluster ? 100.0 : 200.0) * (ctx->num_sms - P);
}

template <typename T>
static int la_loop(luhot_ctx* ctx, int m, int n, T* a, int64_t lda, int* piv, int nb, void* oz_ws, void* oz_hi,
                   int* k0_io) {
  cudaStream_t hs = ctx->la_hi, ls = ctx->la_lo;
  // Columns [c0, c1) of step k0: interchanges (also on [0, cl1)), rows of U, update.
  auto columns = [&](const int* mv, int k0, int cl1, int c0, int c1, void* ws, cudaStream_t st) -> int {
    const int r1 = k0 + nb, M = m - r1, N = c1 - c0;
    const bool slices = std::is_same<T, double>::value && update_on_slices(ws, ctx->fp64_update, M, n - r1);
    SplitOut split;
    if (slices) split = ozaki_split_out(ws, r1, M, N);
    int rc = launch_swap_solve<T, false>(ctx, a, lda, mv, k0, nb, 0, cl1, c0, c1, slices ? &split : nullptr, st);
    if (rc) return rc;
    if constexpr (std::is_same<T, double>::value) {
      if (slices) return ozaki_update_split(ctx, a, lda, nb, r1, m, c0, c1, ws, st);
    }
    return launch_gemm<T, false>(ctx, a, lda, r1, c0, k0, nb, M, N, st);
  };
  int k0 = *k0_io;
  for (int step = 0; la_pays<T>(ctx, oz_ws, m, n, k0, nb); ++step, k0 += nb) {
    const int par = step & 1, k1 = k0 + nb, e1 = k1 + nb;
    int* mv = la_saved_moves(ctx, par, 0);
    {
      OnStream on(ctx, hs);
      int rc = launch_panel<T, false>(ctx, a, lda, m, k0, nb, piv, hs, mv);
      if (rc) return rc;
      if (step > 0) LUHOT_CUDA_TRY(ctx, cudaStreamWaitEvent(hs, ctx->la_ev[2 + (par ^ 1)], 0));
      rc = columns(mv, k0, 0, k1, e1, oz_hi, hs);
      if (rc) return rc;
      LUHOT_CUDA_TRY(ctx, cudaEventRecord(ctx->la_ev[1], hs));
    }
    {
      OnStream on(ctx, ls);
      LUHOT_CUDA_TRY(ctx, cudaStreamWaitEvent(ls, ctx->la_ev[1], 0));
      ctx->tc_grid_cap =
          std::max(1, ctx->num_sms - (panel_cluster_fits<T, false>(ctx, m - k1, nb) ? ctx->panel_cluster : panel_ctas<T>(ctx, m - k1)));
      const int rc = columns(mv, k0, k0, e1, n, oz_ws, ls);
      ctx->tc_grid_cap = 0;
      if (rc) return rc;
      LUHOT_CUDA_TRY(ctx, cudaEventRecord(ctx->la_ev[2 + par], ls));
    }
  }
  *k0_io = k0;
  return LUHOT_OK;
}

// `run` on the look-ahead streams, behind what is on `stream` and before what
// comes on it next (also after an error).
template <typename F>
static int la_fork_join(luhot_ctx* ctx, cudaStream_t stream, F run) {
  int rc = la_setup(ctx);
  if (rc) return rc;
  LUHOT_CUDA_TRY(ctx, cudaEventRecord(ctx->la_ev[0], stream));
  LUHOT_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->la_hi, ctx->la_ev[0], 0));
  LUHOT_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->la_lo, ctx->la_ev[0], 0));
  rc = run();
  ctx->tc_grid_cap = 0;
  cudaError_t e = cudaEventRecord(ctx->la_ev[0], ctx->la_hi);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, ctx->la_ev[0], 0);
  if (e == cudaSuccess) e = cudaEventRecord(ctx->la_ev[1], ctx->la_lo);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(stream, ctx->la_ev[1], 0);
  if (rc) return rc;
  if (e != cudaSuccess) return set_error(ctx, LUHOT_ERR_CUDA, std::string("look-ahead join: ") + cudaGetErrorString(e));
  return LUHOT_OK;
}

template <typename T, bool kExact>
static int getrf_impl(luhot_ctx* ctx, int m, int n, T* a, int64_t lda, int* piv, int nb, void* oz_ws, void* oz_hi,
                      cudaStream_t stream) {
  const int dim_min = std::min(m, n);
  // Exchange words carry step tags; clear them so no word of an earlier
  // factorization carries a live tag.  Cluster panels exchange none, and once a panel
  // fits a cluster all that follow do.
  if (!panel_cluster_fits<T, kExact>(ctx, m, nb))
    LUHOT_CUDA_TRY(ctx, cudaMemsetAsync(ctx->panel_scratch, 0, kPanelScratchBytes, stream));
  for (int k0 = 0; k0 < dim_min; k0 += nb) {
    if constexpr (std::is_same<T, double>::value && !kExact) {
      const int64_t M2 = m - k0 - 2 * nb, N2 = n - k0 - 2 * nb;
      if (nb == kDefaultPanelWidth && oz_ws && ctx->fp64_update != LUHOT_UPDATE_DMMA && dim_min - k0 >= 2 * nb &&
          M2 > 0 && N2 > 0 && M2 * N2 >= kPairElems) {
        int rc = fp64_panel_pair(ctx, a, lda, m, n, k0, piv, oz_ws, stream);
        if (rc) return rc;
        k0 += nb;  // and the loop's own step
        continue;
      }
    }
    if constexpr (!kExact) {
      if (la_pays<T>(ctx, oz_ws, m, n, k0, nb)) {
        int rc = la_fork_join(ctx, stream, [&] { return la_loop<T>(ctx, m, n, a, lda, piv, nb, oz_ws, oz_hi, &k0); });
        if (rc) return rc;
      }
    }
    const int w = std::min(nb, dim_min - k0);
    int rc = launch_panel<T, kExact>(ctx, a, lda, m, k0, w, piv, stream);
    if (rc) return rc;
    // Everything between the panel and the update in one launch, then the
    // update: on the FP16 tensor cores (fast FP64, large blocks), whose operand
    // slices that launch has written, else FP64 / FP32 arithmetic.
    const int r1 = k0 + w, M = m - r1, N = n - r1;
    const bool slices = !kExact && std::is_same<T, double>::value && w <= 64 &&
                        update_on_slices(oz_ws, ctx->fp64_update, M, N);
    SplitOut split;
    if (slices) split = ozaki_split_out(oz_ws, r1, M, N);
    rc = launch_swap_solve<T, kExact>(ctx, a, lda, live_moves(ctx), k0, w, 0, k0, r1, n, slices ? &split : nullptr,
                                      stream);
    if (rc) return rc;
    if constexpr (std::is_same<T, double>::value && !kExact) {
      if (slices) {
        rc = ozaki_update_split(ctx, a, lda, w, r1, m, r1, n, oz_ws, stream);
        if (rc) return rc;
        continue;
      }
    }
    rc = launch_gemm<T, kExact>(ctx, a, lda, r1, r1, k0, w, M, N, stream);
    if (rc) return rc;
  }
  return LUHOT_OK;
}

// The tensor-core factorization in slabs of two 128-column panels: the
// trailing matrix is updated once per slab (K = 256), which halves its reads
// and writes, the bound of that update.  The two K = 128 updates inside a
// slab (128 columns, or 128 rows) run as FP32 CUDA-core GEMMs: one launch
// each, at least as accurate as any of the tensor-core operand formats.
//
// Look-ahead: the trailing update of slab s is cut at the next slab's
// columns.  A high-priority stream (hs) factors slab s (panels A and B,
// their interchanges on the slab's own columns, the K = 128 step between
// them), then brings the next slab's columns up to date (interchanges, rows
// of U, update).  A low-priority stream (ls) then does the rest of slab s:
// its interchanges on the columns left of it and right of the next slab,
// the rows of U there and the update of those columns, on at most SM count
// - 64 CTAs, so that slab s + 1's panels (64 CTAs) run beside it.  hs waits
// for the rest of slab s - 2 before slab s's panels (it covered slab s's
// columns) and for the rest of slab s - 1 before the next slab's columns.
// Each panel's list of moved rows is saved per slab parity for ls.
// The slab's interchanges (mv_a, mv_b: its panels' moved rows) on the columns
// [cl0, cl1) and [c0, c1); rows [s0, s1) of U on the columns [c0, c1) (two
// solves with the K = 128 update of panel B's rows between them), then the
// update of rows [s1, m) x columns [c0, c1) on the tensor cores (K = s1 - s0).
static int slab_columns(luhot_ctx* ctx, float* a, int64_t lda, int m, int s0, int h0, int h1, const int* mv_a,
                        const int* mv_b, int cl0, int cl1, int c0, int c1, int tc_kind, void* tc_a, void* tc_b,
                        float* tc_scal, cudaStream_t st) {
  if (c0 >= c1) {  // no columns to the right: the interchanges on the left alone
    int rc = launch_laswp_cols<float>(ctx, a, lda, mv_a, h0, cl0, cl1, 0, 0, st);
    if (!rc && h1 > 0) rc = launch_laswp_cols<float>(ctx, a, lda, mv_b, h1, cl0, cl1, 0, 0, st);
    return rc;
  }
  int rc = launch_swap_solve<float, false>(ctx, a, lda, mv_a, s0, h0, cl0, cl1, c0, c1, nullptr, st);
  if (!rc && h1 > 0) {
    rc = launch_laswp_cols<float>(ctx, a, lda, mv_b, h1, cl0, cl1, c0, c1, st);
    if (!rc) rc = launch_gemm<float, false>(ctx, a, lda, s0 + h0, c0, s0, h0, h1, c1 - c0, st);
    if (!rc) rc = launch_swap_solve<float, false>(ctx, a, lda, nullptr, s0 + h0, h1, 0, 0, c0, c1, nullptr, st);
  }
  const int s1 = s0 + h0 + h1;
  if (!rc) rc = tc_gemm_update(ctx, tc_kind, a, lda, s0, h0 + h1, s1, m, c0, c1, tc_a, tc_b, tc_scal, st);
  return rc;
}

static int tc_slab_loop(luhot_ctx* ctx, int m, int n, float* a, int64_t lda, int* piv, int tc_kind, void* tc_a,
                        void* tc_b, float* tc_scal) {
  const int dim_min = std::min(m, n);
  cudaStream_t hs = ctx->la_hi, ls = ctx->la_lo;
  cudaEvent_t ev_ready = ctx->la_ev[1];
  constexpr int hw = kTcPanelWidth, sl = 2 * hw;
  const int cap_rest = std::max(1, ctx->num_sms - 64);
  int slab = 0;
  for (int s0 = 0; s0 < dim_min; s0 += sl, ++slab) {
    const int sw = std::min(sl, dim_min - s0);
    const int h0 = std::min(hw, sw), h1 = sw - h0;
    const int s1 = s0 + sw;
    const int e1 = std::min(n, s1 + sl);  // the next slab's columns: [s1, e1)
    const int par = slab & 1;
    int* mv_a = la_saved_moves(ctx, par, 0);
    int* mv_b = la_saved_moves(ctx, par, 1);
    {
      OnStream on(ctx, hs);
      if (slab >= 2) LUHOT_CUDA_TRY(ctx, cudaStreamWaitEvent(hs, ctx->la_ev[2 + par], 0));
      int rc = launch_panel<float, false>(ctx, a, lda, m, s0, h0, piv, hs, mv_a);
      if (rc) return rc;
      if (h1 > 0) {
        rc = launch_swap_solve<float, false>(ctx, a, lda, mv_a, s0, h0, 0, 0, s0 + h0, s1, nullptr, hs);
        if (!rc) rc = launch_gemm<float, false>(ctx, a, lda, s0 + h0, s0 + h0, s0, h0, m - (s0 + h0), h1, hs);
        if (!rc) rc = launch_panel<float, false>(ctx, a, lda, m, s0 + h0, h1, piv, hs, mv_b);
        if (!rc) rc = launch_laswp_cols<float>(ctx, a, lda, mv_b, h1, s0, s0 + h0, 0, 0, hs);
      }
      if (!rc && s1 < e1) {
        if (slab >= 1) LUHOT_CUDA_TRY(ctx, cudaStreamWaitEvent(hs, ctx->la_ev[2 + (par ^ 1)], 0));
        rc = slab_columns(ctx, a, lda, m, s0, h0, h1, mv_a, mv_b, 0, 0, s1, e1, tc_kind, tc_a, tc_b, tc_scal, hs);
      }
      if (rc) return rc;
      LUHOT_CUDA_TRY(ctx, cudaEventRecord(ev_ready, hs));
    }
    {
      OnStream on(ctx, ls);
      LUHOT_CUDA_TRY(ctx, cudaStreamWaitEvent(ls, ev_ready, 0));
      ctx->tc_grid_cap = cap_rest;
      int rc = slab_columns(ctx, a, lda, m, s0, h0, h1, mv_a, mv_b, 0, s0, e1, n, tc_kind, tc_a, tc_b, tc_scal, ls);
      ctx->tc_grid_cap = 0;
      if (rc) return rc;
      LUHOT_CUDA_TRY(ctx, cudaEventRecord(ctx->la_ev[2 + par], ls));
    }
  }
  return LUHOT_OK;
}

static int getrf_tc_slabs(luhot_ctx* ctx, int m, int n, float* a, int64_t lda, int* piv, int tc_kind, void* tc_a,
                          void* tc_b, float* tc_scal, cudaStream_t stream) {
  LUHOT_CUDA_TRY(ctx, cudaMemsetAsync(ctx->panel_scratch, 0, kPanelScratchBytes, stream));
  return la_fork_join(ctx, stream,
                      [&] { return tc_slab_loop(ctx, m, n, a, lda, piv, tc_kind, tc_a, tc_b, tc_scal); });
}

template <typename T>
int getrf_device(luhot_ctx* ctx, int m, int n, T* a, int64_t lda, int* piv, int mode,
                 int64_t* singular) {
  if (m < 0 || n < 0 || lda < std::max(1, n)) return set_error(ctx, LUHOT_ERR_INVALID_ARG, "getrf: bad shape or lda");
  if (singular) *singular = -1;
  if (m == 0 || n == 0) return LUHOT_OK;
  cudaStream_t stream = ctx->stream;
  int rc = reset_status(ctx);
  if (rc != LUHOT_OK) return rc;
  int nb = ctx->nb_override > 0 ? std::min(ctx->nb_override, kDefaultPanelWidth) : kDefaultPanelWidth;
  // A matrix of at most 128 columns (and at least as many rows) is one panel
  // when the cluster holds it: one launch, no interchanges, solves or updates
  // outside it (n = 100: 0.10 ms, as two panels of 64 and 36 columns 0.63).  Up to 512
  // (FP64) or 2048 rows: from there on the bulk of a wide panel's updates is slower
  // in one cluster than outside (2048 x 128: FP64 0.48 ms as one panel, 0.32 as two;
  // FP32 0.20 either way).
  if (ctx->nb_override <= 0 && n <= kMaxPanelWidth && m >= n && m <= (sizeof(T) == 8 ? 512 : 2048) &&
      (mode == LUHOT_MODE_EXACT ? panel_cluster_fits<T, true>(ctx, m, n) : panel_cluster_fits<T, false>(ctx, m, n)))
    nb = kMaxPanelWidth;
  void *oz_ws = nullptr, *oz_hi = nullptr;
  if (std::is_same<T, double>::value && mode != LUHOT_MODE_EXACT) {
    rc = ozaki_workspace(ctx, m, n, ctx->fp64_update, &oz_ws, kDefaultPanelWidth, &oz_hi);
    if (rc != LUHOT_OK) return rc;
  }
  if (mode == LUHOT_MODE_EXACT)
    rc = getrf_impl<T, true>(ctx, m, n, a, lda, piv, nb, nullptr, nullptr, stream);
  else
    rc = getrf_impl<T, false>(ctx, m, n, a, lda, piv, nb, oz_ws, oz_hi, stream);
  if (rc != LUHOT_OK) return rc;
  return finish_status(ctx, singular);
}

template int getrf_device<double>(luhot_ctx*, int, int, double*, int64_t, int*, int, int64_t*);
template int getrf_device<float>(luhot_ctx*, int, int, float*, int64_t, int*, int, int64_t*);

int getrf_device_tc(luhot_ctx* ctx, int m, int n, float* a, int64_t lda, int* piv, int tc_kind, int64_t* singular) {
  if (m < 0 || n < 0 || lda < std::max(1, n)) return set_error(ctx, LUHOT_ERR_INVALID_ARG, "getrf: bad shape or lda");
  if (singular) *singular = -1;
  if (m == 0 || n == 0) return LUHOT_OK;
  const int nb = 2 * kTcPanelWidth;  // a slab's K
  const size_t bytes = tc_operand_bytes(tc_kind, m, nb) + tc_operand_bytes(tc_kind, n, nb) + 4096;
  int rc = ensure_buf(ctx, ctx->tc_buf, bytes);
  if (rc) return rc;
  char* base = static_cast<char*>(ctx->tc_buf.ptr);
  void* tc_a = base;
  void* tc_b = base + (tc_operand_bytes(tc_kind, m, nb) + 1023) / 1024 * 1024;
  float* tc_scal = reinterpret_cast<float*>(base + bytes - 1024);
  rc = reset_status(ctx);
  if (rc != LUHOT_OK) return rc;
  rc = getrf_tc_slabs(ctx, m, n, a, lda, piv, tc_kind, tc_a, tc_b, tc_scal, ctx->stream);
  if (rc != LUHOT_OK) return rc;
  return finish_status(ctx, singular);
}

}  // namespace luhot
