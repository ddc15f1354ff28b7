// Panel factorization by one thread-block cluster (up to 16 CTAs), for panels
// whose rows fit in the cluster's shared memory.
//
// The rows [k0, m) x columns [k0, k0 + w) are spread over the CTAs and held in
// shared memory for the whole panel; rows never move, an interchange swaps the
// global row ids of two slots, and the write-back sends every row to the row
// its id names (as in panel_kernel, getrf.cu).  What differs is the exchange:
// every CTA pushes its candidate's header (pivot key and sign, row id, value
// in column j+1) into every peer's shared memory with st.async, which counts
// its bytes on the receiver's mbarrier, so a column costs one one-way cluster
// latency (an all-to-all of 16 CTAs with the reduction: 390 cycles measured)
// instead of a store to L2 and a poll of it (about 1.5 us).  The winner then
// pushes its row segment the same way; it is needed only by the next column's
// updates.
//
// Warps.  W owner warps (1 .. 4) own the rows: owner thread t keeps for its
// rows t, t + 128, .. the value in column j (its candidate), the value in
// column j+1 and the row id in registers, and every owner warp takes part in
// the exchange by itself, so no block barrier lies on the column's chain:
//   push of the warp's candidate (lanes = peers); wait; winner (every warp
//   reduces all P W headers alike); column j scaled and column j+1 updated in
//   registers; the warp's next candidate; with the first piece of the winner's
//   segment, the candidate's column j+2, then the push; the other rows' column
//   j+2 while that is under way.
// The divider (FP64) forms the candidates' reciprocals as soon as they are known
// and adds them to their headers: a division is some 340 cycles of dependent operations,
// which on the winner's side of the exchange would be the longest link.
// The helper brings the candidates' rows up to date while their headers
//   travel, arms the barriers, pushes the segment if this CTA won (its first 16
//   bytes, which hold column j+2, to all peers at once and on a barrier of its
//   own) and records the pivot.
// The bulk warps apply step j's update to columns j+3.. of the active rows
// (all but the next candidates) one column behind: "column j scaled" and
// "update of step j done" are named barriers, the second of which the owners
// pass a column later.  FP64: the pipe of each quarter of an SM takes 64 cycles
// a warp instruction, so the bulk update, not the exchange, bounds a panel of
// many rows per CTA, and such panels are kept narrow.
// What bounds a small panel is the length of that chain, some 1700 cycles a column
// at one instruction every four cycles or so: no array of it is indexed by a
// variable (such arrays live in local memory, whose lines the waits' acquire
// discards), nor is there an integer division, and the waits' loops are out of line.
// us a 64-column panel (the launch alone), with the divider and without local arrays:
// FP64 75.6 -> 61 at 64 rows, 77 -> 64 at 256, 82 -> 71 at 512, 100 -> 96 at 1024, 156 ->
// 143 at 2048; FP32 61.4 -> 59 at 64, 69 -> 63 at 512, 73 -> 68 at 1024, 91 -> 92 at 2048.
//
// Reuse of the exchange buffers (two, by step parity): a warp pushes step j+2
// only after it has every header of step j+1, and a warp sends that header only
// after it has read all of step j and the bulk warps are done with the row of
// step j-1.  All CTAs meet in a cluster barrier before they exit, so no push
// can reach a CTA that is gone.  Waits are bounded like all others of the
// library; a warp that gave up goes on through the barriers without pushing.
//
// Arithmetic and its order per element are those of panel_kernel, so exact
// mode keeps lair's bits (src/lapack/getrf.rs:56-89).
#include <algorithm>

#include "cluster.cuh"
#include "common.cuh"
#include "luhot_internal.h"
#include "panel.cuh"

namespace luhot {

constexpr int kClMaxCtas = 16;
constexpr int kClSegPad = 4;
constexpr int kClOwners = 4;  // owner warps at most
constexpr int kClOwnRows = 32 * kClOwners;
// FP64: 17 warps.  The owners (warps 0, 4, 8, 12) and the divider (4 W) have one
// quarter of the SM to themselves, the helper (1) and eleven bulk warps the other
// three: a bulk warp on the same FP64 pipe would make each of the dependent
// operations of a column's chain wait for one or two of its own, 64 cycles each.
// FP32: 20 warps (bound by shared-memory latency), owners 0 .. W-1, helper W.
template <typename T>
__host__ __device__ constexpr int cl_threads() {
  return sizeof(T) == 8 ? 544 : 640;
}
// Odd row stride for FP64 (conflict-free column and row access); 16-byte rows
// for FP32's float4 updates.
template <typename T>
static int cl_lds(int w) {
  return sizeof(T) == 4 ? ((w + 3) & ~3) + 4 : (w + 1) | 1;
}
template <typename T>
static size_t cl_smem_bytes(int rows_per, int w) {
  return ((((size_t)rows_per * cl_lds<T>(w) + 3) & ~(size_t)3) + 2 * (kMaxPanelWidth + kClSegPad)) * sizeof(T) +
         2 * (size_t)rows_per * sizeof(int);
}

// A warp's header: 16 bytes (FP32: key | id, value) or 32 (FP64: key, id; value;
// reciprocal, pushed by the divider).
template <typename T>
struct ClHeader;
template <>
struct ClHeader<float> {
  using K = unsigned int;
  static constexpr unsigned kBytes = 16;
  static constexpr K kSign = 0x80000000u;
  __device__ static void push(unsigned dst, unsigned bar, K key, int id, float u1) {
    cl_push16(dst, bar, key, ((unsigned long long)__float_as_uint(u1) << 32) | (unsigned)id);
  }
  __device__ static void read_key(const unsigned long long* h, K& key, int& id) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(h);
    key = (unsigned)v.x;
    id = (int)(unsigned)v.y;
  }
  __device__ static void read_value(const unsigned long long* h, float& u1, float&) {
    u1 = __uint_as_float((unsigned)(h[1] >> 32));
  }
};
template <>
struct ClHeader<double> {
  using K = unsigned long long;
  static constexpr unsigned kBytes = 32;
  static constexpr K kSign = 0x8000000000000000ull;
  __device__ static void push(unsigned dst, unsigned bar, K key, int id, double u1) {
    cl_push16(dst, bar, key, (unsigned)id);
    cl_push8(dst + 16, bar, (unsigned long long)__double_as_longlong(u1));
  }
  __device__ static void read_key(const unsigned long long* h, K& key, int& id) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(h);
    key = v.x;
    id = (int)(unsigned)v.y;
  }
  __device__ static void read_value(const unsigned long long* h, double& u1, double& recip) {
    const double2 v = *reinterpret_cast<const double2*>(h + 2);
    u1 = v.x;
    recip = v.y;
  }
};

__device__ __forceinline__ void cl_bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void cl_bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// The winner among the n headers of one step (the same answer in every warp): its
// index, row id, signed key (0: no pivot), column j+1 value and (FP64) reciprocal,
// read from its header.
template <typename T>
__device__ __forceinline__ void cl_winner(const unsigned long long (*box)[4], int n, int lane, int& win, int& pr,
                                          typename ClHeader<T>::K& kraw, T& u1, T& recip) {
  using H = ClHeader<T>;
  using K = typename H::K;
  K k = 0;
  pr = INT_MAX;
  win = lane;
  if (lane < n) {
    H::read_key(box[lane], k, pr);
    k &= ~H::kSign;
  }
  if (lane + 32 < n) {
    K hk;
    int hid;
    H::read_key(box[lane + 32], hk, hid);
    hk &= ~H::kSign;
    if (hk > k || (hk == k && hid < pr)) {
      k = hk;
      pr = hid;
      win = lane + 32;
    }
  }
  const int src = warp_best(k, pr);
  if (n > 32)
    win = __shfl_sync(0xffffffffu, win, src);
  else
    win = src;
  H::read_key(box[win], kraw, pr);
  H::read_value(box[win], u1, recip);
}

// S[r][c] -= S[r][jj] u[c] for the rows r of [0, n) that are active after step
// jj (ret[r] > jj) and no candidates, and the columns [c0, w), by threads t of
// nt.  FP64: (row, column) pairs flattened, so the lanes of a warp instruction
// work (the FP64 pipe bounds it).
template <bool kExact>
__device__ __forceinline__ void cl_update(double* S, int lds, const int* ret, int n, int4 cand, int jj, int c0, int w,
                                          const double* u, int t, int nt) {
  const int wc = w - c0;
  const int total = n * wc;
  const int step_r = nt / wc, step_c = nt - step_r * wc;
  int r = t / wc, c = t - (t / wc) * wc;
  for (int idx = t; idx < total; idx += 2 * nt) {
    const int ra = r, ca = c;
    r += step_r;
    c += step_c;
    if (c >= wc) {
      c -= wc;
      ++r;
    }
    const int rb = r, cb = c;
    bool do_b = idx + nt < total;
    r += step_r;
    c += step_c;
    if (c >= wc) {
      c -= wc;
      ++r;
    }
    const bool do_a = ret[ra] > jj && ra != cand.x && ra != cand.y && ra != cand.z && ra != cand.w;
    do_b = do_b && ret[rb] > jj && rb != cand.x && rb != cand.y && rb != cand.z && rb != cand.w;
    double xa = 0, la = 0, ua = 0, xb = 0, lb = 0, ub = 0;
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
}
// FP32: float4 chunks, lane (sub, ch) takes chunk ch of its warp's row sub;
// two row groups in flight.  Columns left of c0 in the first chunk are not
// written (other warps own them meanwhile).
template <int CH, bool kExact>
__device__ __forceinline__ void cl_update_f32(float* S, int lds, const int* ret, int n, int4 cand, int jj, int c0,
                                              int w, const float* u, int t, int nt) {
  constexpr int RPW = 32 / CH, kR = 2;
  const int lane = t & 31, wi = t >> 5, nw = nt >> 5;
  const int ch = lane % CH, sub = lane / CH;
  const int c = ch * 4;
  if (c + 4 <= c0 || c >= w) return;
  const bool whole = c >= c0;
  const float4 uv = *reinterpret_cast<const float4*>(u + c);
  const int G = nw * RPW;
  for (int q = wi * RPW + sub; q < n; q += kR * G) {
    int r[kR];
    bool on[kR];
    float l[kR];
    float4 x[kR];
#pragma unroll
    for (int e = 0; e < kR; ++e) {
      on[e] = q + e * G < n;
      r[e] = on[e] ? q + e * G : q;
      const float* row = S + r[e] * lds;
      on[e] = on[e] && ret[r[e]] > jj && r[e] != cand.x && r[e] != cand.y && r[e] != cand.z && r[e] != cand.w;
      l[e] = row[jj];
      x[e] = *reinterpret_cast<const float4*>(row + c);
    }
#pragma unroll
    for (int e = 0; e < kR; ++e) {
      if (!on[e]) continue;
      float* dst = S + r[e] * lds + c;
      if (whole) {
        float4 y;
        y.x = upd<kExact>(x[e].x, l[e], uv.x);
        y.y = upd<kExact>(x[e].y, l[e], uv.y);
        y.z = upd<kExact>(x[e].z, l[e], uv.z);
        y.w = upd<kExact>(x[e].w, l[e], uv.w);
        *reinterpret_cast<float4*>(dst) = y;
      } else {
        if (c + 1 >= c0) dst[1] = upd<kExact>(x[e].y, l[e], uv.y);
        if (c + 2 >= c0) dst[2] = upd<kExact>(x[e].z, l[e], uv.z);
        if (c + 3 >= c0) dst[3] = upd<kExact>(x[e].w, l[e], uv.w);
      }
    }
  }
}
template <bool kExact>
__device__ __forceinline__ void cl_update(float* S, int lds, const int* ret, int n, int4 cand, int jj, int c0, int w,
                                          const float* u, int t, int nt) {
  if (w <= 32)
    cl_update_f32<8, kExact>(S, lds, ret, n, cand, jj, c0, w, u, t, nt);
  else if (w <= 64)
    cl_update_f32<16, kExact>(S, lds, ret, n, cand, jj, c0, w, u, t, nt);
  else
    cl_update_f32<32, kExact>(S, lds, ret, n, cand, jj, c0, w, u, t, nt);
}

// kNR: rows of one owner thread (rows of a CTA <= 128 kNR).
template <typename T, bool kExact, int kNR>
__global__ void __launch_bounds__(cl_threads<T>(), 1) panel_cluster_kernel(PanelArgs<T> p) {
  using H = ClHeader<T>;
  using K = typename H::K;
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kThreads = cl_threads<T>(), kOwnRows = kClOwnRows;
  constexpr bool kDivider = sizeof(T) == 8;
  constexpr int kWarps = kThreads / 32;
  constexpr int kVec = 16 / (int)sizeof(T);  // elements of one pushed piece
  constexpr int kSeg = kMaxPanelWidth + kClSegPad;
  constexpr int kBarScaled = 1, kBarDone = 2;  // named barriers: scaled; done (two, by step parity)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* S = reinterpret_cast<T*>(smem_raw);                  // [rows_per][lds]
  T* segb = S + (size_t)((p.rows_per * p.lds + 3) & ~3);  // [2][kSeg] pivot rows
  int* ids = reinterpret_cast<int*>(segb + 2 * kSeg);     // final global row of each slot
  int* ret = ids + p.rows_per;                            // step in which a slot's row retired
  __shared__ __align__(16) unsigned long long box[2][kClMaxCtas * kClOwners][4];  // every warp's header
  // Headers; the winner's segment, its first 16 bytes apart: column j+2 is on the
  // next column's chain.
  __shared__ __align__(8) unsigned long long hbar[2], ebar[2], sbar[2];
  // The owner warps' next candidates.
  __shared__ __align__(16) int s_cand[2][kClOwners];
  __shared__ T s_mult[2][kClOwners], s_val[2][kClOwners];  // its multiplier in the last step; its pivot
  __shared__ int s_pivoted[2], s_ok;

  const int P = gridDim.x, b = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r_begin = p.k0 + b * p.rows_per;
  const int nloc = max(0, min(p.m, r_begin + p.rows_per) - r_begin);
  const int w = p.w, lds = p.lds;
  const int W = (min(p.rows_per, kOwnRows) + 31) / 32;  // owner warps, the same in every CTA
  // Roles.  The barriers "scaled" (all of them) and "done" (but the divider).
  enum { kOwner, kHelper, kDivide, kBulk, kIdle };
  int role, index = 0;  // of an owner or bulk warp
  if (kDivider) {
    index = (warp & 3) == 0 ? warp >> 2 : (warp >> 2) * 3 + (warp & 3) - 2;
    role = warp == 1 ? kHelper : (warp & 3) != 0 ? kBulk : index < W ? kOwner : index == W ? kDivide : kIdle;
  } else {
    index = warp < W ? warp : warp - W - 1;
    role = warp < W ? kOwner : warp == W ? kHelper : kBulk;
  }
  const int bulk_threads = kDivider ? 11 * 32 : kThreads - 32 * (W + 1);
  const int n_done = 32 * (W + 1) + bulk_threads, n_scaled = n_done + (kDivider ? 32 : 0);

  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cl_smem(&hbar[i])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cl_smem(&ebar[i])));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cl_smem(&sbar[i])));
    }
    asm volatile("fence.mbarrier_init.release.cluster;");
    s_ok = 1;
    if (b == 0) *p.move_count = 0;
  }
  if (tid < 2 * kClOwners) {
    s_cand[tid / kClOwners][tid % kClOwners] = -1;
    s_val[tid / kClOwners][tid % kClOwners] = T(1);
  }
  for (int r = warp; r < nloc; r += kWarps) {
    const T* src = p.a + (int64_t)(r_begin + r) * p.lda + p.k0;
    for (int c = lane; c < w; c += 32) S[r * lds + c] = src[c];
  }
  for (int r = tid; r < nloc; r += kThreads) ret[r] = INT_MAX;
  cl_sync();  // barriers initialised everywhere, move_count cleared, this CTA's rows loaded

  if (role == kOwner) {
    // ------------------------------------------------------------- owners
    const int ot = 32 * index + lane;
    T a[kNR], c1[kNR], lv[kNR];  // column j, column j+1, multiplier of the last step
    int id[kNR];                 // global row, -1: none or retired
#pragma unroll
    for (int i = 0; i < kNR; ++i) {
      const int r = ot + kOwnRows * i;
      const bool on = r < nloc;
      id[i] = on ? r_begin + r : -1;
      a[i] = on ? S[r * lds] : T(0);
      c1[i] = on && w > 1 ? S[r * lds + 1] : T(0);
      lv[i] = T(0);
    }
    // This lane's places in the peer of its number (lanes below P), step parity 0.
    const unsigned peer_box = cl_peer(cl_smem(&box[0][b * W + index][0]), min(lane, P - 1));
    const unsigned peer_bar = cl_peer(cl_smem(&hbar[0]), min(lane, P - 1));
    K ck = 0;          // the warp's candidate: key with the pivot's sign,
    int cid = 0;       // row id,
    int cslot = -1;    // slot,
    T cl = T(0);       // multiplier of the last step,
    T cu = T(0);       // column j+1 value
    auto candidate = [&](int par) {
      K bk = 0;
      int bid = INT_MAX, bslot = -1;
      T bv = T(1), bl = T(0);
#pragma unroll
      for (int i = 0; i < kNR; ++i) {
        const K k = PivotKey<T>::of(a[i]);
        if (id[i] >= 0 && (bslot < 0 || k > bk || (k == bk && id[i] < bid))) {
          bk = k;
          bid = id[i];
          bslot = ot + kOwnRows * i;
          bv = a[i];
          bl = lv[i];
        }
      }
      const int src = warp_best(bk, bid);
      ck = __shfl_sync(kFull, bslot >= 0 && signbit(bv) ? bk | H::kSign : bk, src);
      cid = __shfl_sync(kFull, bid, src);
      cslot = __shfl_sync(kFull, bslot, src);
      cl = __shfl_sync(kFull, bl, src);
      if (lane == src) {
        s_cand[par][index] = bslot;
        s_mult[par][index] = bl;
        s_val[par][index] = bv;
      }
    };
    candidate(1);
    cu = cslot >= 0 && w > 1 ? S[cslot * lds + 1] : T(0);
    __syncwarp();
    cl_bar_sync(kBarScaled, n_scaled);
    unsigned seg_phase = 0u;  // bit q: phase of segment barrier q's next use (an array would live in local memory)
    bool ok = true;
    bool was_pivot = false;  // the last step had a pivot; un: its row's next element
    T un = T(0);
    for (int j = 0; j < w; ++j) {
      const int ul = p.k0 + j;
      const int par = j & 1;
      if (ok && lane < P) H::push(peer_box + (unsigned)par * (unsigned)sizeof(box[0]), peer_bar + 8u * (unsigned)par, ck, cid, cu);
      if (j > 0 && j + 1 < w) {
        // While the headers travel: column j+1 of this thread's rows (the
        // candidate's went with the header).
#pragma unroll
        for (int i = 0; i < kNR; ++i) {
          if (id[i] < 0) continue;
          const T x = S[(ot + kOwnRows * i) * lds + j + 1];
          c1[i] = was_pivot ? upd<kExact>(x, lv[i], un) : x;
        }
      }
      ok = ok && cl_wait(cl_smem(&hbar[par]), (unsigned)((j >> 1) & 1), p.st, ul);
      int win, pr;
      K kraw;
      T u1, recip;
      cl_winner<T>(box[par], P * W, lane, win, pr, kraw, u1, recip);
      const bool pivot = ok && (kraw & ~H::kSign) > 0;
      if (!pivot) pr = ul;
      if constexpr (!kDivider) recip = T(1) / PivotKey<T>::value(kraw);
      // The row with id pr takes id ul and retires, the row with id ul takes
      // id pr; the other rows' column j is scaled and column j+1 updated.
#pragma unroll
      for (int i = 0; i < kNR; ++i) {
        if (id[i] < 0) continue;
        const int r = ot + kOwnRows * i;
        T* row = S + r * lds + j;
        if (id[i] == pr) {
          row[0] = a[i];
          if (j + 1 < w) row[1] = c1[i];
          ids[r] = ul;
          ret[r] = j;
          id[i] = -1;
          continue;
        }
        if (id[i] == ul) id[i] = pr;
        if (pivot) {
          const T l = mul_rn(a[i], recip);
          row[0] = l;
          lv[i] = l;
          a[i] = upd<kExact>(c1[i], l, u1);
        } else {
          row[0] = a[i];
          a[i] = c1[i];
        }
      }
      if (j + 1 < w) candidate(par);
      __syncwarp();
      // The helper passes "done" of step j-1 after "scaled" of step j, so the
      // owners never arrive twice at one "scaled"; the first one they wait for.
      if (j > 0) {
        cl_bar_arrive(kBarScaled, n_scaled);
        cl_bar_sync(kBarDone + ((j - 1) & 1), n_done);
      } else {
        cl_bar_sync(kBarScaled, n_scaled);
      }
      if (j + 2 < w) {
        // Column j+2 of this thread's rows: step j-1's update is in (the
        // barrier), step j's with the winner's segment.
        if (pivot) {
          ok = ok && cl_wait(cl_smem(&ebar[par]), (seg_phase >> par) & 1u, p.st, ul);
          seg_phase ^= 1u << par;
        }
        un = segb[par * kSeg + j + 2];
        if (cslot >= 0) {
          const T x = S[cslot * lds + j + 2];
          cu = pivot ? upd<kExact>(x, cl, un) : x;
        }
      }
      was_pivot = pivot;
    }
#pragma unroll
    for (int i = 0; i < kNR; ++i)
      if (id[i] >= 0) ids[ot + kOwnRows * i] = id[i];
    if (!ok && lane == 0) s_ok = 0;
  } else if (role == kHelper) {
    // ------------------------------------------------------------- helper
    unsigned seg_phase = 0u;
    bool ok = true;
    int dj = -1;  // step whose update of the candidates' rows is pending
    if (lane == 0) cl_expect(cl_smem(&hbar[0]), (unsigned)(P * W) * H::kBytes);
    cl_bar_sync(kBarScaled, n_scaled);
    for (int j = 0; j < w; ++j) {
      const int ul = p.k0 + j;
      const int par = j & 1;
      const int* cand = s_cand[par ^ 1];
      if (dj >= 0 && j + 1 < w) {
        // Columns j+2.. of the candidates' rows (the owners hold j and j+1):
        // step j-1's update, once step j-2's is in (barrier of the last pass).
        const int sp = dj & 1;
        ok = ok && cl_wait(cl_smem(&ebar[sp]), (seg_phase >> sp) & 1u, p.st, ul) &&
             cl_wait(cl_smem(&sbar[sp]), (seg_phase >> sp) & 1u, p.st, ul);
        seg_phase ^= 1u << sp;
        const T* up = segb + sp * kSeg;
        for (int q = 0; q < W; ++q) {
          const int cs = cand[q];
          if (cs < 0) continue;
          const T l = s_mult[par ^ 1][q];
          T* row = S + cs * lds;
          for (int c = j + 2 + lane; c < w; c += 32) row[c] = upd<kExact>(row[c], l, up[c]);
        }
        __syncwarp();
      }
      ok = ok && cl_wait(cl_smem(&hbar[par]), (unsigned)((j >> 1) & 1), p.st, ul);
      int win, pr;
      K kraw;
      T u1, recip;
      cl_winner<T>(box[par], P * W, lane, win, pr, kraw, u1, recip);
      const bool pivot = ok && (kraw & ~H::kSign) > 0;
      if (pivot && j + 2 < w) {
        // The winner's segment j+2.. in 16-byte pieces, from an aligned column on;
        // the first one to all peers at once.
        const unsigned sb = cl_smem(&sbar[par]), eb = cl_smem(&ebar[par]);
        const int c0 = (j + 2) & ~(kVec - 1);
        const int pieces = (w - c0 + kVec - 1) / kVec;
        if ((unsigned)(win - b * W) < (unsigned)W) {
          const T* row = S + cand[win - b * W] * lds;
          const unsigned dst = cl_smem(segb + par * kSeg);
          auto piece = [&](int c, unsigned long long(&v)[2]) {
            if constexpr (sizeof(T) == 8) {
              v[0] = (unsigned long long)__double_as_longlong(row[c]);
              v[1] = (unsigned long long)__double_as_longlong(row[c + 1]);
            } else {
              const uint4 x = *reinterpret_cast<const uint4*>(row + c);
              v[0] = ((unsigned long long)x.y << 32) | x.x;
              v[1] = ((unsigned long long)x.w << 32) | x.z;
            }
          };
          unsigned long long v[2];
          if (lane < P) {
            piece(c0, v);
            cl_push16(cl_peer(dst + (unsigned)c0 * (unsigned)sizeof(T), lane), cl_peer(eb, lane), v[0], v[1]);
          }
          for (int q = 1 + lane; q < pieces; q += 32) {
            const int c = c0 + q * kVec;
            piece(c, v);
            for (int cta = 0; cta < P; ++cta)
              cl_push16(cl_peer(dst + (unsigned)c * (unsigned)sizeof(T), cta), cl_peer(sb, cta), v[0], v[1]);
          }
        }
        if (lane == 0) {
          cl_expect(eb, 16u);
          cl_expect(sb, (unsigned)(pieces - 1) * 16u);
        }
      }
      if (lane == 0) {
        // Every header of step j is here, so the other barrier's phase of step
        // j-1 is over and step j+1's can be armed.
        if (j + 1 < w) cl_expect(cl_smem(&hbar[par ^ 1]), (unsigned)(P * W) * H::kBytes);
        s_pivoted[par] = pivot ? 1 : 0;
        if (b == 0 && ok) {
          p.piv[ul] = pivot ? pr : ul;
          // lair: max == 0 -> the step is singular, no swap, no update
          // (src/lapack/getrf.rs:72-73).  The last such step wins.
          if (!pivot) atomicMax(&p.st->singular, ul);
        }
      }
      dj = pivot ? j : -1;
      __syncwarp();
      cl_bar_sync(kBarScaled, n_scaled);
      if (j > 0) cl_bar_sync(kBarDone + ((j - 1) & 1), n_done);
    }
    if (!ok && lane == 0) s_ok = 0;
  } else if (role == kDivide) {
    // ------------------------------------------------------------ divider
    // The candidates' reciprocals, while their headers are still being prepared.
    // A division is some 340 cycles of dependent operations: on the winner's
    // side of the exchange it would be the longest link of the chain.
    if constexpr (kDivider) {
      // Lane (q, cta) pushes candidate q's (and q + 2's) to peer cta.
      const int cta = lane & (kClMaxCtas - 1), q0 = lane / kClMaxCtas;
      const unsigned dst = cl_peer(cl_smem(&box[0][b * W + min(q0, W - 1)][3]), min(cta, P - 1));
      const unsigned bar = cl_peer(cl_smem(&hbar[0]), min(cta, P - 1));
      for (int j = -1; j < w; ++j) {
        cl_bar_sync(kBarScaled, n_scaled);  // the candidates for step j+1 are known
        if (j + 1 >= w) break;
        const int par = j & 1, nxt = par ^ 1;
        const unsigned to = dst + (unsigned)nxt * (unsigned)sizeof(box[0]), on = bar + 8u * (unsigned)nxt;
        if (cta < P && q0 < W)
          cl_push8(to, on, (unsigned long long)__double_as_longlong(1.0 / (double)s_val[par][q0]));
        if (cta < P && q0 + 2 < W)
          cl_push8(to + 2u * (unsigned)sizeof(box[0][0]), on,
                   (unsigned long long)__double_as_longlong(1.0 / (double)s_val[par][q0 + 2]));
      }
    }
  } else if (role == kBulk) {
    // ------------------------------------------------------------- bulk
    unsigned seg_phase = 0u;
    bool ok = true;
    cl_bar_sync(kBarScaled, n_scaled);
    for (int j = 0; j < w; ++j) {
      const int par = j & 1;
      cl_bar_sync(kBarScaled, n_scaled);
      if (s_pivoted[par] && j + 3 < w) {
        const int4 cand = *reinterpret_cast<const int4*>(s_cand[par]);
        ok = ok && cl_wait(cl_smem(&ebar[par]), (seg_phase >> par) & 1u, p.st, p.k0 + j) &&
             cl_wait(cl_smem(&sbar[par]), (seg_phase >> par) & 1u, p.st, p.k0 + j);
        seg_phase ^= 1u << par;
        if (ok)
          cl_update<kExact>(S, lds, ret, nloc, cand, j, j + 3, w, segb + par * kSeg, index * 32 + lane, bulk_threads);
      }
      __syncwarp();
      if (j + 1 < w) cl_bar_arrive(kBarDone + par, n_done);
    }
    if (!ok && lane == 0) s_ok = 0;
  }
  __syncthreads();
  if (s_ok) {
    for (int r = warp; r < nloc; r += kWarps) {
      T* dst = p.a + (int64_t)ids[r] * p.lda + p.k0;
      for (int c = lane; c < w; c += 32) dst[c] = S[r * lds + c];
    }
    // The rows that changed place, for the interchanges outside the panel.
    for (int r = tid; r < nloc; r += kThreads) {
      if (ids[r] != r_begin + r) {
        const int e = atomicAdd(p.move_count, 1);
        if (e < 2 * kMaxPanelWidth) {  // at most 2w rows move; the bound guards the list
          p.moves[2 * e] = ids[r];
          p.moves[2 * e + 1] = r_begin + r;
        }
      }
    }
  }
  cl_sync();  // every CTA's pushes have been received, or its waits were given up
  if (!s_ok) cl_drain();
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
// CTAs: a power of two (the last ones may hold no rows) with at least 16 (FP64)
// or 32 (FP32) rows each, up to the largest cluster the device schedules.
template <typename T>
static void cl_split(luhot_ctx* ctx, int rows, int* P, int* rows_per) {
  const int min_rows = sizeof(T) == 8 ? 16 : 32;
  *P = 1;
  while (*P < ctx->panel_cluster && *P * min_rows < rows) *P *= 2;
  *rows_per = (rows + *P - 1) / *P;
}

// Static shared memory of the kernel and rounding, left out of the budget.
constexpr size_t kClStaticSmem = 8192;

int panel_cluster_limit(luhot_ctx* ctx) {
  auto kern = panel_cluster_kernel<double, false, 2>;
  const size_t smem = (size_t)ctx->max_smem_optin - kClStaticSmem;
  if (allow_max_dynamic_smem(kern) != cudaSuccess ||
      allow_wide_clusters(reinterpret_cast<const void*>(kern)) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  for (int P = kClMaxCtas; P >= 1; P /= 2) {
    cudaLaunchAttribute attr;
    cudaLaunchConfig_t cfg = cl_config(P, cl_threads<double>(), smem, nullptr, &attr);
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) == cudaSuccess && clusters > 0) return P;
    cudaGetLastError();
  }
  return 0;
}

// Rows of a CTA up to which the cluster is the faster form.  us a 64-column panel (a
// getrf call), cluster of 16 / exchange through L2 on up to 96 (FP64) or 64 (FP32)
// CTAs: FP64 fast 166 / 235 at 2000 rows, 193 / 233 at 2500, 200 / 230 at 2600, 212 / 230
// at 3000, 225 / 230 at 3200, 237 / 230 at 3500 (the rank-1 updates of 200 rows fill one
// SM's FP64 pipes); exact, whose updates are two operations, 200 / 231 at 1500, 225 / 231 at
// 1700, 239 / 231 at 2000, 286 / 230 at 2500; FP32, either mode, 116 / 180 at 2000, 150 / 181
// at 5000, 165 / 180 at 6000.
template <typename T, bool kExact>
constexpr int cl_max_rows() {
  return sizeof(T) == 4 ? 384 : kExact ? 112 : 192;
}

template <typename T, bool kExact>
bool panel_cluster_fits(luhot_ctx* ctx, int rows, int w) {
  if (ctx->panel_cluster < 1 || w > kMaxPanelWidth || rows < 1) return false;
  int P, rows_per;
  cl_split<T>(ctx, rows, &P, &rows_per);
  return rows_per <= cl_max_rows<T, kExact>() && cl_smem_bytes<T>(rows_per, w) + kClStaticSmem <= (size_t)ctx->max_smem_optin;
}

template <typename T, bool kExact>
int launch_panel_cluster(luhot_ctx* ctx, T* a, int64_t lda, int m, int k0, int w, int* piv, int* moves,
                         cudaStream_t stream) {
  const int rows = m - k0;
  int P, rows_per;
  cl_split<T>(ctx, rows, &P, &rows_per);
  constexpr int kMost = cl_max_rows<T, kExact>();  // owner threads hold kMost / kClOwnRows rows at most
  static_assert(kMost <= 4 * kClOwnRows, "an owner thread holds at most four rows");
  auto kern = panel_cluster_kernel<T, kExact, 1>;
  if constexpr (kMost > kClOwnRows)
    if (rows_per > kClOwnRows) kern = panel_cluster_kernel<T, kExact, 2>;
  if constexpr (kMost > 2 * kClOwnRows)
    if (rows_per > 2 * kClOwnRows) kern = panel_cluster_kernel<T, kExact, 4>;
  LUHOT_CUDA_TRY(ctx, allow_max_dynamic_smem(kern));
  LUHOT_CUDA_TRY(ctx, allow_wide_clusters(reinterpret_cast<const void*>(kern)));
  PanelArgs<T> args{};
  args.a = a;
  args.lda = lda;
  args.m = m;
  args.k0 = k0;
  args.w = w;
  args.rows_per = rows_per;
  args.lds = cl_lds<T>(w);
  args.piv = piv;
  args.moves = moves;
  args.move_count = args.moves + 4 * kMaxPanelWidth;
  args.st = ctx->d_status;
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = cl_config(P, cl_threads<T>(), cl_smem_bytes<T>(rows_per, w), stream, &attr);
  prof_begin(ctx, kProfPanel);
  LUHOT_CUDA_TRY(ctx, cudaLaunchKernelEx(&cfg, kern, args));
  double fl = 0.0;
  for (int j = 0; j < w; ++j) fl += (double)(rows - j - 1) * (1.0 + 2.0 * (w - j - 1));
  prof_end(ctx, kProfPanel, fl, 2.0 * rows * w * sizeof(T));
  return LUHOT_OK;
}

template bool panel_cluster_fits<double, false>(luhot_ctx*, int, int);
template bool panel_cluster_fits<double, true>(luhot_ctx*, int, int);
template bool panel_cluster_fits<float, false>(luhot_ctx*, int, int);
template bool panel_cluster_fits<float, true>(luhot_ctx*, int, int);
template int launch_panel_cluster<double, false>(luhot_ctx*, double*, int64_t, int, int, int, int*, int*, cudaStream_t);
template int launch_panel_cluster<double, true>(luhot_ctx*, double*, int64_t, int, int, int, int*, int*, cudaStream_t);
template int launch_panel_cluster<float, false>(luhot_ctx*, float*, int64_t, int, int, int, int*, int*, cudaStream_t);
template int launch_panel_cluster<float, true>(luhot_ctx*, float*, int64_t, int, int, int, int*, int*, cudaStream_t);

}  // namespace luhot
