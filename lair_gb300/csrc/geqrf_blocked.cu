// Blocked Householder QR (fast mode, FP64) on one GB300: panels of 32 columns,
// compact WY updates (Schreiber & Van Loan, 1989; the triangular factor is not
// formed, see qr_y_kernel).  The reflectors are lair's (src/lapack/larfg.rs:9-43):
// beta = -sign(alpha) sqrt(alpha^2 + x.x), tau = (beta - alpha) / beta, v = [1,
// x / (alpha - beta)]; a column whose x.x is zero gets tau = 0 and keeps its x.
// (larfg's rescaling loop needs |beta| below 2^-969 with x.x > 0, which a sum of
// FP64 squares cannot give.)  The level-2 form (geqrf.cu) took three launches and
// two passes over the trailing block per column, 55 us each at 2000 x 1500.
//
// Per panel of w <= 32 columns from row and column k0 (rows = m - k0):
//   qr_panel_kernel  one thread-block cluster of up to 16 CTAs, the panel's rows
//                    in shared memory.  Column j needs, over the rows below its
//                    diagonal, the products of x with itself and with every later
//                    panel column; one pass over the rows applies reflector j-1
//                    and forms those sums, one all-to-all push (cluster.cuh) of the
//                    CTAs' sums and of row k0 + j gives every CTA the totals, and
//                    every CTA derives the same beta, tau and row factors.  FP64:
//                    a pass is two FMAs an element and fills the SMs' FP64 pipes
//                    (2 us a column at 2000 rows); the exchange with its square
//                    root and division takes about 1 us.  The products are of x itself,
//                    not of v: columns whose products with others could leave the range
//                    of FP64 (largest element outside 2^-450 .. 2^450) are held divided
//                    by a power of two, on which V and tau do not depend.
//   qr_w_kernel      W = V^T [V A2] by FP64 MMAs, 32 columns x a range of rows per
//                    CTA, partial sums per range (summed in a fixed order);
//   qr_y_kernel      Y = T^T W: T^-1 is the upper triangle of V^T V with 1 / tau on
//                    its diagonal, so y_j = tau_j (w_j - sum_{i<j} (V^T V)_ij y_i);
//   qr_update_kernel A2 -= V Y by FP64 MMAs.  (Slice products, ozaki.cu, on large blocks:
//                    13.3 ms at 2000 x 1500 against 15.7, but they hold V and Y relative to the
//                    largest of its row or column: where reflectors of rows of
//                    different scale meet, 3e-9 of |V||Y| in place of 3e-16.)
#include <algorithm>

#include "cluster.cuh"
#include "common.cuh"
#include "luhot_internal.h"

namespace luhot {

namespace {

constexpr int kQb = 32;           // panel columns
constexpr int kQbLd = kQb + 1;    // odd row stride: conflict-free rows and columns
constexpr int kQbMaxCtas = 16;
constexpr int kQbThreads = 256;
constexpr int kQbWarps = kQbThreads / 32;
constexpr size_t kQbStatic = 16 * 1024;  // static shared memory of the panel kernel, rounded up
constexpr int kQbRange = 450;

struct QrPanelArgs {
  double* a;  // the matrix at (k0, k0)
  int64_t lda;
  int rows, w, rows_per;
  double* tau;  // w entries
  double* v;    // rows x 32: unit lower trapezoidal V, zero columns past w
  DeviceStatus* st;
};

__global__ void __launch_bounds__(kQbThreads, 1) qr_panel_kernel(QrPanelArgs p) {
  constexpr unsigned kFull = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* S = reinterpret_cast<double*>(smem_raw);  // [rows_per][33]; column j holds x_j unscaled once j is done
  __shared__ __align__(16) double box[2][kQbMaxCtas][kQb];  // every CTA's sums
  __shared__ __align__(16) double arow[2][kQb];             // the diagonal's row
  __shared__ double part[kQbWarps][kQb], tot[kQb], scale_of[kQb];
  __shared__ double s_unit[kQb];  // the power of two that a column is divided by
  __shared__ double s_tau, s_scale, s_beta;
  __shared__ __align__(8) unsigned long long bar[2];
  __shared__ int s_ok;
  const int P = gridDim.x, b = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int r_begin = b * p.rows_per;
  const int nloc = max(0, min(p.rows, r_begin + p.rows_per) - r_begin);
  const int w = p.w;

  if (tid == 0) {
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cl_smem(&bar[i])));
    asm volatile("fence.mbarrier_init.release.cluster;");
    s_ok = 1;
  }
  cl_sync();  // barriers initialised, every CTA there
  {
    // The columns' largest finite elements (bits of |x|), over the warps in `part`,
    // over the CTAs in box[1], which step 1 is the first to use.
    unsigned long long(*top)[kQb] = reinterpret_cast<unsigned long long(*)[kQb]>(part);
    unsigned long long hi = 0;
    for (int r = warp; r < nloc; r += kQbWarps) {
      const double v = lane < w ? p.a[(int64_t)(r_begin + r) * p.lda + lane] : 0.0;
      S[r * kQbLd + lane] = v;
      const unsigned long long bits = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
      if (bits < 0x7ff0000000000000ull) hi = max(hi, bits);
    }
    top[warp][lane] = hi;
    __syncthreads();
    for (int idx = tid; idx < P * kQb; idx += kQbThreads) {
      const int cta = idx / kQb, c = idx - cta * kQb;
      unsigned long long t = 0;
      for (int q = 0; q < kQbWarps; ++q) t = max(t, top[q][c]);
      asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(cl_peer(cl_smem(&box[1][b][c]), cta)), "l"(t) : "memory");
    }
    cl_sync();
    if (warp == 0) {
      unsigned long long t = 0;
      for (int q = 0; q < P; ++q) t = max(t, (unsigned long long)__double_as_longlong(box[1][q][lane]));
      const int e = t != 0 ? ilogb(__longlong_as_double((long long)t)) : 0;
      const int unit = e > kQbRange || e < -kQbRange ? max(-1000, min(1000, e)) : 0;
      s_unit[lane] = __hiloint2double((unit + 1023) << 20, 0);
    }
    __syncthreads();
    const double unit = s_unit[lane];
    if (__any_sync(kFull, unit != 1.0)) {
      const double down = __hiloint2double((2046 << 20) - __double2hiint(unit), 0);  // 1 / unit
      for (int r = warp; r < nloc; r += kQbWarps) S[r * kQbLd + lane] *= down;
    }
    __syncthreads();
  }

  bool ok = true;
  double g = 0.0;  // this lane's column: the factor of x in the pending update
  // Step j: the totals for column j; first the pending update of reflector j-1.
  for (int j = 0; j < w; ++j) {
    const int par = j & 1;
    // Columns j.. lie in the last `width` ones: a warp takes 32 / width rows at
    // once.
    const int width = j < 16 ? 32 : j < 24 ? 16 : 8;
    const int col = 32 - width + lane % width, sub = lane / width, per = 32 / width;
    const int src = sub * width + (j - (32 - width));  // lane of column j in this lane's row
    // The factor for this pass's column (g is per lane column of the full width).
    const double gc = __shfl_sync(kFull, g, col);
    double acc = 0.0;
    const int first = max(0, j - r_begin);  // local row of the diagonal's row j, or 0
    // Rows above row j are finished; row j itself is updated, not summed.
    for (int r0 = first + warp * per; r0 < nloc; r0 += kQbWarps * per) {
      const int r = r0 + sub;
      const bool on = r < nloc;
      double v = 0.0;
      if (on) {
        v = S[r * kQbLd + col];
        if (j > 0 && col >= j) {
          v = fma(S[r * kQbLd + j - 1], gc, v);
          S[r * kQbLd + col] = v;
        }
      }
      const double x = __shfl_sync(kFull, v, src);
      if (on && r_begin + r > j) acc = fma(x, v, acc);
    }
    // Sum over the rows of a warp instruction, then over the warps.
    if (width <= 16) acc += __shfl_xor_sync(kFull, acc, 16);
    if (width <= 8) acc += __shfl_xor_sync(kFull, acc, 8);
    if (sub == 0) part[warp][col] = acc;
    if (sub == 0 && width < 32 && lane < width) {
      // columns left of the pass are done: zero, so that every push is whole
      for (int c = lane; c < 32 - width; c += width) part[warp][c] = 0.0;
    }
    __syncthreads();
    {
      // Warp q sums columns 4q .. 4q + 3, eight lanes a column, and pushes the sums
      // (and the row of the diagonal, from the CTA that holds it) to the peers.
      const int c = 4 * warp + (lane >> 3), q = lane & 7;
      double s = part[q][c];
      s += __shfl_xor_sync(kFull, s, 1);
      s += __shfl_xor_sync(kFull, s, 2);
      s += __shfl_xor_sync(kFull, s, 4);
      if (tid == 0 && ok) cl_expect(cl_smem(&bar[par]), (unsigned)((P + 1) * kQb * sizeof(double)));
      if (ok) {
        const bool owner = j >= r_begin && j < r_begin + nloc;
        const double ar = owner ? S[(j - r_begin) * kQbLd + c] : 0.0;
        for (int cta = q; cta < P; cta += 8) {
          const unsigned pb = cl_peer(cl_smem(&bar[par]), cta);
          cl_push8(cl_peer(cl_smem(&box[par][b][c]), cta), pb, (unsigned long long)__double_as_longlong(s));
          if (owner)
            cl_push8(cl_peer(cl_smem(&arow[par][c]), cta), pb, (unsigned long long)__double_as_longlong(ar));
        }
      }
      ok = ok && cl_wait(cl_smem(&bar[par]), (unsigned)((j >> 1) & 1), p.st, j);
      double t = 0.0;
      if (ok) {
        for (int cta = q; cta < P; cta += 8) t += box[par][cta][c];
      }
      t += __shfl_xor_sync(kFull, t, 1);
      t += __shfl_xor_sync(kFull, t, 2);
      t += __shfl_xor_sync(kFull, t, 4);
      if (q == 0) tot[c] = t;
      if (warp == j >> 2) {
        // The reflector: lane 0 its tau, lane 1 the scale of x.
        const double ss = __shfl_sync(kFull, t, (j & 3) * 8);
        const double alpha = ok ? arow[par][j] : 0.0;
        const double beta = -copysign(sqrt(fma(alpha, alpha, ss)), alpha);
        // lair's norm is zero where the squares underflow, in the column's own unit.
        const bool zero = ss * s_unit[j] * s_unit[j] == 0.0;
        const double num = lane == 0 ? beta - alpha : 1.0, den = lane == 0 ? beta : alpha - beta;
        const double quot = zero ? 0.0 : num / den;
        if (lane == 0) {
          s_tau = quot;
          s_beta = zero ? alpha : beta;
        }
        if (lane == 1) {
          s_scale = quot;
          scale_of[j] = zero ? s_unit[j] : quot;
        }
      }
      if (!ok && lane == 0) s_ok = 0;
    }
    __syncthreads();
    if (!s_ok) break;
    // Row factors of the update: a_rc += x_r g_c (rows below), a_jc += f_c.
    const double tau = s_tau, scale = s_scale;
    double f = 0.0;
    g = 0.0;
    if (tau != 0.0 && lane > j) {
      f = -tau * fma(scale, tot[lane], arow[par][lane]);
      g = scale * f;
    }
    if (b == 0 && tid == 0) p.tau[j] = tau;
    if (warp == 0 && j >= r_begin && j < r_begin + nloc) {
      double* row = S + (j - r_begin) * kQbLd;
      if (lane > j) row[lane] += f;
      if (lane == j) row[j] = s_beta;
    }
    // Row j is finished: the next pass starts below it.
    __syncthreads();
  }
  __syncthreads();
  if (s_ok) {
    // x scaled to v where it was kept, R above; V with its unit diagonal.
    for (int r = warp; r < nloc; r += kQbWarps) {
      const int i = r_begin + r;
      double e = S[r * kQbLd + lane];
      if (lane < w) e *= i > lane ? scale_of[lane] : s_unit[lane];
      if (lane < w) p.a[(int64_t)i * p.lda + lane] = e;
      p.v[(int64_t)i * kQb + lane] = lane >= w || i < lane ? 0.0 : i == lane ? 1.0 : e;
    }
  }
  cl_sync();  // every push has been received, or its wait was given up
  if (!s_ok) cl_drain();
}

__device__ __forceinline__ void qr_dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// wp[range][i][c] = sum over the range's rows r of V[r][i] B[r][c], B = [V A2]:
// column tile 0 is V itself, tile t >= 1 the columns 32 (t-1) .. of A2.  CTA =
// (tile, range), four warps of 16 x 16 of the 32 x 32 sums, 32 rows a stage,
// the next stage's loads in flight during a stage.
__global__ void __launch_bounds__(128) qr_w_kernel(const double* __restrict__ v, const double* __restrict__ a2,
                                                   int64_t lda, int rows, int n2, int rows_per, double* wp,
                                                   int64_t ldw) {
  __shared__ double Vs[32][36], Bs[32][36];  // [row][column]; stride 36: conflict-free fragments
  const int tile = blockIdx.x, r0 = blockIdx.y * rows_per, r1 = min(rows, r0 + rows_per);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wi = (warp >> 1) * 16, wc = (warp & 1) * 16;
  const int g = lane >> 2, t4 = lane & 3;
  const int c = (tile - 1) * 32 + lane;  // this lane's column of A2 in the loads
  const bool on = tile == 0 || c < n2;
  double acc[2][2][2] = {};
  double nv[8], nb[8];
  auto load = [&](int r) {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int row = r + warp + 4 * e;
      const bool in = row < r1;
      nv[e] = in ? v[(int64_t)row * kQb + lane] : 0.0;
      nb[e] = in && on ? (tile == 0 ? nv[e] : a2[(int64_t)row * lda + c]) : 0.0;
    }
  };
  load(r0);
  for (int r = r0; r < r1; r += 32) {
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      Vs[warp + 4 * e][lane] = nv[e];
      Bs[warp + 4 * e][lane] = nb[e];
    }
    __syncthreads();
    if (r + 32 < r1) load(r + 32);
#pragma unroll
    for (int k = 0; k < 32; k += 4) {
      double af[2], bf[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        af[q] = Vs[k + t4][wi + 8 * q + g];
        bf[q] = Bs[k + t4][wc + 8 * q + g];
      }
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) qr_dmma(acc[x][y][0], acc[x][y][1], af[x], bf[y]);
    }
  }
  double* out = wp + (int64_t)blockIdx.y * kQb * ldw + tile * 32;
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int y = 0; y < 2; ++y)
#pragma unroll
      for (int e = 0; e < 2; ++e) out[(int64_t)(wi + 8 * x + g) * ldw + wc + 8 * y + 2 * t4 + e] = acc[x][y][e];
}

// Y = T^T W for the columns of A2: a CTA sums the ranges' partials of V^T V and of
// its 8 columns, then solves (two columns a warp, 16 lanes each, a lane the rows
// lane and lane + 16).
__global__ void __launch_bounds__(128) qr_y_kernel(const double* __restrict__ wp, int64_t ldw, int ranges,
                                                   const double* __restrict__ tau, int w, int n2, double* y,
                                                   int64_t ldy) {
  constexpr unsigned kFull = 0xffffffffu;
  __shared__ double G[kQb][kQb + 1], W[kQb][9];
  const int tid = threadIdx.x, lane = tid & 31;
  const int c0 = blockIdx.x * 8;
  for (int idx = tid; idx < kQb * kQb; idx += 128) {
    const int i = idx >> 5, j = idx & 31;
    double s = 0.0;
    if (j > i)
      for (int q = 0; q < ranges; ++q) s += wp[((int64_t)q * kQb + i) * ldw + j];
    G[i][j] = s;
  }
  for (int idx = tid; idx < kQb * 8; idx += 128) {
    const int i = idx >> 3, j = idx & 7;
    double s = 0.0;
    if (c0 + j < n2)
      for (int q = 0; q < ranges; ++q) s += wp[((int64_t)q * kQb + i) * ldw + 32 + c0 + j];
    W[i][j] = s;
  }
  __syncthreads();
  const int half = lane >> 4, g16 = lane & 15, col = 2 * (tid >> 5) + half;
  const double t0 = g16 < w ? tau[g16] : 0.0, t1 = g16 + 16 < w ? tau[g16 + 16] : 0.0;
  double x0 = W[g16][col], x1 = W[g16 + 16][col];
#pragma unroll
  for (int kb = 0; kb < 2; ++kb)
    for (int kk = 0; kk < 16; ++kk) {
      const int k = 16 * kb + kk;
      if (g16 == kk) (kb ? x1 : x0) *= kb ? t1 : t0;
      const double yk = __shfl_sync(kFull, kb ? x1 : x0, (lane & 16) | kk);
      if (kb == 0 && g16 > kk) x0 = fma(-G[k][g16], yk, x0);
      if (kb == 0 || g16 > kk) x1 = fma(-G[k][g16 + 16], yk, x1);
    }
  if (c0 + col < n2) {
    y[(int64_t)g16 * ldy + c0 + col] = x0;
    y[(int64_t)(g16 + 16) * ldy + c0 + col] = x1;
  }
}

// C -= V Y (K = 32) by FP64 MMAs, 32 x 32 per CTA.
__global__ void __launch_bounds__(128) qr_update_kernel(double* c, int64_t ldc, int M, int N,
                                                        const double* __restrict__ v, const double* __restrict__ y,
                                                        int64_t ldy) {
  __shared__ double Vs[32][36], Ys[32][36];
  const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wr = (warp >> 1) * 16, wc = (warp & 1) * 16;
  const int g = lane >> 2, t4 = lane & 3;
  double cv[2][2][2];
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = r0 + wr + 8 * x + g, cc = c0 + wc + 8 * q + 2 * t4 + e;
        cv[x][q][e] = (r < M && cc < N) ? c[(int64_t)r * ldc + cc] : 0.0;
      }
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int r = warp + 4 * e;
    Vs[r][lane] = r0 + r < M ? v[(int64_t)(r0 + r) * kQb + lane] : 0.0;
    Ys[r][lane] = c0 + lane < N ? y[(int64_t)r * ldy + c0 + lane] : 0.0;
  }
  __syncthreads();
  double acc[2][2][2] = {};
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    double af[2], bf[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      af[q] = Vs[wr + 8 * q + g][k + t4];
      bf[q] = Ys[k + t4][wc + 8 * q + g];
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int q = 0; q < 2; ++q) qr_dmma(acc[x][q][0], acc[x][q][1], af[x], bf[q]);
  }
#pragma unroll
  for (int x = 0; x < 2; ++x)
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = r0 + wr + 8 * x + g, cc = c0 + wc + 8 * q + 2 * t4 + e;
        if (r < M && cc < N) c[(int64_t)r * ldc + cc] = cv[x][q][e] - acc[x][q][e];
      }
}

// st->singular = 0 if an element of A is NaN or infinite: a warp a row, so that the
// loads are whole lines whatever lda is.
__global__ void __launch_bounds__(256) qr_finite_kernel(const double* __restrict__ a, int64_t lda, int m, int n,
                                                        DeviceStatus* st) {
  const int lane = threadIdx.x & 31;
  bool bad = false;
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < m; r += gridDim.x * 8) {
    const double* row = a + (int64_t)r * lda;
#pragma unroll 4
    for (int c = lane; c < n; c += 32) bad |= !isfinite(row[c]);
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) st->singular = 0;
}

size_t panel_smem(int rows_per) { return (size_t)rows_per * kQbLd * sizeof(double); }

// CTAs: a power of two with at least 16 rows each.
void panel_split(luhot_ctx* ctx, int rows, int* P, int* rows_per) {
  *P = 1;
  while (*P < std::min(ctx->panel_cluster, kQbMaxCtas) && *P * 16 < rows) *P *= 2;
  *rows_per = (rows + *P - 1) / *P;
}

// Row ranges of qr_w_kernel: enough CTAs for two per SM, at least 64 rows each.
int w_ranges(luhot_ctx* ctx, int rows, int tiles) {
  const int want = (2 * ctx->num_sms + tiles - 1) / tiles;
  return std::max(1, std::min({want, (rows + 63) / 64, 16}));
}

}  // namespace

bool geqrf_blocked_fits(luhot_ctx* ctx, int m, int n) {
  // Below 32 columns there is no trailing block to gain from.
  if (std::min(m, n) < kQb || ctx->panel_cluster < 1) return false;
  int P, rows_per;
  panel_split(ctx, m, &P, &rows_per);
  return panel_smem(rows_per) + kQbStatic <= (size_t)ctx->max_smem_optin;
}

int geqrf_all_finite(luhot_ctx* ctx, int m, int n, const double* a, int64_t lda, bool* finite) {
  int rc = reset_status(ctx);
  if (rc) return rc;
  qr_finite_kernel<<<std::min((m + 7) / 8, 8 * ctx->num_sms), 256, 0, ctx->stream>>>(a, lda, m, n, ctx->d_status);
  LUHOT_CUDA_TRY(ctx, cudaGetLastError());
  int64_t first = -1;
  rc = finish_status(ctx, &first);
  *finite = first < 0;
  return rc;
}

int geqrf_blocked(luhot_ctx* ctx, int m, int n, double* a, int64_t lda, double* tau) {
  const int k = std::min(m, n);
  cudaStream_t stream = ctx->stream;
  const int64_t ldy = (n + 31) / 32 * 32, ldw = ldy + 32;
  const size_t v_elems = (size_t)m * kQb, y_elems = (size_t)kQb * ldy, w_elems = 16 * (size_t)kQb * ldw;
  int rc = ensure_buf(ctx, ctx->work[2], (v_elems + y_elems + w_elems) * sizeof(double));
  if (rc) return rc;
  double* v = static_cast<double*>(ctx->work[2].ptr);
  double* y = v + v_elems;
  double* wp = y + y_elems;
  LUHOT_CUDA_TRY(ctx, allow_max_dynamic_smem(qr_panel_kernel));
  LUHOT_CUDA_TRY(ctx, allow_wide_clusters(reinterpret_cast<const void*>(qr_panel_kernel)));
  rc = reset_status(ctx);
  if (rc) return rc;
  for (int k0 = 0; k0 < k; k0 += kQb) {
    const int w = std::min(kQb, k - k0), rows = m - k0, n2 = n - k0 - w;
    double* at = a + (int64_t)k0 * lda + k0;
    QrPanelArgs args;
    args.a = at;
    args.lda = lda;
    args.rows = rows;
    args.w = w;
    args.tau = tau + k0;
    args.v = v;
    args.st = ctx->d_status;
    int P;
    panel_split(ctx, rows, &P, &args.rows_per);
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = cl_config(P, kQbThreads, panel_smem(args.rows_per), stream, &attr);
    prof_begin(ctx, kProfPanel);
    LUHOT_CUDA_TRY(ctx, cudaLaunchKernelEx(&cfg, qr_panel_kernel, args));
    prof_end(ctx, kProfPanel, 2.0 * rows * w * w, 24.0 * rows * w);
    if (n2 <= 0) continue;
    double* a2 = at + w;
    const int tiles = (n2 + 31) / 32 + 1, ranges = w_ranges(ctx, rows, tiles);
    const int rows_per = ((rows + ranges - 1) / ranges + 31) / 32 * 32;
    prof_begin(ctx, kProfTrsm);
    qr_w_kernel<<<dim3(tiles, ranges), 128, 0, stream>>>(v, a2, lda, rows, n2, rows_per, wp, ldw);
    prof_end(ctx, kProfTrsm, 2.0 * rows * kQb * (n2 + kQb), 8.0 * rows * n2);
    prof_begin(ctx, kProfTrsm);
    qr_y_kernel<<<(n2 + 7) / 8, 128, 0, stream>>>(wp, ldw, ranges, tau + k0, w, n2, y, ldy);
    prof_end(ctx, kProfTrsm, (double)kQb * kQb * n2, 8.0 * kQb * n2 * (ranges + 1));
    LUHOT_CUDA_TRY(ctx, cudaGetLastError());
    prof_begin(ctx, kProfGemm);
    qr_update_kernel<<<dim3((n2 + 31) / 32, (rows + 31) / 32), 128, 0, stream>>>(a2, lda, rows, n2, v, y, ldy);
    prof_end(ctx, kProfGemm, 2.0 * rows * n2 * kQb, 16.0 * rows * n2);
    LUHOT_CUDA_TRY(ctx, cudaGetLastError());
  }
  // Its panels wait on one another: a wait that gave up is reported by this call, and
  // the status and workspace are free when it returns.
  return finish_status(ctx, nullptr);
}

}  // namespace luhot
