// FP64 Schur update on the FP16 tensor cores (Ozaki scheme, see ozaki.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "swap_solve.cuh"

struct luhot_ctx;

namespace luhot {

// Workspace of ozaki_update for a trailing block of at most m rows and n
// columns: the FP16 digit slices of L21 and U12 and their exponents.
size_t ozaki_workspace_bytes(int m, int n);
// The device has the shared memory and the driver the tensor-map encoder.
bool ozaki_available(luhot_ctx* ctx);
// a[r1..m, c1..n] -= a[r1..m, k0..k0+w] a[k0..k0+w, c1..n] for the row-major
// FP64 matrix a (lda), w <= 128; ws holds
// ozaki_workspace_bytes(m - r1, n - c1) bytes.  Asynchronous on `stream`.
int ozaki_update(luhot_ctx* ctx, double* a, int64_t lda, int k0, int w, int r1, int m, int c1, int n, void* ws,
                 cudaStream_t stream);
// c (M x N, ldc) -= l (M x w, ldl) u (w x N, ldu), w <= 128, separate operands.
int ozaki_product(luhot_ctx* ctx, const double* l, int64_t ldl, const double* u, int64_t ldu, int w, double* c,
                  int64_t ldc, int M, int N, void* ws, cudaStream_t stream);
// ozaki_update in two parts: where the digit slices of the operands go (for
// launch_swap_solve), and the product of the slices that are there (w <= 64).
SplitOut ozaki_split_out(void* ws, int r1, int M, int N);
int ozaki_update_split(luhot_ctx* ctx, double* a, int64_t lda, int w, int r1, int m, int c1, int n, void* ws,
                       cudaStream_t stream);

}  // namespace luhot
