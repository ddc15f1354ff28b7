// Row interchanges, U12 solve and operand split of one block step (see
// swap_solve.cu).
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

struct luhot_ctx;

namespace luhot {

// Where the digit slices of the tensor-core FP64 update go (ozaki.cuh): rows
// [r1, r1 + M) of the panel's columns and the right columns.
struct SplitOut {
  __half* as = nullptr;
  int* ea = nullptr;
  int r1 = 0, M = 0;
  __half* bs = nullptr;
  int* eb = nullptr;
};

// One launch, for the panel of columns [k0, k0 + w) that is factored:
//   columns [cl0, cl1) and [cr0, cr1): the panel's interchanges (`moves`, the
//     list it reported, kPanelMovesBytes; nullptr: none);
//   columns [cr0, cr1): rows [k0, k0 + w) <- L11^-1 rows [k0, k0 + w);
//   split (FP64, w <= 64; nullptr: none): the digit slices of both operands of
//     the update that follows.
template <typename T, bool kExact>
int launch_swap_solve(luhot_ctx* ctx, T* a, int64_t lda, const int* moves, int k0, int w, int cl0, int cl1, int cr0,
                      int cr1, const SplitOut* split, cudaStream_t stream);

}  // namespace luhot
