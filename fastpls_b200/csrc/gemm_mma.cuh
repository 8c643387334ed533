// The FP64 tensor-core GEMM kernel's launch (gemm_mma.cu) and its schedule
// (gemm.cu).
#pragma once

#include "kernels.cuh"

namespace fpls {

// Block tile (128 x 128, 64, 32 or 16, or 64 x 64) and slices over K.
struct GemmPlan {
  int tm = 128, tn = 128, splits = 1;
};
GemmPlan gemm_plan(int M, int N, int K, bool lower, int k_slice);

// C (or, with plan.splits > 1, slice z at C + z * split_stride) = alpha
// op(A) op(B) - coff (+ beta C) over the whole K (or the slice's part of it);
// with g.lower only the block tiles on and below the diagonal.
void gemm_mma_launch(const GemmArgs& g, const GemmPlan& plan, double* C, long ldc, long split_stride,
                     double alpha, double beta, const double* coff, cudaStream_t stream);

}  // namespace fpls
