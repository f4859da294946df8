// Internal interface of the exact (fp32 FMA) products of the module (gemm_fp32.cu).
#pragma once

#include "host_common.h"

namespace ltca {

// C[M,N] = op(A) op(B) (+ bias[N]); row-major storage with row pitches in elements.
struct Gemm32Problem {
    const float *A, *B, *bias;
    float* C;
    int M, N, K;
    int lda, ldb, ldc;
};
constexpr int kMaxGemm32 = 4;

// Up to four products of the same operand form in one launch.
//   ta == 0: A is [M,K], ta == 1: A is stored [K,M];  tb == 0: B is [K,N], tb == 1: B is stored [N,K].
//   sum: the products have one shape and one result, C of problem 0 = sum of them in order (each summed by itself first).
// A launch whose contraction is long against its tiles is cut into slices that a second kernel sums in slice order: the
// same bits every time on one device and with one size of scratch, which the number of slices follows.  `scratch` (or
// null: no slices) holds the slice results, with too little of it the slices get longer; with it the products take no bias.
//   any_order: the sums need not run in ascending order of the contraction.  What the attention kernels read (the Q, K, V
//   projections, the gradient at the context) keeps that order, so that it does not depend on the tile a launch takes.
int gemm_fp32(ltca_ctx* ctx, const Gemm32Problem* p, int n, int ta, int tb, bool sum, bool any_order, float* scratch = nullptr,
              size_t scratch_bytes = 0);
// The gradients behind the attention backward: dx = sum of n_dx products A [M,K] B [N,K], and n_dw products A [K,M] B [K,N];
// one launch for both where they are small.
int gemm_fp32_grads(ltca_ctx* ctx, const Gemm32Problem* dx, int n_dx, const Gemm32Problem* dw, int n_dw, float* scratch,
                    size_t scratch_bytes);

}  // namespace ltca
