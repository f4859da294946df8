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
// A launch whose contraction is long against its tiles is cut into slices that a second kernel sums in slice order, so the
// result does not depend on the launch; `scratch` (or null) holds the slice results, with too little of it the slices
// get longer.
int gemm_fp32(ltca_ctx* ctx, const Gemm32Problem* p, int n, int ta, int tb, bool sum, float* scratch = nullptr,
              size_t scratch_bytes = 0);

}  // namespace ltca
