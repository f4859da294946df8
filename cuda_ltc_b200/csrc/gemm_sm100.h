// Internal interface of the tensor-pipe projection GEMM (gemm_sm100.cu).
#pragma once

#include "host_common.h"
#include "sm100_ptx.cuh"

namespace ltca {

// A bf16 matrix operand in HBM.  mn_major == 0: stored [M or N, K] (K contiguous);
// mn_major == 1: stored [K, M or N].  `ld` is the row pitch in elements, a multiple of 8.
struct GemmOperand {
    const void* ptr;
    int64_t ld;
    int mn_major;
};

// C_i[M,N] = A_i B_i (+ bias_i) for i < n_problems (n_sum == 1), or
// C_0[M,N] = sum_{p < n_sum} A_p B_p (+ bias_0)            (n_problems == 1).
constexpr int kMaxGemmProblems = 4;
struct GemmProblem {
    int M = 0, N = 0, K = 0;
    int n_problems = 1, n_sum = 1;
    int ksplit = 1;                 // > 1: K range cut into slices, summed in order from `partial`
    GemmOperand a[kMaxGemmProblems] = {}, b[kMaxGemmProblems] = {};
    void* c[kMaxGemmProblems] = {};
    const float* bias[kMaxGemmProblems] = {};
    int64_t ldc = 0;
    int out_bf16 = 0;               // result element type: bf16 or fp32
    void* c_lo = nullptr;           // with out_bf16, one problem, no split of K: also write bf16(x - bf16(x)) here,
                                    // laid out like C, so that C + c_lo carry 16 significant bits of the fp32 result
    float* partial = nullptr;       // gemm_sm100_partial_bytes() bytes when ksplit > 1
    // A grid of batch_h x batch_b independent products of the same shape (heads x sequences of the materialised
    // attention path): operand i of batch entry (h, b) starts h * bs[0] + b * bs[1] elements after its pointer.
    // Needs n_problems == 1 and ksplit == 1 (n_sum is allowed); strides must keep 16-byte alignment.
    int batch_h = 1, batch_b = 1;
    int64_t a_bs[2] = {0, 0}, b_bs[2] = {0, 0}, c_bs[2] = {0, 0};
    int a_shared = 0, b_shared = 0; // every head of the batch (or of the sum) reads the same A / B
    int sum_h = 1;                  // > 1, batch_h == 1: C_b = sum over h < sum_h of A_hb B_hb, the heads one after the other in
                                    // one accumulator (a_bs[0], b_bs[0] as in a batch)
    int add_to_c = 0;               // fp32 results without a split of K: C += ... (one add per element, so the bits are
                                    // those of any other run)
};

int gemm_sm100(ltca_ctx* ctx, const GemmProblem& gp);

// Up to five products in one launch, each of its own shape, operand forms and number of summed terms, for every one
// of `heads` (strides a_hs, b_hs, c_hs between them).  c_lo as in GemmProblem.  Results need 16-byte aligned rows
// (gemm_group_aligned).  ksplit > 1 (one head, fp32 results, rows of N): `c` takes the slices, [ksplit][M][N], for sum_splits.
constexpr int kMaxGemmGroup = 5;
struct GemmGroup {
    struct Member {
        int M = 0, N = 0, K = 0, ksplit = 1;
        int terms = 1;
        GemmOperand a[3] = {}, b[3] = {};
        int64_t a_hs = 0, b_hs = 0, c_hs = 0, ldc = 0;
        void* c = nullptr;
        void* c_lo = nullptr;
    };
    int heads = 1, n = 0, out_bf16 = 0;
    Member m[kMaxGemmGroup];
};
// Whether all its tiles fit beside one another on the SMs as 128 x 128 ones: then a launch of its own for each of its members
// would leave SMs idle.
bool gemm_group_one_wave(const ltca_ctx* ctx, const GemmGroup& gg);
bool gemm_group_aligned(const GemmGroup& gg);
int gemm_sm100_group(ltca_ctx* ctx, const GemmGroup& gg);
// dst[i][e] = sum over s < ksplit of partial[i][s][e], e < mn, in slice order.
int sum_splits(ltca_ctx* ctx, const float* partial, void* const* dst, int n, int64_t mn, int ksplit);
int gemm_sm100_pick_ksplit(int M, int N, int K, int n_problems, int sm_count);
size_t gemm_sm100_partial_bytes(int M, int N, int n_problems, int ksplit);
// dst[r, c] = bf16(src[r, c]) for a [rows, cols] block with row pitches ld_src / ld_dst (elements).
int convert_rows_bf16(ltca_ctx* ctx, const float* src, int64_t ld_src, void* dst, int64_t ld_dst, int64_t rows,
                      int cols);
// Several matrices of any sizes whose 16-byte pieces form one index range: what one launch rounds to bf16.
constexpr int kMaxCvtMany = 6;
struct CvtMany {
    const float* src[kMaxCvtMany];
    __nv_bfloat16* dst[kMaxCvtMany];
    __nv_bfloat16* lo[kMaxCvtMany];         // second term bf16(x - bf16(x)), laid out like dst, or null
    int64_t ld_src[kMaxCvtMany], ld_dst[kMaxCvtMany];
    uint32_t cols4[kMaxCvtMany];
    uint32_t start4[kMaxCvtMany + 1];       // first piece of matrix m; start4[n] = all pieces
    int n;
};
// Fills `b`; false when a matrix has rows that are no multiple of 16 bytes (those go one at a time).
bool make_cvt_many(CvtMany* b, int n, const float* const* src, const int64_t* ld_src, void* const* dst, const int64_t* ld_dst,
                   const int64_t* rows, const int* cols, void* const* lo);
// The same for up to six matrices of any sizes in one launch (16-byte aligned rows; otherwise one launch each).
// `lo` (or an entry of it) non-null: also the second term bf16(x - bf16(x)), laid out like the first.
int convert_many_bf16(ltca_ctx* ctx, int n, const float* const* src, const int64_t* ld_src, void* const* dst,
                      const int64_t* ld_dst, const int64_t* rows, const int* cols, void* const* lo = nullptr);

#ifdef __CUDACC__
// Pieces i, i + step, ... of the range.
__device__ __forceinline__ void cvt_many_pieces(const CvtMany& b, uint32_t i, uint32_t step) {
    const uint32_t total = b.start4[b.n];
    for (; i < total; i += step) {
        int m = 0;
        while (m + 1 < b.n && i >= b.start4[m + 1]) ++m;
        const uint32_t j = i - b.start4[m];
        const uint32_t r = j / b.cols4[m], c4 = j - r * b.cols4[m];
        const float4 v = __ldg(reinterpret_cast<const float4*>(b.src[m] + (int64_t)r * b.ld_src[m]) + c4);
        const uint2 h = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
        reinterpret_cast<uint2*>(b.dst[m] + (int64_t)r * b.ld_dst[m])[c4] = h;
        if (b.lo[m]) {
            const uint2 l = make_uint2(pack_bf16x2(v.x - __uint_as_float(h.x << 16), v.y - __uint_as_float(h.x & 0xffff0000u)),
                                       pack_bf16x2(v.z - __uint_as_float(h.y << 16), v.w - __uint_as_float(h.y & 0xffff0000u)));
            reinterpret_cast<uint2*>(b.lo[m] + (int64_t)r * b.ld_dst[m])[c4] = l;
        }
    }
}
#endif

}  // namespace ltca
