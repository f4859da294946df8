// TimeSelfAttention module: out = LayerNorm(x + MHA(x)) and its backward, as the reference's
// CuDNNTimeSelfAttention computes them (reference src/ml/cudnn_time_self_attention.cu:211-368
// with the attention configured by include/cuDNN_ops.h:152-178).
//
// Data flow of the forward (all buffers fp32, row = one (batch, time) position):
//   x [rows,E] --Wq,Wk,Wv--> q,k,v [rows,H*W] --attention core--> ctx [rows,H*W] --Wo--> y [rows,E]
//   out = LayerNorm(y + x)        (residual and LayerNorm fused into one row pass)
// The attention core reads q/k/v and writes ctx through strided [B,H,S,W] views of the
// row-major projection buffers, so the reference's reshape kernels
// (src/ml/flash_attention.cu:402-455) have no counterpart here.
//
// Two pipelines:
//   - exact (LTCA_MODE_FP32, or shapes the tensor-pipe attention kernels do not cover): fp32 FMA GEMMs,
//     fp32 buffers between the kernels;
//   - tensor pipe (other modes): x, dy and the weights are rounded to bf16 once, every projection is
//     a tcgen05 GEMM (gemm_sm100.cu), q / k / v / ctx and their gradients stay in bf16 between the
//     kernels (the attention kernels read them through strides, nothing is packed or permuted), Q, K
//     and V share one launch, dx is one GEMM over the three (dq, W^T) pairs, the weight gradients
//     split their long contraction (batch x time) across CTAs and are summed in a fixed order.
// Backward follows the reference:
// the incoming gradient passes through LayerNorm and the residual unchanged
// (src/ml/cudnn_time_self_attention.cu:291-299), dx = dQ Wq^T + dK Wk^T + dV Wv^T.
#include "attn_mask.cuh"
#include "gemm_fp32.h"
#include "gemm_sm100.h"
#include "attn_wide.h"
#include "host_common.h"
#include "sm100_ptx.cuh"

namespace ltca {

namespace {

// Where a row of results goes: fp32, bf16, or both; rows are `ld` elements apart in either.
struct RowOut {
    float* f32;
    __nv_bfloat16* bf16;
    int64_t ld_f32, ld_bf16;
};
__device__ __forceinline__ void put4(const RowOut& o, int64_t row, int c, float4 v) {
    if (o.f32) *reinterpret_cast<float4*>(o.f32 + row * o.ld_f32 + c) = v;
    if (o.bf16) *reinterpret_cast<uint2*>(o.bf16 + row * o.ld_bf16 + c) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
}
__device__ __forceinline__ void put1(const RowOut& o, int64_t row, int c, float v) {
    if (o.f32) o.f32[row * o.ld_f32 + c] = v;
    if (o.bf16) o.bf16[row * o.ld_bf16 + c] = __float2bfloat16_rn(v);
}

__device__ __forceinline__ float warp_total(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float4 ldg4(const float* row, int i) { return __ldg(reinterpret_cast<const float4*>(row) + i); }

// Rows of up to 1024 floats that stay in a warp's registers, E / 128 pieces of 16 bytes per lane: kN4 of them, where the loads of
// a row all go out before the first is waited for, or (0) as many as E says, one after the other.  With few rows per SM a row
// kernel lasts as long as one row's chain of loads and sums: residual + LayerNorm of 32768 x 512 37.5 us with one piece at a
// time, 28.2 so (192 MB); 8192 x 512 12.3 and 10.3; module forward of 32768 rows of 128 52.9 and 47.1, of 384 139 and 135, of 1024
// 398 and 390.  (The prepare launch below, whose other parts need the warps that the registers would cost, 7.7 us with one at a
// time, 9.8 with all.)
int row_pieces(int E) { return (E & 127) == 0 && E <= 1024 ? E >> 7 : 0; }
template <int kN4>
struct RowPieces {
    static constexpr int kMax = kN4 > 0 ? kN4 : 8;
    int n;
    __device__ __forceinline__ explicit RowPieces(int E) : n(kN4 > 0 ? kN4 : E >> 7) {}
    __device__ __forceinline__ bool has(int i) const { return kN4 > 0 || i < n; }
};

template <int kN4>
__device__ __forceinline__ void layer_norm_pieces(const float* __restrict__ yr, const float* __restrict__ xr, const float* __restrict__ gamma,
                                                  const float* __restrict__ beta, const RowOut& out, int64_t row, int E, bool use_res,
                                                  float eps) {
    const RowPieces<kN4> p(E);
    constexpr int kMax = RowPieces<kN4>::kMax;
    constexpr bool kEarly = kN4 > 0 && kN4 <= 4;       // gamma and beta with the row, while registers last
    const int lane = threadIdx.x & 31;
    float4 v[kMax], r[kN4 > 0 ? kMax : 1], gm[kEarly ? kMax : 1], bt[kEarly ? kMax : 1];
    const float4 one = make_float4(1.f, 1.f, 1.f, 1.f), zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kMax; ++i)
        if (p.has(i)) {
            v[i] = ldg4(yr, lane + 32 * i);
            if constexpr (kN4 > 0) r[i] = use_res ? ldg4(xr, lane + 32 * i) : zero;
        }
    if constexpr (kEarly) {
#pragma unroll
        for (int i = 0; i < kMax; ++i) {
            gm[i] = gamma ? ldg4(gamma, lane + 32 * i) : one;
            bt[i] = beta ? ldg4(beta, lane + 32 * i) : zero;
        }
    }
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < kMax; ++i)
        if (p.has(i)) {
            if (use_res) {
                const float4 x = kN4 > 0 ? r[kN4 > 0 ? i : 0] : ldg4(xr, lane + 32 * i);
                v[i].x += x.x; v[i].y += x.y; v[i].z += x.z; v[i].w += x.w;
            }
            sum += (v[i].x + v[i].y) + (v[i].z + v[i].w);
        }
    const float mean = warp_total(sum) / E;
    float var = 0.f;
#pragma unroll
    for (int i = 0; i < kMax; ++i)
        if (p.has(i)) {
            const float a = v[i].x - mean, b = v[i].y - mean, c = v[i].z - mean, d = v[i].w - mean;
            var = fmaf(a, a, var); var = fmaf(b, b, var); var = fmaf(c, c, var); var = fmaf(d, d, var);
        }
    const float inv = rsqrtf(warp_total(var) / E + eps);
#pragma unroll
    for (int i = 0; i < kMax; ++i)
        if (p.has(i)) {
            const float4 g = kEarly ? gm[kEarly ? i : 0] : gamma ? ldg4(gamma, lane + 32 * i) : one;
            const float4 t = kEarly ? bt[kEarly ? i : 0] : beta ? ldg4(beta, lane + 32 * i) : zero;
            put4(out, row, 4 * (lane + 32 * i), make_float4((v[i].x - mean) * inv * g.x + t.x, (v[i].y - mean) * inv * g.y + t.y,
                                                            (v[i].z - mean) * inv * g.z + t.z, (v[i].w - mean) * inv * g.w + t.w));
        }
}

// One row by one warp: LayerNorm(y (+ x)), or just the sum / a copy.  `vec`: every row of every operand starts on a
// 16-byte boundary and E is a multiple of 4.  kN4 > 0: rows of 128 kN4 floats, all of a row's loads in flight (see RowPieces).
template <int kN4>
__device__ __forceinline__ void layer_norm_row(const float* __restrict__ y, const float* __restrict__ x,
                                               const float* __restrict__ gamma, const float* __restrict__ beta, const RowOut& out,
                                               int64_t row, int E, bool use_res, bool use_ln, float eps, bool vec) {
    const int lane = threadIdx.x & 31;
    const float* yr = y + row * E;
    const float* xr = x + row * E;
    if (use_ln && vec && (E & 127) == 0 && E <= 1024) {
        // one read of y and x, one write of the result
        layer_norm_pieces<kN4>(yr, xr, gamma, beta, out, row, E, use_res, eps);
        return;
    }
    auto value = [&](int i) { return yr[i] + (use_res ? xr[i] : 0.f); };
    if (!use_ln) {
        for (int i = lane; i < E; i += 32) put1(out, row, i, value(i));
        return;
    }
    // any width: the lane's elements are formed again for each pass
    float sum = 0.f;
    for (int i = lane; i < E; i += 32) sum += value(i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float mean = sum / E;
    float var = 0.f;
    for (int i = lane; i < E; i += 32) {
        const float d = value(i) - mean;
        var = fmaf(d, d, var);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) var += __shfl_xor_sync(0xffffffffu, var, o);
    const float inv_std = rsqrtf(var / E + eps);
    for (int i = lane; i < E; i += 32)
        put1(out, row, i, fmaf((value(i) - mean) * inv_std, gamma ? gamma[i] : 1.f, beta ? beta[i] : 0.f));
}
__host__ __device__ __forceinline__ bool aligned16(const void* a, const void* b, const void* c, const void* d, const void* e) {
    return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c) |
             reinterpret_cast<uintptr_t>(d) | reinterpret_cast<uintptr_t>(e)) & 15) == 0;
}

template <int kN4>
__global__ void residual_layer_norm_kernel(const float* __restrict__ y, const float* __restrict__ x,
                                           const float* __restrict__ gamma,
                                           const float* __restrict__ beta, float* __restrict__ out,
                                           int64_t rows, int E, int use_res, int use_ln, float eps) {
    grid_dependency_wait();
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const RowOut o{out, nullptr, E, 0};
    layer_norm_row<kN4>(y, x, gamma, beta, o, row, E, use_res != 0, use_ln != 0, eps, aligned16(y, x, gamma, beta, out));
    // y is scratch and this was its only reader: whole lines of it that still lie in L2 need not be written to HBM
    // (32768 x 512: 45.3 -> 43.6 us, and the module forward of 8192 rows 58.6 -> 57.1).  The row's stores above depend on
    // every lane's loads, so nothing of it is still on its way.
    if ((E & 31) == 0 && (reinterpret_cast<uintptr_t>(y) & 127) == 0) {
        __syncwarp();
        for (int l = threadIdx.x & 31; l < E / 32; l += 32) discard_line(y + row * E + 32 * l);
    }
}

int residual_layer_norm(ltca_ctx* ctx, const ltca_tsa_params* t, const float* y, int64_t rows) {
    const int wpb = 8;
    auto kern = residual_layer_norm_kernel<0>;
    switch (row_pieces(t->E)) {
        case 1: kern = residual_layer_norm_kernel<1>; break;
        case 2: kern = residual_layer_norm_kernel<2>; break;
        case 3: kern = residual_layer_norm_kernel<3>; break;
        case 4: kern = residual_layer_norm_kernel<4>; break;
        case 5: kern = residual_layer_norm_kernel<5>; break;
        case 6: kern = residual_layer_norm_kernel<6>; break;
        case 7: kern = residual_layer_norm_kernel<7>; break;
        case 8: kern = residual_layer_norm_kernel<8>; break;
    }
    LTCA_CUDA_OK(ctx, launch_dependent(kern, dim3((unsigned)((rows + wpb - 1) / wpb)), dim3(wpb * 32),
                                       0, ctx->stream, y, t->x, t->ln_gamma, t->ln_beta, t->out, rows, t->E,
                                       t->use_residual, t->use_layer_norm, 1e-5f));
    return LTCA_OK;
}

// The end of a small exact forward in one launch: out = LayerNorm(x + ctx Wo + bo), a warp to a row of at most 64 columns, Wo in
// shared memory.  As a product and a row kernel these were two of the eight dependent launches of a small training step, each
// of which costs 3 to 4 us whatever it computes: step of B8 S32 E32 H4 32.3 -> 29.3 us, forward of B32 S128 E32 H4 34.8 -> 33.8.
// Every block reads all of Wo: with 64 KB of it 2048 rows of the forward B32 S64 E64 H8 width 32 take 33.9 us instead of 32.7,
// so it is limited to 32 KB and 4096 rows, and to the multiply-adds of 3072 rows with 32 KB.  Forward of 3072 rows with 8192
// weights 25.1 -> 24.5 us, of 4096 with 6144 34.7 -> 34.4, with 512 (E4) 22.7 -> 21.0; of 4096 with 7680 40.2 -> 41.8, with
// 8192 27.3 -> 28.3.
constexpr int kProjThreads = 256, kProjMaxE = 64, kProjMaxWeights = 8192, kProjRows = 4096;
constexpr int64_t kProjProducts = 3072ll * kProjMaxWeights;
__global__ void __launch_bounds__(kProjThreads) project_norm_kernel(const float* __restrict__ ctx, const float* __restrict__ wo,
                                                                    const float* __restrict__ bo, const float* __restrict__ x,
                                                                    const float* __restrict__ gamma, const float* __restrict__ beta,
                                                                    float* __restrict__ out, int rows, int HW, int E, int use_res, int use_ln,
                                                                    float eps) {
    grid_dependency_wait();
    extern __shared__ __align__(16) float proj_sm[];
    float* ws = proj_sm;                                       // [HW][E]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float* cs = proj_sm + HW * E + warp * HW;                  // this warp's row of ctx
    const int row = blockIdx.x * (kProjThreads / 32) + warp;
    const bool live = row < rows;
    for (int i = threadIdx.x; i < HW * E / 4; i += kProjThreads)
        reinterpret_cast<float4*>(ws)[i] = __ldg(reinterpret_cast<const float4*>(wo) + i);
    if (live)
        for (int i = lane; i < HW / 4; i += 32)
            reinterpret_cast<float4*>(cs)[i] = __ldg(reinterpret_cast<const float4*>(ctx + (int64_t)row * HW) + i);
    float v[kProjMaxE / 32], res[kProjMaxE / 32], gm[kProjMaxE / 32], bt[kProjMaxE / 32];
#pragma unroll
    for (int j = 0; j < kProjMaxE / 32; ++j) {
        const int c = lane + 32 * j;
        const bool in = live && c < E;
        res[j] = (in && use_res ? __ldg(x + (int64_t)row * E + c) : 0.f) + (in && bo ? __ldg(bo + c) : 0.f);
        gm[j] = in && gamma ? __ldg(gamma + c) : 1.f;
        bt[j] = in && beta ? __ldg(beta + c) : 0.f;
    }
    __syncthreads();
    if (!live) return;
#pragma unroll
    for (int j = 0; j < kProjMaxE / 32; ++j) {
        const int c = lane + 32 * j;
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        if (c < E) {
#pragma unroll 4
            for (int k = 0; k < HW; k += 4) {
                const float4 a = *reinterpret_cast<const float4*>(cs + k);
                acc[0] = fmaf(a.x, ws[k * E + c], acc[0]);
                acc[1] = fmaf(a.y, ws[(k + 1) * E + c], acc[1]);
                acc[2] = fmaf(a.z, ws[(k + 2) * E + c], acc[2]);
                acc[3] = fmaf(a.w, ws[(k + 3) * E + c], acc[3]);
            }
        }
        v[j] = (acc[0] + acc[1]) + (acc[2] + acc[3]) + res[j];
    }
    float mean = 0.f, inv = 1.f;
    if (use_ln) {
        float sum = 0.f, var = 0.f;
#pragma unroll
        for (int j = 0; j < kProjMaxE / 32; ++j) sum += v[j];      // (columns beyond E hold zeros)
        mean = warp_total(sum) / E;
#pragma unroll
        for (int j = 0; j < kProjMaxE / 32; ++j)
            if (lane + 32 * j < E) var = fmaf(v[j] - mean, v[j] - mean, var);
        inv = rsqrtf(warp_total(var) / E + eps);
    }
#pragma unroll
    for (int j = 0; j < kProjMaxE / 32; ++j)
        if (lane + 32 * j < E) out[(int64_t)row * E + lane + 32 * j] = use_ln ? fmaf((v[j] - mean) * inv, gm[j], bt[j]) : v[j];
}
// Whether that kernel takes the call (ctx is the library's own buffer, aligned and contiguous).
bool projects_and_norms(const ltca_tsa_params* t, int64_t rows, int HW) {
    return t->E <= kProjMaxE && (t->E % 4) == 0 && (HW % 4) == 0 && HW * t->E <= kProjMaxWeights && rows <= kProjRows &&
           rows * HW * t->E <= kProjProducts && (reinterpret_cast<uintptr_t>(t->wo) & 15) == 0;
}
int project_norm(ltca_ctx* ctx, const ltca_tsa_params* t, const float* core, int64_t rows, int HW) {
    static SmemOptIn once;
    constexpr int kMost = (kProjMaxWeights + kProjThreads / 32 * kProjMaxWeights / 4) * (int)sizeof(float);   // HW <= kProjMaxWeights / 4
    const int smem = (HW * t->E + kProjThreads / 32 * HW) * (int)sizeof(float);
    LTCA_CUDA_OK(ctx, opt_in_dynamic_smem(once, ctx->device, project_norm_kernel, kMost));
    constexpr int wpb = kProjThreads / 32;
    LTCA_CUDA_OK(ctx, launch_dependent(project_norm_kernel, dim3((unsigned)((rows + wpb - 1) / wpb)), dim3(kProjThreads), smem, ctx->stream,
                                       core, t->wo, t->bo, t->x, t->ln_gamma, t->ln_beta, t->out, (int)rows, HW, t->E, t->use_residual,
                                       t->use_layer_norm, 1e-5f));
    return LTCA_OK;
}

// ---- pieces of the FlashAttention form: dropout, LayerNorm backward, column sums -----------------

// u in [0,1) from (seed, element index): splitmix64 finaliser, top 24 bits.  The same function runs on the host
// in the oracle, so masks can be compared element by element.
__host__ __device__ inline float dropout_uniform(uint64_t seed, uint64_t idx) {
    uint64_t z = seed + (idx + 1) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (float)(z >> 40) * (1.0f / 16777216.0f);
}

// Inverted dropout of element i (reference src/ml/flash_attention.cu:380-399; the reference draws from curand with a
// time-dependent offset, so only the distribution can match).
__device__ __forceinline__ float dropout(float v, int64_t i, float p, float scale, uint64_t seed) {
    return dropout_uniform(seed, (uint64_t)i) >= p ? v * scale : 0.f;
}

// Everything the FlashAttention form does before its first product, in one launch whose blocks take one of four parts:
// packing of the dense mask, LayerNorm of the input rows, dropout of the incoming gradient, rounding of the weights to
// bf16.  As launches of their own (with a separate rounding of LayerNorm's and dropout's results) these were five of 13
// kernels of a few microseconds; the mask's took 6.5 us of latency in each direction of B16 S200.
struct PrepareArgs {
    const float *x, *gamma, *beta;      // rows [rows, E]; LayerNorm when use_ln, else a copy
    RowOut xo;
    const float* dy;                    // backward: gradient behind the dropout, [rows, E], or null
    RowOut go;
    int64_t rows;
    int E, use_ln;
    float eps, p;
    uint64_t seed;
    MaskArgs mask;                      // words to write, or no mask
    int B;
    int mask_blocks, row_blocks, dy_blocks;      // blocks of the first three parts
    CvtMany w;                          // matrices to round
};
constexpr int kPrepareThreads = 256;
__global__ void __launch_bounds__(kPrepareThreads) prenorm_prepare_kernel(const __grid_constant__ PrepareArgs a) {
    grid_dependency_wait();
    int block = blockIdx.x;
    if (block < a.mask_blocks) {
        write_mask_words(a.mask, a.B, (int64_t)block * (kPrepareThreads / 32) + (threadIdx.x >> 5), (int64_t)a.mask_blocks * (kPrepareThreads / 32));
        return;
    }
    block -= a.mask_blocks;
    if (block < a.row_blocks) {
        const int64_t row = (int64_t)block * (kPrepareThreads / 32) + (threadIdx.x >> 5);
        if (row >= a.rows) return;
        const bool vec = aligned16(a.x, a.gamma, a.beta, a.xo.f32, a.xo.bf16);
        layer_norm_row<0>(a.x, a.x, a.gamma, a.beta, a.xo, row, a.E, false, a.use_ln != 0, a.eps, vec);
        return;
    }
    block -= a.row_blocks;
    if (block < a.dy_blocks) {
        const float scale = 1.0f / (1.0f - a.p);
        const int64_t n = a.rows * a.E, first = (int64_t)block * kPrepareThreads + threadIdx.x;
        const int64_t step = (int64_t)a.dy_blocks * kPrepareThreads;
        if ((a.E & 3) == 0 && (a.go.ld_bf16 & 3) == 0 && n < (1ll << 32) && aligned16(a.dy, a.go.f32, a.go.bf16, nullptr, nullptr)) {
            const uint32_t e4 = (uint32_t)a.E / 4;
            for (int64_t i = first; i < n / 4; i += step) {
                const uint32_t row = (uint32_t)i / e4, c = ((uint32_t)i - row * e4) * 4;
                float4 v = __ldg(reinterpret_cast<const float4*>(a.dy) + i);
                if (a.p > 0.f) {
                    v.x = dropout(v.x, 4 * i, a.p, scale, a.seed);
                    v.y = dropout(v.y, 4 * i + 1, a.p, scale, a.seed);
                    v.z = dropout(v.z, 4 * i + 2, a.p, scale, a.seed);
                    v.w = dropout(v.w, 4 * i + 3, a.p, scale, a.seed);
                }
                put4(a.go, row, (int)c, v);
            }
            return;
        }
        for (int64_t i = first; i < n; i += step) {
            const int64_t row = i / a.E;
            const float v = a.p > 0.f ? dropout(a.dy[i], i, a.p, scale, a.seed) : a.dy[i];
            put1(a.go, row, (int)(i - row * a.E), v);
        }
        return;
    }
    block -= a.dy_blocks;
    cvt_many_pieces(a.w, (uint32_t)block * kPrepareThreads + threadIdx.x,
                    (gridDim.x - a.mask_blocks - a.row_blocks - a.dy_blocks) * kPrepareThreads);
}

// out = dropout(y (+ x)): the end of the FlashAttention form's forward.
__global__ void __launch_bounds__(256) residual_dropout_kernel(const float* __restrict__ y, const float* __restrict__ x, float* __restrict__ out,
                                                               int64_t n, int use_res, float p, uint64_t seed) {
    grid_dependency_wait();
    const float scale = 1.0f / (1.0f - p);
    const int64_t first = (int64_t)blockIdx.x * 256 + threadIdx.x, step = (int64_t)gridDim.x * 256;
    if ((n & 3) == 0 && aligned16(y, x, out, nullptr, nullptr)) {
        for (int64_t i = first; i < n / 4; i += step) {
            float4 v = __ldg(reinterpret_cast<const float4*>(y) + i);
            if (use_res) {
                const float4 r = __ldg(reinterpret_cast<const float4*>(x) + i);
                v.x += r.x; v.y += r.y; v.z += r.z; v.w += r.w;
            }
            if (p > 0.f) {
                v.x = dropout(v.x, 4 * i, p, scale, seed);
                v.y = dropout(v.y, 4 * i + 1, p, scale, seed);
                v.z = dropout(v.z, 4 * i + 2, p, scale, seed);
                v.w = dropout(v.w, 4 * i + 3, p, scale, seed);
            }
            reinterpret_cast<float4*>(out)[i] = v;
        }
        return;
    }
    for (int64_t i = first; i < n; i += step) {
        float v = y[i];
        if (use_res) v += x[i];
        out[i] = p > 0.f ? dropout(v, i, p, scale, seed) : v;
    }
}

// Its registers form: rows of 128 kN4 floats, read once in 16-byte pieces, with gamma and the residual in flight beside them.
template <int kN4>
__device__ __forceinline__ void layer_norm_bwd_pieces(const float* __restrict__ gr, const float* __restrict__ xr, const float* __restrict__ gamma,
                                                      const float* __restrict__ res, float* __restrict__ dx, float* __restrict__ prod, int E,
                                                      float eps) {
    const int lane = threadIdx.x & 31;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 xh[kN4], gv[kN4], gm[kN4], r[kN4];
#pragma unroll
    for (int i = 0; i < kN4; ++i) {
        xh[i] = ldg4(xr, lane + 32 * i);
        gv[i] = ldg4(gr, lane + 32 * i);
        gm[i] = ldg4(gamma, lane + 32 * i);
        r[i] = dx && res ? ldg4(res, lane + 32 * i) : zero;
    }
    float s0 = 0.f;
#pragma unroll
    for (int i = 0; i < kN4; ++i) s0 += (xh[i].x + xh[i].y) + (xh[i].z + xh[i].w);
    const float mean = warp_total(s0) / E;
    float s1 = 0.f;
#pragma unroll
    for (int i = 0; i < kN4; ++i) {
        xh[i].x -= mean; xh[i].y -= mean; xh[i].z -= mean; xh[i].w -= mean;
        s1 = fmaf(xh[i].x, xh[i].x, s1); s1 = fmaf(xh[i].y, xh[i].y, s1);
        s1 = fmaf(xh[i].z, xh[i].z, s1); s1 = fmaf(xh[i].w, xh[i].w, s1);
    }
    const float inv_std = rsqrtf(warp_total(s1) / E + eps);
    float a1 = 0.f, a2 = 0.f;
#pragma unroll
    for (int i = 0; i < kN4; ++i) {
        xh[i].x *= inv_std; xh[i].y *= inv_std; xh[i].z *= inv_std; xh[i].w *= inv_std;
        const float4 gg = make_float4(gv[i].x * gm[i].x, gv[i].y * gm[i].y, gv[i].z * gm[i].z, gv[i].w * gm[i].w);
        a1 += (gg.x + gg.y) + (gg.z + gg.w);
        a2 = fmaf(gg.x, xh[i].x, a2); a2 = fmaf(gg.y, xh[i].y, a2);
        a2 = fmaf(gg.z, xh[i].z, a2); a2 = fmaf(gg.w, xh[i].w, a2);
        if (prod)
            reinterpret_cast<float4*>(prod)[lane + 32 * i] =
                make_float4(gv[i].x * xh[i].x, gv[i].y * xh[i].y, gv[i].z * xh[i].z, gv[i].w * xh[i].w);
        gv[i] = gg;
    }
    if (!dx) return;
    const float m1 = warp_total(a1) / E, m2 = warp_total(a2) / E;
#pragma unroll
    for (int i = 0; i < kN4; ++i) {
        float4 d = r[i];
        d.x += inv_std * (gv[i].x - m1 - xh[i].x * m2);
        d.y += inv_std * (gv[i].y - m1 - xh[i].y * m2);
        d.z += inv_std * (gv[i].z - m1 - xh[i].z * m2);
        d.w += inv_std * (gv[i].w - m1 - xh[i].w * m2);
        reinterpret_cast<float4*>(dx)[lane + 32 * i] = d;
    }
}

// LayerNorm backward, one warp per row.  g = gradient at the LayerNorm output, x = its input.
//   dx = inv_std * (g*gamma - mean(g*gamma) - xhat * mean(g*gamma*xhat))  (+ res[row] when res != null)
// dx and prod are optional; prod receives g * xhat, whose column sums are dgamma.
template <int kN4>
__global__ void layer_norm_bwd_kernel(const float* __restrict__ g, const float* __restrict__ x,
                                      const float* __restrict__ gamma, const float* __restrict__ res,
                                      float* __restrict__ dx, float* __restrict__ prod, int64_t rows, int E,
                                      float eps) {
    grid_dependency_wait();
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const int lane = threadIdx.x & 31;
    const float* xr = x + row * E;
    const float* gr = g + row * E;
    if constexpr (kN4 > 0) {
        if (aligned16(g, x, gamma, res, dx) && (reinterpret_cast<uintptr_t>(prod) & 15) == 0) {
            const float* rr = res ? res + row * E : nullptr;
            float *dr = dx ? dx + row * E : nullptr, *pr = prod ? prod + row * E : nullptr;
            layer_norm_bwd_pieces<kN4>(gr, xr, gamma, rr, dr, pr, E, eps);
            return;
        }
    }
    float sum = 0.f;
    for (int i = lane; i < E; i += 32) sum += xr[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float mean = sum / E;
    float var = 0.f;
    for (int i = lane; i < E; i += 32) { const float d = xr[i] - mean; var = fmaf(d, d, var); }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) var += __shfl_xor_sync(0xffffffffu, var, o);
    const float inv_std = rsqrtf(var / E + eps);
    float m1 = 0.f, m2 = 0.f;
    for (int i = lane; i < E; i += 32) {
        const float xh = (xr[i] - mean) * inv_std;
        const float gg = gr[i] * gamma[i];
        m1 += gg;
        m2 = fmaf(gg, xh, m2);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m1 += __shfl_xor_sync(0xffffffffu, m1, o);
        m2 += __shfl_xor_sync(0xffffffffu, m2, o);
    }
    m1 /= E; m2 /= E;
    for (int i = lane; i < E; i += 32) {
        const float xh = (xr[i] - mean) * inv_std;
        const float gi = gr[i];
        if (dx) {
            float v = inv_std * (gi * gamma[i] - m1 - xh * m2);
            if (res) v += res[row * E + i];
            dx[row * E + i] = v;
        }
        if (prod) prod[row * E + i] = gi * xh;
    }
}

// Column sums of up to six [rows, cols] matrices in two fixed-order stages (no atomics): kColChunks row chunks, then
// the chunks.  One launch per stage for all of them: each is a microsecond of reading behind two of launching.
constexpr int kColChunks = 64, kMaxColJobs = 6;
struct ColSum {
    const void* src[kMaxColJobs];
    float* dst[kMaxColJobs];
    int64_t ld[kMaxColJobs];
    int cols[kMaxColJobs], bf16[kMaxColJobs];
    int64_t rows;
    int n, max_cols;
    float* partial;                     // [n][kColChunks][max_cols]
    // What module_tail also does where `tail` says that one follows: the slices of split products (sum_splits) ...
    bool tail;
    const float* split;
    float* split_dst[kMaxGemmProblems];
    int64_t split_mn;
    int splits, split_n;
    // ... and the LayerNorm's backward, whose products' column sums go to ln_partial, [chunks of ln_rows rows][2][E]
    const float *ln_g, *ln_x, *ln_gamma, *ln_res;
    float *ln_dx, *ln_partial, *ln_dgamma, *ln_dbeta;
    int E, ln_rows, ln_chunks;
    int ln_blocks, col_blocks;          // blocks of the launch; the slices' come behind them
    float eps;
    void add(const void* s, bool is_bf16, int64_t pitch, int c, float* d) {
        if (!d) return;
        src[n] = s; dst[n] = d; ld[n] = pitch; cols[n] = c; bf16[n] = is_bf16 ? 1 : 0;
        if (c > max_cols) max_cols = c;
        ++n;
    }
};
__device__ __forceinline__ float ld_f(const float* p) { return *p; }
__device__ __forceinline__ float ld_f(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T>
__device__ __forceinline__ float column_chunk(const T* src, int64_t ld, int64_t r0, int64_t r1) {
    float acc = 0.f;
#pragma unroll 16
    for (int64_t r = r0; r < r1; ++r) acc += ld_f(src + r * ld);
    return acc;
}
__device__ __forceinline__ void column_partial(const ColSum& a, int j, int chunk, int c) {
    const int64_t per = (a.rows + kColChunks - 1) / kColChunks;
    const int64_t r0 = chunk * per, r1 = r0 + per < a.rows ? r0 + per : a.rows;
    a.partial[((int64_t)j * kColChunks + chunk) * a.max_cols + c] =
        a.bf16[j] ? column_chunk(static_cast<const __nv_bfloat16*>(a.src[j]) + c, a.ld[j], r0, r1)
                  : column_chunk(static_cast<const float*>(a.src[j]) + c, a.ld[j], r0, r1);
}
__device__ __forceinline__ void column_final(const ColSum& a, int j, int c) {
    a.dst[j][c] = column_chunk(a.partial + (int64_t)j * kColChunks * a.max_cols + c, a.max_cols, 0, kColChunks);
}
__global__ void __launch_bounds__(128) column_sum_partial_kernel(const __grid_constant__ ColSum a) {
    grid_dependency_wait();
    const int j = blockIdx.z, c = blockIdx.x * 128 + threadIdx.x;
    if (c < a.cols[j]) column_partial(a, j, blockIdx.y, c);
}
__global__ void __launch_bounds__(128) column_sum_final_kernel(const __grid_constant__ ColSum a) {
    grid_dependency_wait();
    const int j = blockIdx.y, c = blockIdx.x * 128 + threadIdx.x;
    if (c < a.cols[j]) column_final(a, j, c);
}
int column_sums(ltca_ctx* ctx, ColSum a, int64_t rows, float* scratch) {
    if (a.n == 0) return LTCA_OK;
    a.rows = rows;
    a.partial = scratch;
    const unsigned bx = (unsigned)((a.max_cols + 127) / 128);
    LTCA_CUDA_OK(ctx, launch_dependent(column_sum_partial_kernel, dim3(bx, kColChunks, a.n), dim3(128), 0, ctx->stream, a));
    LTCA_CUDA_OK(ctx, launch_dependent(column_sum_final_kernel, dim3(bx, a.n), dim3(128), 0, ctx->stream, a));
    return LTCA_OK;
}

// The end of the FlashAttention form's backward: LayerNorm backward, the column sums' first stage and the sums over split products'
// slices need nothing of one another, so they share a launch, and the second stage of all column sums follows.  As launches of
// their own they were five of 3 to 5 us each: backward B16 S200 E256 H4 72.5 -> 70.2, B32 S300 147 -> 137.  dgamma and dbeta are summed where their products are
// formed, a warp its rows, the warps of a block in order, then the blocks: the products are neither written nor read.
// kN4 = E / 128, or 0 for rows of up to 128 columns.
constexpr int kTailThreads = 256, kTailWarps = kTailThreads / 32, kMaxLnChunks = 256, kLnParts = 4;
template <int kN4>
__device__ __forceinline__ void tail_layer_norm(const ColSum& a, float (*sm)[kTailThreads / 32][kN4 > 0 ? 128 * kN4 : 128]) {
    constexpr int kC = kN4 > 0 ? 4 * kN4 : 4;              // columns of a lane
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, E = a.E;
    const int64_t r0 = (int64_t)blockIdx.x * a.ln_rows, r1 = r0 + a.ln_rows < a.rows ? r0 + a.ln_rows : a.rows;
    // element e of this lane: column 4 (lane + 32 (e / 4)) + e % 4 in 16-byte pieces, lane + 32 e otherwise
    auto col = [&](int e) { return kN4 > 0 ? 4 * (lane + 32 * (e / 4)) + e % 4 : lane + 32 * e; };
    auto read = [&](const float* p, float (&v)[kC]) {
        if constexpr (kN4 > 0) {
#pragma unroll
            for (int e = 0; e < kC; e += 4) {
                const float4 x = ldg4(p, lane + 8 * e);
                v[e] = x.x; v[e + 1] = x.y; v[e + 2] = x.z; v[e + 3] = x.w;
            }
        } else {
#pragma unroll
            for (int e = 0; e < kC; ++e) v[e] = col(e) < E ? __ldg(p + col(e)) : 0.f;
        }
    };
    float gm[kC], dg[kC], db[kC];
    read(a.ln_gamma, gm);
#pragma unroll
    for (int e = 0; e < kC; ++e) dg[e] = db[e] = 0.f;
    for (int64_t row = r0 + warp; row < r1; row += kTailWarps) {
        float xh[kC], gv[kC], rs[kC];
        read(a.ln_x + row * E, xh);
        read(a.ln_g + row * E, gv);
#pragma unroll
        for (int e = 0; e < kC; ++e) rs[e] = 0.f;
        if (a.ln_dx && a.ln_res) read(a.ln_res + row * E, rs);
        float s0 = 0.f;
#pragma unroll
        for (int e = 0; e < kC; e += 4) s0 += (xh[e] + xh[e + 1]) + (xh[e + 2] + xh[e + 3]);
        const float mean = warp_total(s0) / E;
        float s1 = 0.f;
#pragma unroll
        for (int e = 0; e < kC; ++e) {
            xh[e] = kN4 > 0 || col(e) < E ? xh[e] - mean : 0.f;
            s1 = fmaf(xh[e], xh[e], s1);
        }
        const float inv_std = rsqrtf(warp_total(s1) / E + a.eps);
        float a1 = 0.f, a2 = 0.f;
#pragma unroll
        for (int e = 0; e < kC; ++e) {
            xh[e] *= inv_std;
            dg[e] = fmaf(gv[e], xh[e], dg[e]);
            db[e] += gv[e];
            gv[e] *= gm[e];
            a1 += gv[e];
            a2 = fmaf(gv[e], xh[e], a2);
        }
        if (!a.ln_dx) continue;
        const float m1 = warp_total(a1) / E, m2 = warp_total(a2) / E;
        float* dx = a.ln_dx + row * E;
#pragma unroll
        for (int e = 0; e < kC; ++e) rs[e] += inv_std * (gv[e] - m1 - xh[e] * m2);
        if constexpr (kN4 > 0) {
#pragma unroll
            for (int e = 0; e < kC; e += 4) reinterpret_cast<float4*>(dx)[lane + 8 * e] = make_float4(rs[e], rs[e + 1], rs[e + 2], rs[e + 3]);
        } else {
#pragma unroll
            for (int e = 0; e < kC; ++e)
                if (col(e) < E) dx[col(e)] = rs[e];
        }
    }
    if (!a.ln_partial) return;
#pragma unroll
    for (int e = 0; e < kC; ++e) {
        sm[0][warp][col(e)] = dg[e];
        sm[1][warp][col(e)] = db[e];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * E; i += kTailThreads) {
        const int k = i / E, c = i - k * E;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < kTailWarps; ++w) v += sm[k][w][c];
        a.ln_partial[((int64_t)blockIdx.x * 2 + k) * E + c] = v;
    }
}
template <int kN4>
__global__ void __launch_bounds__(kTailThreads) module_tail_kernel(const __grid_constant__ ColSum a) {
    grid_dependency_wait();
    extern __shared__ __align__(16) float tail_sm[];
    int block = blockIdx.x;
    if (block < a.ln_blocks) {
        tail_layer_norm<kN4>(a, reinterpret_cast<float (*)[kTailWarps][kN4 > 0 ? 128 * kN4 : 128]>(tail_sm));
        return;
    }
    block -= a.ln_blocks;
    if (block < a.col_blocks) {                        // two runs of 128 columns of a chunk a block, chunks fastest
        const int u = 2 * block + (threadIdx.x >> 7), per_job = kColChunks * ((a.max_cols + 127) / 128);
        const int j = u / per_job, chunk = u % per_job % kColChunks, c = u % per_job / kColChunks * 128 + (threadIdx.x & 127);
        if (j < a.n && c < a.cols[j]) column_partial(a, j, chunk, c);
        return;
    }
    block -= a.col_blocks;                             // a slice sum as gemm_splitk_reduce_kernel has it
    const int per = (int)((a.split_mn + kTailThreads - 1) / kTailThreads);
    const int p = block / per;
    const int64_t i = (int64_t)(block - p * per) * kTailThreads + threadIdx.x;
    if (i >= a.split_mn) return;
    const float* src = a.split + (int64_t)p * a.splits * a.split_mn + i;
    float acc = 0.f;
    for (int s = 0; s < a.splits; s += 4) {
        float v[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = s + e < a.splits ? __ldg(src + (int64_t)(s + e) * a.split_mn) : 0.f;
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (s + e < a.splits) acc += v[e];
    }
    a.split_dst[p][i] = acc;
}
// Second stage: jobs as in column_sum_final_kernel, then dgamma and dbeta (32 columns a block, the blocks' sums in four parts).
__global__ void __launch_bounds__(128) module_tail_final_kernel(const __grid_constant__ ColSum a) {
    grid_dependency_wait();
    const int j = blockIdx.y;
    if (j < a.n) {
        const int c = blockIdx.x * 128 + threadIdx.x;
        if (c < a.cols[j]) column_final(a, j, c);
        return;
    }
    __shared__ float part[kLnParts][32];
    const int k = j - a.n, c = blockIdx.x * 32 + (threadIdx.x & 31), p = threadIdx.x >> 5;
    float* dst = k == 0 ? a.ln_dgamma : a.ln_dbeta;
    if (!dst || blockIdx.x * 32 >= a.E) return;
    const int per = (a.ln_chunks + kLnParts - 1) / kLnParts, c0 = p * per, c1 = min(c0 + per, a.ln_chunks);
    part[p][threadIdx.x & 31] = c < a.E ? column_chunk(a.ln_partial + (int64_t)k * a.E + c, 2 * (int64_t)a.E, c0, c1) : 0.f;
    __syncthreads();
    if (p == 0 && c < a.E) dst[c] = ((part[0][threadIdx.x] + part[1][threadIdx.x]) + part[2][threadIdx.x]) + part[3][threadIdx.x];
}
// Row widths that the tail's LayerNorm takes.
bool tail_width(int E) { return row_pieces(E) > 0 || E <= 128; }
// `scratch` as for column_sums.  Pointers of the LayerNorm have been checked (16 bytes, where row_pieces(E) > 0).
int module_tail(ltca_ctx* ctx, ColSum a, int64_t rows, float* scratch) {
    a.rows = rows;
    a.partial = scratch;
    int64_t per = (rows + kMaxLnChunks - 1) / kMaxLnChunks;
    per = (per + kTailWarps - 1) / kTailWarps * kTailWarps;            // whole rounds of the warps
    a.ln_rows = (int)per;
    a.ln_chunks = a.ln_blocks = (int)((rows + per - 1) / per);
    a.ln_partial = a.ln_dgamma || a.ln_dbeta ? scratch + (int64_t)a.n * kColChunks * a.max_cols : nullptr;
    a.col_blocks = (a.n * kColChunks * ((a.max_cols + 127) / 128) + 1) / 2;
    const int64_t blocks = a.ln_blocks + a.col_blocks + a.split_n * ((a.split_mn + kTailThreads - 1) / kTailThreads);
    auto kern = module_tail_kernel<0>;
    switch (row_pieces(a.E)) {
        case 1: kern = module_tail_kernel<1>; break;
        case 2: kern = module_tail_kernel<2>; break;
        case 3: kern = module_tail_kernel<3>; break;
        case 4: kern = module_tail_kernel<4>; break;
        case 5: kern = module_tail_kernel<5>; break;
        case 6: kern = module_tail_kernel<6>; break;
        case 7: kern = module_tail_kernel<7>; break;
        case 8: kern = module_tail_kernel<8>; break;
    }
    const size_t smem = (size_t)2 * kTailWarps * (a.E < 128 ? 128 : a.E) * sizeof(float);
    static SmemOptIn once[9];
    if (smem > 48 * 1024) LTCA_CUDA_OK(ctx, opt_in_dynamic_smem(once[row_pieces(a.E)], ctx->device, kern, (int)smem));
    LTCA_CUDA_OK(ctx, launch_dependent(kern, dim3((unsigned)blocks), dim3(kTailThreads), smem, ctx->stream, a));
    const int ln_jobs = a.ln_partial ? 2 : 0;
    if (a.n + ln_jobs == 0) return LTCA_OK;
    const unsigned bx = (unsigned)((a.max_cols + 127) / 128), lx = ln_jobs ? (unsigned)((a.E + 31) / 32) : 0;
    LTCA_CUDA_OK(ctx, launch_dependent(module_tail_final_kernel, dim3(bx > lx ? bx : lx, a.n + ln_jobs), dim3(128), 0, ctx->stream, a));
    return LTCA_OK;
}
// Four jobs' chunks and the LayerNorm's, or six jobs' chunks.
size_t colsum_scratch_bytes(const ltca_tsa_params* t) {
    const int hw = t->H * t->head_width;
    return align_up((size_t)((kMaxColJobs - 2) * kColChunks + 2 * kMaxLnChunks) * (hw > t->E ? hw : t->E) * sizeof(float), 256);
}

// `xo` receives LayerNorm(x) (or x), `go` the gradient behind the dropout (null outputs: no such part); w: matrices to
// round; mask: words to write (null: no such part).
int prenorm_prepare(ltca_ctx* ctx, const ltca_tsa_params* t, const RowOut& xo, const RowOut* go, const CvtMany* w,
                    const MaskArgs* mask = nullptr) {
    PrepareArgs a;
    memset(&a, 0, sizeof(a));
    a.x = t->x; a.gamma = t->ln_gamma; a.beta = t->ln_beta;
    a.xo = xo;
    a.rows = (int64_t)t->B * t->S;
    a.E = t->E;
    a.use_ln = t->use_layer_norm;
    a.eps = 1e-5f;
    if (!t->use_layer_norm) a.gamma = a.beta = nullptr;
    if (xo.f32 || xo.bf16) a.row_blocks = (int)((a.rows + kPrepareThreads / 32 - 1) / (kPrepareThreads / 32));
    const int sms = ctx->sm_count > 0 ? ctx->sm_count : kPlanSms;
    if (go && (go->f32 || go->bf16)) {
        a.dy = t->dy;
        a.go = *go;
        a.p = t->dropout_prob;
        a.seed = t->dropout_seed;
        const int64_t blocks = (a.rows * a.E + 4 * kPrepareThreads - 1) / (4 * kPrepareThreads);
        a.dy_blocks = (int)(blocks < 8 * sms ? blocks : 8 * sms);
    }
    int w_blocks = 0;
    if (w && w->n) {
        a.w = *w;
        const uint32_t blocks = (w->start4[w->n] + 2 * kPrepareThreads - 1) / (2 * kPrepareThreads);
        w_blocks = blocks < 4u * sms ? (int)blocks : 4 * sms;
    }
    if (mask) {
        a.mask = *mask;
        a.B = t->B;
        const int64_t blocks = ((int64_t)t->B * mask->nq * mask->nk + kPrepareThreads / 32 - 1) / (kPrepareThreads / 32);
        a.mask_blocks = (int)(blocks < 8 * sms ? blocks : 8 * sms);
    }
    const int blocks = a.mask_blocks + a.row_blocks + a.dy_blocks + w_blocks;
    if (blocks == 0) return LTCA_OK;
    LTCA_CUDA_OK(ctx, launch_dependent(prenorm_prepare_kernel, dim3((unsigned)blocks),
                                       dim3(kPrepareThreads), 0, ctx->stream, a));
    return LTCA_OK;
}
int prenorm_finish(ltca_ctx* ctx, const ltca_tsa_params* t, const float* y) {
    const int64_t n = (int64_t)t->B * t->S * t->E, blocks = (n + 511) / 512;
    LTCA_CUDA_OK(ctx, launch_dependent(residual_dropout_kernel, dim3((unsigned)(blocks < 2368 ? blocks : 2368)), dim3(256), 0, ctx->stream,
                                       y, t->x, t->out, n, t->use_residual, t->dropout_prob, t->dropout_seed));
    return LTCA_OK;
}

struct Plan {
    int64_t rows;
    int HW;
    size_t buf;          // bytes of one [rows, HW] fp32 buffer
    size_t lse;          // bytes of lse
    size_t y;            // bytes of one [rows, E] buffer
    size_t attn_fwd, attn_bwd;
};
// Whether a call's workspace has the room that ltca_tsa_workspace_bytes asks for, or lacks the exact backward's shares of dQ.
enum Room { kLeastRoom, kFullRoom };

void fill_attn(const ltca_tsa_params* t, ltca_attn_params* a) {
    memset(a, 0, sizeof(*a));
    const int HW = t->H * t->head_width;
    a->B = t->B; a->H = t->H; a->Sq = t->S; a->Sk = t->S; a->D = t->head_width;
    a->dtype = LTCA_F32;
    a->mode = t->mode == LTCA_MODE_SPLIT ? LTCA_MODE_AUTO : t->mode;     // the module has no split mode of its own
    a->causal = t->causal;
    a->scale = t->scale;
    a->score_clamp = t->score_clamp;
    ltca_strides st;
    st.head = t->head_width;
    if (t->time_major) { st.batch = HW; st.seq = (int64_t)t->B * HW; }
    else               { st.batch = (int64_t)t->S * HW; st.seq = HW; }
    a->q_strides = a->k_strides = a->v_strides = a->o_strides = st;
    a->do_strides = a->dq_strides = a->dk_strides = a->dv_strides = st;
    a->keep_mask = t->keep_mask;
    a->kv_len = t->kv_len;
    // the module's gradients stay bit-identical from run to run (the reference's tests pin backward
    // repeatability on the module, src/ml/time_self_attention_test.cu:799-838)
    a->bwd_deterministic = 1;
}

int make_plan(const ltca_tsa_params* t, Plan* pl, Room room = kFullRoom) {
    pl->rows = (int64_t)t->B * t->S;
    pl->HW = t->H * t->head_width;
    pl->buf = align_up((size_t)pl->rows * pl->HW * sizeof(float), 256);
    pl->lse = align_up((size_t)t->B * t->H * t->S * sizeof(float), 256);
    pl->y = align_up((size_t)pl->rows * t->E * sizeof(float), 256);
    ltca_attn_params a;
    fill_attn(t, &a);
    // pointers only need to be non-null for the size queries
    int rc = ltca_attn_workspace_bytes(&a, 0, &pl->attn_fwd);
    if (rc) return rc;
    if (room == kLeastRoom && attn_bwd_exact(&a)) {
        pl->attn_bwd = attn_bwd_fp32_workspace(&a, false);
        return LTCA_OK;
    }
    return ltca_attn_workspace_bytes(&a, 1, &pl->attn_bwd);
}

int check(ltca_ctx* ctx, const ltca_tsa_params* t) {
    if (!ctx) return LTCA_ERR_INVALID;
    if (!t) return fail(ctx, LTCA_ERR_INVALID, "null parameter block");
    if (t->B < 1 || t->S < 1 || t->E < 1 || t->H < 1 || t->head_width < 1)
        return fail(ctx, LTCA_ERR_INVALID, "B, S, E, H, head_width must be positive");
    // same validation as the reference constructor (src/ml/time_self_attention.cu:25-35)
    if (t->E % t->H != 0)
        return fail(ctx, LTCA_ERR_INVALID, "input_dim (%d) must be divisible by num_heads (%d)",
                    t->E, t->H);
    if (!t->x || !t->wq || !t->wk || !t->wv || !t->wo)
        return fail(ctx, LTCA_ERR_INVALID, "x and the four weight matrices must be non-null");
    if (!(t->scale > 0.f)) return fail(ctx, LTCA_ERR_INVALID, "scale must be positive");
    if (reinterpret_cast<uintptr_t>(t->workspace) & 255)
        return fail(ctx, LTCA_ERR_INVALID, "workspace must be 256-byte aligned");
    if (t->reuse_forward && !t->saved)
        return fail(ctx, LTCA_ERR_INVALID, "reuse_forward needs the saved block of the forward call");
    if (t->saved) {
        if (t->pre_norm)
            return fail(ctx, LTCA_ERR_UNSUPPORTED, "the saved block is not available in the pre_norm form");
        if (reinterpret_cast<uintptr_t>(t->saved) & 255)
            return fail(ctx, LTCA_ERR_INVALID, "saved must be 256-byte aligned");
        size_t need = 0;
        int rc = ltca_tsa_saved_bytes(t, &need);
        if (rc) return fail(ctx, rc, "bad shape for the saved block");
        if (t->saved_bytes < need)
            return fail(ctx, LTCA_ERR_WORKSPACE, "the saved block needs %zu bytes", need);
    }
    if (t->weight_cache) {
        if (reinterpret_cast<uintptr_t>(t->weight_cache) & 255)
            return fail(ctx, LTCA_ERR_INVALID, "weight_cache must be 256-byte aligned");
        size_t need = 0;
        int rc = ltca_tsa_weight_cache_bytes(t, &need);
        if (rc) return fail(ctx, rc, "bad shape for the weight cache");
        if (t->weight_cache_bytes < need)
            return fail(ctx, LTCA_ERR_WORKSPACE, "the weight cache needs %zu bytes", need);
    }
    return LTCA_OK;
}

// Projections + attention forward into workspace; returns pointers into it.
struct FwdBufs { float *q, *k, *v, *ctx, *lse; char* rest; };

// With a caller-kept `saved` block (ltca_tsa_params.saved) q, k, v, ctx and lse live there and the
// workspace only holds the attention scratch; with reuse_forward they are taken as they are.
int forward_core(ltca_ctx* ctx, const ltca_tsa_params* t, const Plan& pl, char* w, FwdBufs* fb,
                 size_t attn_ws_bytes) {
    char* rest = w;
    if (t->saved) w = reinterpret_cast<char*>(t->saved);
    fb->q = reinterpret_cast<float*>(w);   w += pl.buf;
    fb->k = reinterpret_cast<float*>(w);   w += pl.buf;
    fb->v = reinterpret_cast<float*>(w);   w += pl.buf;
    fb->ctx = reinterpret_cast<float*>(w); w += pl.buf;
    fb->lse = reinterpret_cast<float*>(w); w += pl.lse;
    fb->rest = t->saved ? rest : w;
    if (t->saved && t->reuse_forward) return LTCA_OK;
    const int rows = (int)pl.rows, E = t->E, HW = pl.HW;
    int rc;
    const Gemm32Problem qkv[3] = {{t->x, t->wq, t->bq, fb->q, rows, HW, E, E, HW, HW},
                                  {t->x, t->wk, t->bk, fb->k, rows, HW, E, E, HW, HW},
                                  {t->x, t->wv, t->bv, fb->v, rows, HW, E, E, HW, HW}};
    if ((rc = gemm_fp32(ctx, qkv, 3, 0, 0, false, false))) return rc;
    ltca_attn_params a;
    fill_attn(t, &a);
    a.q = fb->q; a.k = fb->k; a.v = fb->v; a.o = fb->ctx; a.lse = fb->lse;
    a.workspace = attn_ws_bytes ? fb->rest : nullptr;
    a.workspace_bytes = attn_ws_bytes;
    rc = ltca_attn_fwd(ctx, &a);
    return rc;
}

// ---- tensor-pipe pipeline ---------------------------------------------------------------------

void fill_attn_bf16(const ltca_tsa_params* t, ltca_attn_params* a) {
    fill_attn(t, a);
    a->dtype = LTCA_BF16;
    a->mode = LTCA_MODE_BF16;
}

// A forward that leaves something for the backward (its intermediates, or the weights' copies) takes the pipeline
// the backward will take, so that both calls agree on what the blocks hold.
bool keeps_for_backward(const ltca_tsa_params* t) { return t->saved != nullptr || t->weight_cache != nullptr; }

// Whether the attention core of the tensor pipeline is the materialised-score path (attn_wide_sm100.cu): head
// widths the streaming kernels do not cover.  Taken for heads wider than 128 (the reference's configuration gives
// every head the model's width) and, on explicit request (LTCA_MODE_BF16), for any width that is a multiple of 8;
// narrow heads under LTCA_MODE_AUTO stay on the exact pipeline, whose handful of small kernels is faster there.
bool use_wide(const ltca_tsa_params* t, bool /*backward*/) {
    if (t->mode == LTCA_MODE_FP32) return false;
    if (t->head_width < 8 || (t->head_width % 8)) return false;
    ltca_attn_params a;
    fill_attn_bf16(t, &a);
    // one choice for forward and backward calls, so that a forward call computes what the backward recomputes
    // (width 128 has a streaming forward but no streaming backward: it takes this path for both)
    if (attn_fwd_sm100_supported(&a) && attn_bwd_sm100_supported(&a)) return false;
    return t->mode == LTCA_MODE_BF16 || t->head_width > 128;
}

// Whether the module runs on the tensor pipe: the caller allows it, an attention path on the tensor pipe covers
// the head width, and the bf16 rows keep the 16-byte pitch TMA needs.
bool use_tensor(const ltca_tsa_params* t, bool backward) {
    if (t->mode == LTCA_MODE_FP32) return false;
    if ((t->H * t->head_width) % 8) return false;
    if (use_wide(t, backward)) return true;
    ltca_attn_params a;
    fill_attn_bf16(t, &a);
    if (!attn_fwd_sm100_supported(&a)) return false;
    if (backward && !attn_bwd_sm100_supported(&a)) return false;
    return true;
}

// Whether the written-out-score path runs on per-head products of the weights: heads as wide as the model (the reference's
// form) and enough rows.  With M_h = Wq_h Wk_h^T and N_h = Wv_h Wo_h, both [E, E],
//   scores   q_h k_h^T = (x M_h) x^T            output   sum_h P_h v_h Wo_h = sum_h P_h (x N_h)
// so k, ctx and the output projection are never formed, and in the backward, with dS and dP as before,
//   dP_h = dy z_h^T, dz_h = P_h^T dy, dT_h = dS_h x        (T_h = x M_h, z_h = x N_h)
//   dx = sum_h dT_h M_h^T + dz_h N_h^T + dS_h^T T_h        dM_h = x^T dT_h, dN_h = x^T dz_h
//   dWq_h = dM_h Wk_h, dWk_h = dM_h^T Wq_h, dWv_h = dN_h Wo_h^T, dWo_h = Wv_h^T dN_h.
// In units of rows x E x (H E) multiply-adds the projections cost 4 instead of 8 forward (T counts three, its operands have two
// terms) and 4 instead of 8 backward; products of weights add 6 and 10 in units of E x E x (H E), and three launches.  From
// four rows per column of x on that is the faster path: forward and backward of a kept forward, us, B32 S256 E512 H8 365 + 407
// -> 271 + 307; at the line, B8 S256 E512 H8 155 + 183 -> 125 + 159, B32 S32 E256 H4 65 + 82 -> 60 + 79; half as many rows
// gained nothing (B4 S256 E512 H8).  Fewer bf16 roundings lie between the inputs and a result than on the other path, and the
// products of weights have two terms, as q and k have there: errors against 64 bits 4.0e-3 -> 3.2e-3 (output), 5.7e-3 ->
// 4.8e-3 (dx), 5.8e-3 -> 5.2e-3 (dWq, dWk), 4.0e-3 -> 3.6e-3 (dWv, dWo), the like at every size.
constexpr int kComposedRows = 4;
// Kept weights serve calls of any number of rows, so a weight cache has what either path needs from E and the mode alone.  Heads of up
// to 128, which come here on explicit request, keep the block of their q, k, v and ctx (B16 S256 E128 H2 step 112 us, on products
// of the weights 102: the block would have to grow for it).
bool composed_weights(const ltca_tsa_params* t) { return t->head_width == t->E && t->head_width > 128 && use_wide(t, false); }
bool composed_shape(const ltca_tsa_params* t) {
    return composed_weights(t) && (int64_t)t->B * t->S >= (int64_t)kComposedRows * t->E;
}
bool use_composed(const ltca_tsa_params* t) { return composed_shape(t) && !t->bq && !t->bk && !t->bv; }
// Where a call's biases decide between the two paths, a kept forward has either form.  Its block's first word says which: the
// backward that reuses it need not be given the biases, for which it has no use.
enum KeptForm : uint32_t { kKeptProjections = 1, kKeptComposed = 2 };
size_t kept_word_bytes(const ltca_tsa_params* t) { return composed_shape(t) ? 256 : 0; }
char* kept_block(const ltca_tsa_params* t) { return reinterpret_cast<char*>(t->saved) + kept_word_bytes(t); }

struct TPlan {
    int64_t rows;
    int HW, Ep;
    size_t xb, w_in, w_out, act, lse, y;
    size_t attn_fwd, attn_bwd, partial;
    int ks_in, ks_out, n_dw;
    // materialised-score path: low-order parts of x, Wq, Wk, q, k; fp32 projection scratch; score matrices
    bool wide;
    size_t mat32, mat16;
    // ... on products of the weights: one [E, H * E] matrix in bf16
    bool composed;
    size_t me;
    int ks_m;
};

int make_tplan_as(const ltca_tsa_params* t, TPlan* pl, bool backward, bool composed) {
    pl->rows = (int64_t)t->B * t->S;
    pl->HW = t->H * t->head_width;
    pl->Ep = (t->E + 7) / 8 * 8;
    pl->xb = align_up((size_t)pl->rows * pl->Ep * 2, 256);
    pl->w_in = align_up((size_t)t->E * pl->HW * 2, 256);
    pl->w_out = align_up((size_t)pl->HW * pl->Ep * 2, 256);
    pl->act = align_up((size_t)pl->rows * pl->HW * 2, 256);
    pl->lse = align_up((size_t)t->B * t->H * t->S * sizeof(float), 256);
    pl->y = align_up((size_t)pl->rows * t->E * sizeof(float), 256);
    pl->wide = use_wide(t, backward);
    pl->composed = pl->wide && composed;
    pl->me = align_up((size_t)t->E * t->H * t->E * 2, 256);
    pl->mat32 = pl->mat16 = 0;
    pl->attn_fwd = pl->attn_bwd = 0;
    int rc;
    if (pl->wide) {
        const size_t elems = wide_matrix_elems(t->B, t->H, t->S, t->S);
        pl->mat32 = align_up(elems * sizeof(float), 256);
        pl->mat16 = align_up(elems * 2, 256);
    } else {
        ltca_attn_params a;
        fill_attn_bf16(t, &a);
        if ((rc = ltca_attn_workspace_bytes(&a, 0, &pl->attn_fwd))) return rc;
        if ((rc = ltca_attn_workspace_bytes(&a, 1, &pl->attn_bwd))) return rc;
    }
    const int rows = (int)pl->rows;
    // dWq, dWk, dWv are one launch, and dWo with them where it has their shape: 64 pairs of CTAs with work instead of 48 and
    // then 64 with a quarter of it (32768 x 512 x 512: 51 + 21 us and two reductions of 4 and 5, so 55 and one of 4)
    pl->n_dw = t->E == pl->HW ? 4 : 3;
    pl->ks_in = gemm_sm100_pick_ksplit(t->E, pl->HW, rows, pl->n_dw, kPlanSms);
    pl->ks_out = gemm_sm100_pick_ksplit(pl->HW, t->E, rows, 1, kPlanSms);
    const size_t p_in = gemm_sm100_partial_bytes(t->E, pl->HW, pl->n_dw, pl->ks_in);
    const size_t p_out = gemm_sm100_partial_bytes(pl->HW, t->E, 1, pl->ks_out);
    pl->partial = p_in > p_out ? p_in : p_out;
    pl->ks_m = 1;
    if (pl->composed) {
        pl->ks_m = gemm_sm100_pick_ksplit(t->E, pl->HW, rows, 2, kPlanSms);
        pl->partial = gemm_sm100_partial_bytes(t->E, pl->HW, 2, pl->ks_m);
    }
    return LTCA_OK;
}
int make_tplan(const ltca_tsa_params* t, TPlan* pl, bool backward) { return make_tplan_as(t, pl, backward, use_composed(t)); }

// A size is asked for before the biases are known: the larger one of a plan with and one without them.
template <typename Size>
int planned_bytes(const ltca_tsa_params* t, bool backward, Size size, size_t* bytes_out) {
    TPlan pl;
    int rc = make_tplan_as(t, &pl, backward, false);
    if (rc) return rc;
    *bytes_out = size(pl);
    if (!composed_shape(t)) return LTCA_OK;
    if ((rc = make_tplan_as(t, &pl, backward, true))) return rc;
    if (size(pl) > *bytes_out) *bytes_out = size(pl);
    return LTCA_OK;
}

// Extra scratch of the materialised-score path: x_lo, Wq_lo, Wk_lo, q_lo, k_lo, the fp32 projection result that is
// split into q (then k), the raw scores and the probabilities; the backward adds dP.
// What of it a forward keeps for the backward: the low-order parts, the raw scores and the probabilities.
size_t wide_kept(const TPlan& pl) { return pl.wide ? pl.xb + 2 * pl.w_in + 2 * pl.act + pl.mat32 + pl.mat16 : 0; }
size_t wide_extra(const TPlan& pl, int which) {
    if (!pl.wide) return 0;
    return wide_kept(pl) + (which == 0 ? 0 : pl.mat32 + pl.mat16);     // backward: dP and dS
}

// On products of the weights: what a forward keeps (x, the weights with the second terms of Wq and Wk, M, N, T, z, lse, scores,
// probabilities) and what no later call needs (the other second terms).
size_t composed_kept(const TPlan& pl) { return pl.xb + 5 * pl.w_in + pl.w_out + 2 * pl.me + 2 * pl.act + pl.lse + pl.mat32 + pl.mat16; }
size_t composed_scratch(const TPlan& pl) { return pl.xb + pl.w_in + pl.w_out + pl.me + pl.act; }

size_t tensor_workspace(const TPlan& pl, int which) {
    if (pl.composed) {
        const size_t n = composed_kept(pl) + composed_scratch(pl);
        if (which == 0) return n + pl.y;
        // dy; dT, dz and two more for bias gradients; dP, dS; dM and dN in fp32 and in two terms each
        return n + pl.xb + 4 * pl.act + pl.mat32 + pl.mat16 + 4 * pl.me + 4 * pl.me + pl.partial;
    }
    // x, the four weight matrices, q, k, v, ctx, lse
    size_t n = pl.xb + 3 * pl.w_in + pl.w_out + 4 * pl.act + pl.lse + wide_extra(pl, which);
    if (which == 0) return n + pl.y + pl.attn_fwd;
    n += pl.xb + 4 * pl.act;                       // dy, dctx, dq, dk, dv
    n += pl.attn_fwd > pl.attn_bwd ? pl.attn_fwd : pl.attn_bwd;
    return n + pl.partial;
}

size_t tensor_saved_bytes(const TPlan& pl) {
    if (pl.composed) return composed_kept(pl);
    return pl.xb + 3 * pl.w_in + pl.w_out + 4 * pl.act + pl.lse + wide_kept(pl);
}

struct TBufs {
    void *xb, *wq, *wk, *wv, *wo, *q, *k, *v, *ctx;
    float* lse;
    char* rest;
    // materialised-score path
    void *xl, *wql, *wkl, *ql, *kl, *P;
    float* scores;
    // ... on products of the weights
    void *wvl, *wol, *m, *ml, *n, *t, *tl, *z;
};

// What both forms of the module on the written-out-score path have alike comes first.
char* place_scores(const TPlan& pl, char* w, TBufs* tb) {
    tb->lse = reinterpret_cast<float*>(w);    w += pl.lse;
    tb->scores = reinterpret_cast<float*>(w); w += pl.mat32;
    tb->P = w;                                w += pl.mat16;
    return w;
}

// The attention problem of the module for the materialised-score path (bf16 views of the projection outputs).
void fill_wide(const ltca_tsa_params* t, const TBufs& tb, WideArgs* w) {
    ltca_attn_params a;
    fill_attn_bf16(t, &a);
    w->B = t->B; w->H = t->H; w->Sq = t->S; w->Sk = t->S; w->D = t->head_width;
    w->causal = t->causal; w->scale = t->scale; w->clamp = t->score_clamp;
    w->keep_mask = t->keep_mask; w->kv_len = t->kv_len;
    w->qh = tb.q; w->ql = tb.ql; w->kh = tb.k; w->kl = tb.kl; w->v = tb.v;
    w->qs = w->ks = w->vs = w->os = a.q_strides;
    w->dos = w->dqs = w->dks = w->dvs = a.q_strides;
    w->o = tb.ctx; w->o_bf16 = 1; w->lse = tb.lse;
    w->scores = tb.scores; w->P = tb.P;
    w->grads_bf16 = 1;
    if (t->saved && kept_word_bytes(t)) {
        w->mark = reinterpret_cast<uint32_t*>(t->saved);
        w->mark_value = kKeptProjections;
    }
}

// The same on products of the weights: T and z in the places of q and v, x in that of k, for every head.
ltca_strides x_strides(const ltca_tsa_params* t, int64_t ld) {
    ltca_strides st;
    st.head = 0;
    st.batch = t->time_major ? ld : (int64_t)t->S * ld;
    st.seq = t->time_major ? (int64_t)t->B * ld : ld;
    return st;
}
void fill_composed(const ltca_tsa_params* t, const TPlan& pl, const TBufs& tb, WideArgs* w) {
    fill_wide(t, tb, w);
    w->qh = tb.t; w->ql = tb.tl;
    w->kh = tb.xb; w->kl = tb.xl; w->ks = x_strides(t, pl.Ep);
    w->v = tb.z;
    w->o = nullptr;
    w->mark_value = kKeptComposed;
}

// The attention scratch (TBufs::rest) of a call whose buffers start at w; not on the written-out-score path.
char* scratch_of(const ltca_tsa_params* t, const TPlan& pl, char* w) { return t->saved ? w : w + tensor_saved_bytes(pl); }

int workspace_bytes(const ltca_tsa_params* t, int which, Room room, size_t* bytes_out);
// The call as its workspace is laid out.  Packed mask words and the exact backward's shares of dQ are part of what
// ltca_tsa_workspace_bytes asks for, but a workspace that was sized without the mask is laid out without the words (the attention
// kernels then read the dense values), and one that has no room for the shares without those.
struct Layout {
    ltca_tsa_params t;
    Room room;
    size_t need;                   // what it takes: more than there is where no layout fits
    int rc;
};
Layout lay_out(const ltca_tsa_params* t, int which) {
    Layout l{*t, kFullRoom, 0, LTCA_OK};
    for (Room room : {kFullRoom, kLeastRoom}) {
        l.room = room;
        for (int masked = t->keep_mask ? 1 : 0; masked >= 0; --masked) {
            l.t.keep_mask = masked ? t->keep_mask : nullptr;
            l.rc = workspace_bytes(&l.t, which, room, &l.need);
            if (!l.rc && t->workspace_bytes >= l.need) return l;
        }
    }
    return l;
}
ltca_tsa_params laid_out(const ltca_tsa_params* t, int which) { return t->keep_mask ? lay_out(t, which).t : *t; }

// What a module call tells its kernels through the context, taken back when the call returns.
struct CallHints {
    ltca_ctx* ctx;
    ~CallHints() { ctx->mask_packed = nullptr; ctx->mask_words = nullptr; ctx->fwd_pairs = false; ctx->run_if = RunIf(); }
};
// The packed form of the call's dense mask lies in the last bytes of the `bytes` of scratch that its attention kernels
// share; `later`: the call's prepare launch writes it (prenorm_prepare), else it is written now.
int place_mask_words(ltca_ctx* ctx, const ltca_tsa_params* t, const TPlan& pl, char* scratch, size_t bytes, bool later) {
    if (!t->keep_mask || pl.wide) return LTCA_OK;
    ltca_attn_params a;
    fill_attn_bf16(t, &a);
    const size_t need = mask_words_bytes(&a);
    if (bytes < need) return LTCA_OK;
    void* words = scratch + (bytes - need);
    int rc;
    if (!later && (rc = pack_mask_words(ctx, &a, words))) return rc;
    ctx->mask_packed = t->keep_mask;
    ctx->mask_words = words;
    return LTCA_OK;
}

// The steps of tensor_forward_core on products of the weights, up to z and the probabilities.  (No FlashAttention form runs
// its first steps in here: fuses_prenorm.)
int composed_forward_core(ltca_ctx* ctx, const ltca_tsa_params* t, const TPlan& pl, char* w, TBufs* tb, const float* also_src,
                          void* also_dst, bool* also_done) {
    char* r = w;
    if (t->saved) w = kept_block(t);
    w = place_scores(pl, w, tb);
    tb->xb = w;  w += pl.xb;
    tb->wq = w;  w += pl.w_in;
    tb->wk = w;  w += pl.w_in;
    tb->wv = w;  w += pl.w_in;
    tb->wo = w;  w += pl.w_out;
    tb->wql = w; w += pl.w_in;
    tb->wkl = w; w += pl.w_in;
    tb->m = w;   w += pl.me;
    tb->n = w;   w += pl.me;
    tb->t = w;   w += pl.act;
    tb->z = w;   w += pl.act;
    if (!t->saved) r = w;
    tb->xl = r;  r += pl.xb;
    tb->wvl = r; r += pl.w_in;
    tb->wol = r; r += pl.w_out;
    tb->ml = r;  r += pl.me;
    tb->tl = r;  r += pl.act;
    tb->rest = r;
    tb->q = tb->k = tb->v = tb->ctx = tb->ql = tb->kl = nullptr;
    const bool cached = t->weight_cache != nullptr;
    if (cached) {                                      // laid out as on the other path
        char* c = reinterpret_cast<char*>(t->weight_cache);
        tb->wq = c;  c += pl.w_in;
        tb->wk = c;  c += pl.w_in;
        tb->wv = c;  c += pl.w_in;
        tb->wo = c;  c += pl.w_out;
        tb->wql = c; c += pl.w_in;
        tb->wkl = c; c += pl.w_in;
        tb->wvl = c; c += pl.w_in;
        tb->wol = c;
    }
    if (t->saved && t->reuse_forward) return LTCA_OK;
    const int E = t->E, HW = pl.HW, Ep = pl.Ep, rows = (int)pl.rows;
    int rc;
    {
        const float* src[6] = {t->x, t->wq, t->wk, t->wv, t->wo, nullptr};
        void* dst[6] = {tb->xb, tb->wq, tb->wk, tb->wv, tb->wo, nullptr};
        void* lo[6] = {tb->xl, tb->wql, tb->wkl, tb->wvl, tb->wol, nullptr};
        int64_t ld_src[6] = {E, HW, HW, HW, E, E}, ld_dst[6] = {Ep, HW, HW, HW, Ep, Ep};
        int64_t nrows[6] = {pl.rows, E, E, E, HW, pl.rows};
        int ncols[6] = {E, HW, HW, HW, E, E};
        int n = cached && t->weight_cache_valid ? 1 : 5;
        if (also_src) {
            src[n] = also_src; dst[n] = also_dst; lo[n] = nullptr;
            ld_src[n] = E; ld_dst[n] = Ep; nrows[n] = pl.rows; ncols[n] = E;
            ++n;
            *also_done = true;
        }
        if ((rc = convert_many_bf16(ctx, n, src, ld_src, dst, ld_dst, nrows, ncols, lo))) return rc;
    }
    {   // M_h = Wq_h Wk_h^T : both stored [E, HW], the head's columns contiguous; N_h = Wv_h Wo_h : Wo_h is rows [h E, (h + 1) E)
        GemmGroup gg;
        gg.heads = t->H; gg.n = 2; gg.out_bf16 = 1;
        GemmGroup::Member &m = gg.m[0], &n = gg.m[1];
        m.M = m.N = m.K = n.M = n.N = n.K = E;
        m.terms = n.terms = 3;
        m.a[0] = GemmOperand{tb->wq, HW, 0};  m.b[0] = GemmOperand{tb->wk, HW, 0};
        m.a[1] = GemmOperand{tb->wq, HW, 0};  m.b[1] = GemmOperand{tb->wkl, HW, 0};
        m.a[2] = GemmOperand{tb->wql, HW, 0}; m.b[2] = GemmOperand{tb->wk, HW, 0};
        m.a_hs = m.b_hs = E;
        m.c = tb->m; m.c_lo = tb->ml;
        n.a[0] = GemmOperand{tb->wv, HW, 0};  n.b[0] = GemmOperand{tb->wo, Ep, 1};
        n.a[1] = GemmOperand{tb->wv, HW, 0};  n.b[1] = GemmOperand{tb->wol, Ep, 1};
        n.a[2] = GemmOperand{tb->wvl, HW, 0}; n.b[2] = GemmOperand{tb->wo, Ep, 1};
        n.a_hs = E; n.b_hs = (int64_t)E * Ep;
        n.c = tb->n;
        m.ldc = n.ldc = HW;
        m.c_hs = n.c_hs = E;
        if ((rc = gemm_sm100_group(ctx, gg))) return rc;
    }
    {   // T = x M, in two terms
        GemmProblem gp;
        gp.M = rows; gp.N = HW; gp.K = E;
        gp.n_sum = 3;
        gp.a[0] = GemmOperand{tb->xb, Ep, 0}; gp.b[0] = GemmOperand{tb->m, HW, 1};
        gp.a[1] = GemmOperand{tb->xb, Ep, 0}; gp.b[1] = GemmOperand{tb->ml, HW, 1};
        gp.a[2] = GemmOperand{tb->xl, Ep, 0}; gp.b[2] = GemmOperand{tb->m, HW, 1};
        gp.c[0] = tb->t; gp.c_lo = tb->tl;
        gp.out_bf16 = 1;
        gp.ldc = HW;
        if ((rc = gemm_sm100(ctx, gp))) return rc;
    }
    {   // z = x N
        GemmProblem gp;
        gp.M = rows; gp.N = HW; gp.K = E;
        gp.a[0] = GemmOperand{tb->xb, Ep, 0}; gp.b[0] = GemmOperand{tb->n, HW, 1};
        gp.c[0] = tb->z;
        gp.out_bf16 = 1;
        gp.ldc = HW;
        if ((rc = gemm_sm100(ctx, gp))) return rc;
    }
    WideArgs wa;
    fill_composed(t, pl, *tb, &wa);
    return wide_attn_fwd(ctx, wa);
}

// C_b = sum over the heads of op(S_hb) R_hb for one [S, E] matrix of rows per sequence: S_hb a score-shaped matrix (mn_major:
// taken transposed), R the activations [rows, H E]; `add`: to what C holds.
int sum_over_heads(ltca_ctx* ctx, const ltca_tsa_params* t, const TPlan& pl, const void* score, int mn_major, const void* act,
                   float* c, const float* bias, bool add) {
    ltca_attn_params a;
    fill_attn_bf16(t, &a);
    const ltca_strides cs = x_strides(t, t->E);
    const int Skp = wide_padded_keys(t->S);
    GemmProblem gp;
    gp.M = t->S; gp.N = t->E; gp.K = t->S;
    gp.a[0] = GemmOperand{score, Skp, mn_major};
    gp.b[0] = GemmOperand{act, a.q_strides.seq, 1};
    gp.sum_h = t->H; gp.batch_b = t->B;
    gp.a_bs[0] = (int64_t)t->S * Skp;   gp.a_bs[1] = (int64_t)t->H * t->S * Skp;
    gp.b_bs[0] = a.q_strides.head;      gp.b_bs[1] = a.q_strides.batch;
    gp.c_bs[1] = cs.batch;
    gp.c[0] = c;
    gp.ldc = cs.seq;
    gp.bias[0] = bias;
    gp.add_to_c = add ? 1 : 0;
    return gemm_sm100(ctx, gp);
}

// What a backward of either form works on first: dy in bf16, four activations, and on the written-out-score path dP and dS (not in
// P's place: the probabilities stay valid for the next backward from the same forward).
struct BwdBufs { void *dyb, *dctx, *dq, *dk, *dv; float* dP; void* dS; };
// A backward's two parts lie before and behind the step from dP to dS, which is the same in both forms.
enum BwdPart { kUpToScores = 1, kFromScores = 2, kWhole = 3 };

// A product for every head between two of [E, H E] / [rows, H E] / [HW, E] matrices: C_h[M, N] = sum over the terms.
int per_head(ltca_ctx* ctx, const ltca_tsa_params* t, int M, int n_sum, const GemmOperand* a, int64_t a_hs, const GemmOperand* b,
             int64_t b_hs, void* c, int64_t ldc, int64_t c_hs, int out_bf16) {
    GemmProblem gp;
    gp.M = M; gp.N = t->E; gp.K = t->E;
    gp.n_sum = n_sum;
    for (int i = 0; i < n_sum; ++i) { gp.a[i] = a[i]; gp.b[i] = b[i]; }
    gp.batch_h = t->H;
    gp.a_bs[0] = a_hs; gp.b_bs[0] = b_hs; gp.c_bs[0] = c_hs;
    gp.c[0] = c;
    gp.ldc = ldc;
    gp.out_bf16 = out_bf16;
    return gemm_sm100(ctx, gp);
}

// tensor_backward on products of the weights; arguments as projected_backward has them.
int composed_backward(ltca_ctx* ctx, const ltca_tsa_params* t, const TPlan& pl, const BwdBufs& g, char* w, BwdPart part, bool want_dx,
                      bool want_dw) {
    const int rows = (int)pl.rows, E = t->E, HW = pl.HW, Ep = pl.Ep;
    void *dyb = g.dyb, *dt = g.dctx, *dz = g.dk, *dq = g.dq, *dv = g.dv;
    float* dm32 = reinterpret_cast<float*>(w); w += 2 * pl.me;
    float* dn32 = reinterpret_cast<float*>(w); w += 2 * pl.me;
    void* dm = w;     w += pl.me;
    void* dml = w;    w += pl.me;
    void* dn = w;     w += pl.me;
    void* dnl = w;    w += pl.me;
    float* partial = reinterpret_cast<float*>(w); w += pl.partial;
    TBufs tb;
    int rc;
    bool dy_done = part != kWhole;
    if ((rc = composed_forward_core(ctx, t, pl, w, &tb, dy_done ? nullptr : t->dy, dyb, &dy_done))) return rc;
    if (!dy_done && (rc = convert_rows_bf16(ctx, t->dy, E, dyb, Ep, pl.rows, E))) return rc;
    WideArgs wa;
    fill_composed(t, pl, tb, &wa);
    wa.dP = g.dP; wa.dS = g.dS;
    // dP = dy z^T, dz = P^T dy, dS, dT = dS x
    wa.dout = dyb; wa.dos = x_strides(t, Ep);
    wa.dq = dt; wa.dv = dz;
    if ((part & kUpToScores) && (rc = wide_score_value_grads(ctx, wa))) return rc;
    if (part == kWhole && (rc = wide_softmax_grad(ctx, wa))) return rc;
    if (!(part & kFromScores)) return LTCA_OK;
    if ((rc = wide_query_grad(ctx, wa))) return rc;
    if (want_dx) {
        GemmProblem gp;                                // M and N are stored [E, H E] = [N, K]
        gp.M = rows; gp.N = E; gp.K = HW;
        gp.n_sum = 2;
        gp.a[0] = GemmOperand{dt, HW, 0}; gp.b[0] = GemmOperand{tb.m, HW, 0};
        gp.a[1] = GemmOperand{dz, HW, 0}; gp.b[1] = GemmOperand{tb.n, HW, 0};
        gp.c[0] = t->dx;
        gp.ldc = E;
        if ((rc = gemm_sm100(ctx, gp))) return rc;
        if ((rc = sum_over_heads(ctx, t, pl, wa.dS, 1, tb.t, t->dx, nullptr, true))) return rc;
    }
    if (!want_dw) return LTCA_OK;
    {   // dM = x^T dT, dN = x^T dz
        GemmProblem gp;
        gp.M = E; gp.N = HW; gp.K = rows;
        gp.n_problems = 2;
        gp.ksplit = pl.ks_m;
        gp.a[0] = gp.a[1] = GemmOperand{tb.xb, Ep, 1};
        gp.b[0] = GemmOperand{dt, HW, 1}; gp.b[1] = GemmOperand{dz, HW, 1};
        gp.c[0] = dm32; gp.c[1] = dn32;
        gp.ldc = HW;
        gp.partial = partial;
        if ((rc = gemm_sm100(ctx, gp))) return rc;
        const float* src[2] = {dm32, dn32};
        void *hi[2] = {dm, dn}, *lo[2] = {dml, dnl};
        const int64_t ld[2] = {HW, HW}, nrows[2] = {E, E};
        const int ncols[2] = {HW, HW};
        if ((rc = convert_many_bf16(ctx, 2, src, ld, hi, ld, nrows, ncols, lo))) return rc;
    }
    const int64_t wo_h = (int64_t)E * Ep;
    {
        GemmGroup gg;
        gg.heads = t->H; gg.n = 4;
        void* dst[4] = {t->dwq, t->dwk, t->dwv, t->dwo};
        for (int i = 0; i < 4; ++i) {
            GemmGroup::Member& m = gg.m[i];
            const void *hi = i < 2 ? dm : dn, *lo = i < 2 ? dml : dnl;
            m.M = m.N = m.K = E;
            m.terms = i < 2 ? 3 : 2;
            m.a_hs = m.b_hs = m.c_hs = E;
            m.c = dst[i];
            m.ldc = HW;
            for (int k = 0; k < m.terms; ++k) {
                const void* d = k == 1 ? lo : hi;
                if (i == 0) { m.a[k] = GemmOperand{d, HW, 0}; m.b[k] = GemmOperand{k == 2 ? tb.wkl : tb.wk, HW, 1}; }
                if (i == 1) { m.a[k] = GemmOperand{d, HW, 1}; m.b[k] = GemmOperand{k == 2 ? tb.wql : tb.wq, HW, 1}; }
                if (i == 2) { m.a[k] = GemmOperand{d, HW, 0}; m.b[k] = GemmOperand{tb.wo, Ep, 0}; }
                if (i == 3) { m.a[k] = GemmOperand{tb.wv, HW, 1}; m.b[k] = GemmOperand{d, HW, 1}; }
            }
            if (i == 2) m.b_hs = wo_h;
            if (i == 3) { m.ldc = E; m.c_hs = (int64_t)E * E; }
        }
        // results whose rows cannot be stored by TMA: one launch each
        if (gemm_group_aligned(gg)) {
            if ((rc = gemm_sm100_group(ctx, gg))) return rc;
        } else {
            for (int i = 0; i < gg.n; ++i) {
                const GemmGroup::Member& m = gg.m[i];
                if ((rc = per_head(ctx, t, E, m.terms, m.a, m.a_hs, m.b, m.b_hs, m.c, m.ldc, m.c_hs, 0))) return rc;
            }
        }
    }
    if (t->dbq || t->dbk || t->dbv) {
        // Gradients of biases that the module does not have: column sums of dq = dT Wk, dv = dz Wo^T and dk = (dS^T x) Wq.  dk takes
        // dz's place once dv is there, so that the three lie where projected_backward has them.
        const GemmOperand qa = {dt, HW, 0}, qb = {tb.wk, HW, 1}, va = {dz, HW, 0}, vb = {tb.wo, Ep, 0};
        if ((rc = per_head(ctx, t, rows, 1, &qa, E, &qb, E, dq, HW, E, 1))) return rc;
        if ((rc = per_head(ctx, t, rows, 1, &va, E, &vb, wo_h, dv, HW, E, 1))) return rc;
        WideArgs wk = wa;
        wk.qh = tb.xb; wk.ql = nullptr; wk.qs = x_strides(t, Ep);
        wk.dk = dt;
        if ((rc = wide_key_grad(ctx, wk))) return rc;
        const GemmOperand ka = {dt, HW, 0}, kb = {tb.wq, HW, 1};
        if ((rc = per_head(ctx, t, rows, 1, &ka, E, &kb, E, dz, HW, E, 1))) return rc;
    }
    return LTCA_OK;
}

// bf16 copies, fused Q/K/V projection, attention forward.
// `also_src` / `also_dst`: one more [rows, E] fp32 matrix (the backward's dy) to be rounded to bf16 by the same launch
// that rounds x and the weights; *also_done says whether that happened (not on the paths that convert otherwise
// or not at all).
// `outer`: the FlashAttention form around this module; its LayerNorm (of outer->x) and its dropout (of outer->dy, into
// outer_g as fp32 and into also_dst) take the place of those conversions, in the same launch as the weights'.
int tensor_forward_core(ltca_ctx* ctx, const ltca_tsa_params* t, const TPlan& pl, char* w, TBufs* tb,
                        const float* also_src = nullptr, void* also_dst = nullptr, bool* also_done = nullptr,
                        const ltca_tsa_params* outer = nullptr, float* outer_g = nullptr) {
    char* rest = w;
    const bool saved = t->saved != nullptr;
    if (saved) w = kept_block(t);
    w = place_scores(pl, w, tb);
    tb->xb = w;  w += pl.xb;
    tb->wq = w;  w += pl.w_in;
    tb->wk = w;  w += pl.w_in;
    tb->wv = w;  w += pl.w_in;
    tb->wo = w;  w += pl.w_out;
    tb->q = w;   w += pl.act;
    tb->k = w;   w += pl.act;
    tb->v = w;   w += pl.act;
    tb->ctx = w; w += pl.act;
    if (pl.wide) {
        tb->xl = w;  w += pl.xb;
        tb->wql = w; w += pl.w_in;
        tb->wkl = w; w += pl.w_in;
        tb->ql = w;  w += pl.act;
        tb->kl = w;  w += pl.act;
    }
    tb->rest = saved ? rest : w;
    tb->wvl = tb->wol = nullptr;
    // the weights' copies live in the caller's cache when there is one
    const bool cached = t->weight_cache != nullptr;
    if (cached) {
        char* c = reinterpret_cast<char*>(t->weight_cache);
        tb->wq = c;  c += pl.w_in;
        tb->wk = c;  c += pl.w_in;
        tb->wv = c;  c += pl.w_in;
        tb->wo = c;  c += pl.w_out;
        if (pl.wide) { tb->wql = c; c += pl.w_in; tb->wkl = c; c += pl.w_in; }
        // (a call without biases, or with more rows, may find this block valid: composed_forward_core)
        if (composed_weights(t)) { tb->wvl = c; c += pl.w_in; tb->wol = c; }
    }
    const bool convert_weights = !(cached && t->weight_cache_valid);
    if (saved && t->reuse_forward) return LTCA_OK;
    const int E = t->E, HW = pl.HW, Ep = pl.Ep;
    int rc;
    {   // x, the four weight matrices unless their copies are kept, and the caller's extra matrix are rounded to
        // bf16 by one launch.  On the written-out-score path the operands of the products whose rounding would
        // reach the scores - x, Wq, Wk here, q and k below - get a second term.
        const float* src[6] = {t->x, t->wq, t->wk, t->wv, t->wo, nullptr};
        void* dst[6] = {tb->xb, tb->wq, tb->wk, tb->wv, tb->wo, nullptr};
        void* lo[6] = {pl.wide ? tb->xl : nullptr, pl.wide ? tb->wql : nullptr, pl.wide ? tb->wkl : nullptr,
                       tb->wvl, tb->wol, nullptr};
        int64_t ld_src[6] = {E, HW, HW, HW, E, E}, ld_dst[6] = {Ep, HW, HW, HW, Ep, Ep};
        int64_t nrows[6] = {pl.rows, E, E, E, HW, pl.rows};
        int ncols[6] = {E, HW, HW, HW, E, E};
        int n = convert_weights ? 5 : 1;
        if (outer) {
            CvtMany wm;
            const RowOut xo{nullptr, reinterpret_cast<__nv_bfloat16*>(tb->xb), 0, Ep};
            const RowOut go{outer_g, reinterpret_cast<__nv_bfloat16*>(also_dst), E, Ep};
            const bool one = make_cvt_many(&wm, n - 1, src + 1, ld_src + 1, dst + 1, ld_dst + 1, nrows + 1, ncols + 1, nullptr);
            if (!one && n > 1 && (rc = convert_many_bf16(ctx, n - 1, src + 1, ld_src + 1, dst + 1, ld_dst + 1, nrows + 1, ncols + 1)))
                return rc;
            // (the mask's words go where the context says that the call's kernels will find them)
            ltca_attn_params ap;
            fill_attn_bf16(t, &ap);
            const MaskArgs words = mask_args(&ap, ctx->mask_words);
            const bool mask = t->keep_mask && ctx->mask_packed == t->keep_mask;
            if ((rc = prenorm_prepare(ctx, outer, xo, also_src ? &go : nullptr, one ? &wm : nullptr, mask ? &words : nullptr))) return rc;
            if (also_done) *also_done = true;
            n = 0;
        } else if (also_src) {
            src[n] = also_src; dst[n] = also_dst; lo[n] = nullptr;
            ld_src[n] = E; ld_dst[n] = Ep; nrows[n] = pl.rows; ncols[n] = E;
            ++n;
            if (also_done) *also_done = true;
        }
        if (n && (rc = convert_many_bf16(ctx, n, src, ld_src, dst, ld_dst, nrows, ncols, lo))) return rc;
    }
    if (pl.wide) {
        const void* whi[2] = {tb->wq, tb->wk};
        const void* wlo[2] = {tb->wql, tb->wkl};
        void* ohi[2] = {tb->q, tb->k};
        void* olo[2] = {tb->ql, tb->kl};
        const float* bias[2] = {t->bq, t->bk};
        for (int i = 0; i < 2; ++i) {
            // x W = x_hi W_hi + x_hi W_lo + x_lo W_hi in one fp32 accumulator, which the epilogue writes as two
            // bf16 terms
            GemmProblem gp;
            gp.M = (int)pl.rows; gp.N = HW; gp.K = E;
            gp.n_sum = 3;
            gp.a[0] = GemmOperand{tb->xb, Ep, 0}; gp.b[0] = GemmOperand{whi[i], HW, 1};
            gp.a[1] = GemmOperand{tb->xb, Ep, 0}; gp.b[1] = GemmOperand{wlo[i], HW, 1};
            gp.a[2] = GemmOperand{tb->xl, Ep, 0}; gp.b[2] = GemmOperand{whi[i], HW, 1};
            gp.c[0] = ohi[i];
            gp.c_lo = olo[i];
            gp.out_bf16 = 1;
            gp.bias[0] = bias[i];
            gp.ldc = HW;
            if ((rc = gemm_sm100(ctx, gp))) return rc;
        }
        {
            GemmProblem gp;
            gp.M = (int)pl.rows; gp.N = HW; gp.K = E;
            gp.a[0] = GemmOperand{tb->xb, Ep, 0};
            gp.b[0] = GemmOperand{tb->wv, HW, 1};
            gp.c[0] = tb->v;
            gp.bias[0] = t->bv;
            gp.ldc = HW;
            gp.out_bf16 = 1;
            if ((rc = gemm_sm100(ctx, gp))) return rc;
        }
        WideArgs wa;
        fill_wide(t, *tb, &wa);
        return wide_attn_fwd(ctx, wa);
    }
    GemmProblem gp;
    gp.M = (int)pl.rows; gp.N = HW; gp.K = E;
    gp.n_problems = 3;
    const void* wsrc[3] = {tb->wq, tb->wk, tb->wv};
    void* dst[3] = {tb->q, tb->k, tb->v};
    const float* bias[3] = {t->bq, t->bk, t->bv};
    for (int i = 0; i < 3; ++i) {
        gp.a[i] = GemmOperand{tb->xb, Ep, 0};
        gp.b[i] = GemmOperand{wsrc[i], HW, 1};           // stored [E, HW] = [K, N]
        gp.c[i] = dst[i];
        gp.bias[i] = bias[i];
    }
    gp.ldc = HW;
    gp.out_bf16 = 1;
    if ((rc = gemm_sm100(ctx, gp))) return rc;
    ltca_attn_params a;
    fill_attn_bf16(t, &a);
    a.q = tb->q; a.k = tb->k; a.v = tb->v; a.o = tb->ctx; a.lse = tb->lse;
    a.workspace = pl.attn_fwd ? tb->rest : nullptr;
    a.workspace_bytes = pl.attn_fwd;
    return ltca_attn_fwd(ctx, &a);
}

// `outer` (or null): the FlashAttention form around this module, `fused`: its first steps are done in here.
int tensor_forward(ltca_ctx* ctx, const ltca_tsa_params* t, const ltca_tsa_params* outer, bool fused) {
    TPlan pl;
    int rc;
    const ltca_tsa_params layout = laid_out(t, 0);
    if ((rc = make_tplan(&layout, &pl, keeps_for_backward(t)))) return rc;
    const size_t need = tensor_workspace(pl, 0);
    if (!t->workspace || t->workspace_bytes < need)
        return fail(ctx, LTCA_ERR_WORKSPACE, "forward needs %zu bytes of workspace", need);
    char* w = reinterpret_cast<char*>(t->workspace);
    float* y = reinterpret_cast<float*>(w);
    w += pl.y;
    TBufs tb;
    CallHints hints{ctx};
    ctx->fwd_pairs = t->bk != nullptr;
    if (fused && (rc = place_mask_words(ctx, &layout, pl, scratch_of(t, pl, w), pl.attn_fwd, true))) return rc;
    if (pl.composed) {
        if ((rc = composed_forward_core(ctx, t, pl, w, &tb, nullptr, nullptr, nullptr))) return rc;
        if ((rc = sum_over_heads(ctx, t, pl, tb.P, 0, tb.z, y, t->bo, false))) return rc;
        return outer ? prenorm_finish(ctx, outer, y) : residual_layer_norm(ctx, t, y, pl.rows);
    }
    if ((rc = tensor_forward_core(ctx, t, pl, w, &tb, nullptr, nullptr, nullptr, fused ? outer : nullptr))) return rc;
    GemmProblem gp;
    gp.M = (int)pl.rows; gp.N = t->E; gp.K = pl.HW;
    gp.a[0] = GemmOperand{tb.ctx, pl.HW, 0};
    gp.b[0] = GemmOperand{tb.wo, pl.Ep, 1};              // stored [HW, E] = [K, N]
    gp.c[0] = y;
    gp.bias[0] = t->bo;
    gp.ldc = t->E;
    if ((rc = gemm_sm100(ctx, gp))) return rc;
    return outer ? prenorm_finish(ctx, outer, y) : residual_layer_norm(ctx, t, y, pl.rows);
}

// tensor_backward on q, k, v and ctx.  `w`: the workspace behind `g`.  In parts only on the written-out-score path, from a kept forward and
// with dy's bf16 copy in its place.
int projected_backward(ltca_ctx* ctx, const ltca_tsa_params* t, const ltca_tsa_params& layout, const TPlan& pl, const BwdBufs& g, char* w,
                       BwdPart part, bool want_dx, bool want_dw, ColSum* sums, const ltca_tsa_params* outer, float* outer_g) {
    void *dyb = g.dyb, *dctx = g.dctx, *dq = g.dq, *dk = g.dk, *dv = g.dv;
    int rc;
    float* partial = reinterpret_cast<float*>(w); w += pl.partial;
    TBufs tb;
    // the forward is recomputed, as the reference's caller does before each backward
    // (src/ml/ml_liquid_net.cu:715-721)
    // the recomputed attention and its backward read the same mask: packed once, behind what either uses of the scratch
    ctx->fwd_pairs = t->bk != nullptr;
    const size_t most = pl.attn_fwd > pl.attn_bwd ? pl.attn_fwd : pl.attn_bwd;
    if ((rc = place_mask_words(ctx, &layout, pl, scratch_of(t, pl, w), most, outer && !(t->saved && t->reuse_forward)))) return rc;
    bool dy_done = part != kWhole;
    if ((rc = tensor_forward_core(ctx, t, pl, w, &tb, dy_done ? nullptr : t->dy, dyb, &dy_done, outer, outer_g))) return rc;
    const int rows = (int)pl.rows, E = t->E, HW = pl.HW, Ep = pl.Ep;
    if (!dy_done && (rc = convert_rows_bf16(ctx, t->dy, E, dyb, Ep, pl.rows, E))) return rc;
    if (part & kUpToScores) {   // dctx = dy Wo^T : Wo is stored [HW, E] = [N, K]
        GemmProblem gp;
        gp.M = rows; gp.N = HW; gp.K = E;
        gp.a[0] = GemmOperand{dyb, Ep, 0};
        gp.b[0] = GemmOperand{tb.wo, Ep, 0};
        gp.c[0] = dctx;
        gp.ldc = HW;
        gp.out_bf16 = 1;
        if ((rc = gemm_sm100(ctx, gp))) return rc;
    }
    if (pl.wide) {
        WideArgs wa;
        fill_wide(t, tb, &wa);
        wa.dout = dctx; wa.dq = dq; wa.dk = dk; wa.dv = dv;
        wa.dP = g.dP; wa.dS = g.dS;
        if ((part & kUpToScores) && (rc = wide_score_value_grads(ctx, wa))) return rc;
        if (part == kWhole && (rc = wide_softmax_grad(ctx, wa))) return rc;
        if (!(part & kFromScores)) return LTCA_OK;
        if ((rc = wide_query_grad(ctx, wa)) || (rc = wide_key_grad(ctx, wa))) return rc;
    } else {
        ltca_attn_params a;
        fill_attn_bf16(t, &a);
        a.q = tb.q; a.k = tb.k; a.v = tb.v; a.o = tb.ctx; a.lse = tb.lse;
        a.dout = dctx; a.dq = dq; a.dk = dk; a.dv = dv;
        a.workspace = pl.attn_bwd ? tb.rest : nullptr;
        a.workspace_bytes = pl.attn_bwd;
        if ((rc = ltca_attn_bwd(ctx, &a))) return rc;
    }
    const void* grads[3] = {dq, dk, dv};
    if (want_dx && want_dw && pl.n_dw == 4 && part == kWhole && !pl.wide) {
        // dx and the four weight gradients (each below) where their tiles fit beside one another: a launch less (FlashAttention module
        // backward B16 S200 E256 H4 80.5 -> 72.5 us, module backward B8 S128 E256 H4 37 -> 29)
        GemmGroup gg;
        gg.n = 5;
        const void* wsrc[3] = {tb.wq, tb.wk, tb.wv};
        void* dst[4] = {t->dwq, t->dwk, t->dwv, t->dwo};
        GemmGroup::Member& x = gg.m[4];
        x.M = rows; x.N = E; x.K = HW;
        x.terms = 3;
        x.c = t->dx; x.ldc = E;
        for (int i = 0; i < 3; ++i) {
            x.a[i] = GemmOperand{grads[i], HW, 0};
            x.b[i] = GemmOperand{wsrc[i], HW, 0};
        }
        const int64_t mn = (int64_t)E * HW;
        for (int i = 0; i < 4; ++i) {
            GemmGroup::Member& m = gg.m[i];
            m.M = E; m.N = HW; m.K = rows;
            m.ksplit = pl.ks_in;
            m.a[0] = i < 3 ? GemmOperand{tb.xb, Ep, 1} : GemmOperand{tb.ctx, HW, 1};
            m.b[0] = i < 3 ? GemmOperand{grads[i], HW, 1} : GemmOperand{dyb, Ep, 1};
            m.c = pl.ks_in > 1 ? partial + i * pl.ks_in * mn : dst[i];
            m.ldc = HW;
        }
        if (gemm_group_one_wave(ctx, gg) && gemm_group_aligned(gg)) {
            if ((rc = gemm_sm100_group(ctx, gg)) || pl.ks_in == 1) return rc;
            if (sums->tail) {
                sums->split = partial;
                for (int i = 0; i < 4; ++i) sums->split_dst[i] = static_cast<float*>(dst[i]);
                sums->split_mn = mn; sums->splits = pl.ks_in; sums->split_n = 4;
                return LTCA_OK;
            }
            return sum_splits(ctx, partial, dst, 4, mn, pl.ks_in);
        }
    }
    if (want_dx) {
        // dx = dq Wq^T + dk Wk^T + dv Wv^T : each W is stored [E, HW] = [N, K]; one accumulator tile
        GemmProblem gp;
        gp.M = rows; gp.N = E; gp.K = HW;
        gp.n_sum = 3;
        const void* wsrc[3] = {tb.wq, tb.wk, tb.wv};
        for (int i = 0; i < 3; ++i) {
            gp.a[i] = GemmOperand{grads[i], HW, 0};
            gp.b[i] = GemmOperand{wsrc[i], HW, 0};
        }
        gp.c[0] = t->dx;
        gp.ldc = E;
        if ((rc = gemm_sm100(ctx, gp))) return rc;
    }
    if (want_dw) {
        {   // dW = x^T dq : x is stored [rows, E] = [K, M], dq [rows, HW] = [K, N]
            GemmProblem gp;
            gp.M = E; gp.N = HW; gp.K = rows;
            gp.n_problems = pl.n_dw;
            gp.ksplit = pl.ks_in;
            void* dst[3] = {t->dwq, t->dwk, t->dwv};
            for (int i = 0; i < 3; ++i) {
                gp.a[i] = GemmOperand{tb.xb, Ep, 1};
                gp.b[i] = GemmOperand{grads[i], HW, 1};
                gp.c[i] = dst[i];
            }
            if (gp.n_problems == 4) {
                gp.a[3] = GemmOperand{tb.ctx, HW, 1};
                gp.b[3] = GemmOperand{dyb, Ep, 1};
                gp.c[3] = t->dwo;
            }
            gp.ldc = HW;
            gp.partial = partial;
            if ((rc = gemm_sm100(ctx, gp))) return rc;
        }
        if (pl.n_dw == 3) {   // dWo = ctx^T dy
            GemmProblem gp;
            gp.M = HW; gp.N = E; gp.K = rows;
            gp.ksplit = pl.ks_out;
            gp.a[0] = GemmOperand{tb.ctx, HW, 1};
            gp.b[0] = GemmOperand{dyb, Ep, 1};
            gp.c[0] = t->dwo;
            gp.ldc = E;
            gp.partial = partial;
            if ((rc = gemm_sm100(ctx, gp))) return rc;
        }
    }
    return LTCA_OK;
}

// `sums` collects the bias gradients (column sums of buffers that stay as they are until the call ends).
int tensor_backward(ltca_ctx* ctx, const ltca_tsa_params* t, bool want_dx, bool want_dw, ColSum* sums,
                    const ltca_tsa_params* outer, float* outer_g) {
    TPlan pl[2];                                       // projections; products of the weights
    int rc;
    const ltca_tsa_params layout = laid_out(t, 1);
    // A kept forward of either form: both backwards are launched, each to run where the block is its own.  (What the other one's
    // eight or nine launches cost: backward of B32 S256 E512 H8 313 us and 299 without them, B16 S256 E256 H4 113 and 93; by itself
    // the path through q, k, v and ctx takes 405 and 106.)
    const bool either = t->saved && t->reuse_forward && composed_shape(t);
    const bool composed = use_composed(t);
    size_t need = 0;
    for (int i = 0; i < 2; ++i) {
        if (!either && i != (composed ? 1 : 0)) continue;
        if ((rc = make_tplan_as(&layout, &pl[i], true, i == 1))) return rc;
        const size_t n = tensor_workspace(pl[i], 1);
        if (n > need) need = n;
    }
    if (!t->workspace || t->workspace_bytes < need)
        return fail(ctx, LTCA_ERR_WORKSPACE, "backward needs %zu bytes of workspace", need);
    const TPlan& any = pl[composed ? 1 : 0];
    char* w = reinterpret_cast<char*>(t->workspace);
    BwdBufs g;
    g.dyb = w;  w += any.xb;
    g.dctx = w; w += any.act;
    g.dq = w;   w += any.act;
    g.dk = w;   w += any.act;
    g.dv = w;   w += any.act;
    g.dP = reinterpret_cast<float*>(w); w += any.mat32;
    g.dS = w;   w += any.mat16;
    CallHints hints{ctx};
    if (either) {
        // (an ordinary launch, as the kernels that look at the word need before them: skipped, sm100_ptx.cuh)
        if ((rc = convert_rows_bf16(ctx, t->dy, t->E, g.dyb, any.Ep, any.rows, t->E))) return rc;
        for (BwdPart part : {kUpToScores, kFromScores}) {
            if (part == kFromScores) {
                ctx->run_if = RunIf();
                TBufs tb{};
                WideArgs wa;
                place_scores(any, kept_block(t), &tb);
                fill_wide(t, tb, &wa);
                wa.dP = g.dP; wa.dS = g.dS;
                if ((rc = wide_softmax_grad(ctx, wa))) return rc;
            }
            ctx->run_if.word = reinterpret_cast<const uint32_t*>(t->saved);
            ctx->run_if.value = kKeptProjections;
            if ((rc = projected_backward(ctx, t, layout, pl[0], g, w, part, want_dx, want_dw, sums, outer, outer_g))) return rc;
            ctx->run_if.value = kKeptComposed;
            if ((rc = composed_backward(ctx, t, pl[1], g, w, part, want_dx, want_dw))) return rc;
        }
        ctx->run_if = RunIf();
    } else if (composed) {
        if ((rc = composed_backward(ctx, t, pl[1], g, w, kWhole, want_dx, want_dw))) return rc;
    } else {
        if ((rc = projected_backward(ctx, t, layout, pl[0], g, w, kWhole, want_dx, want_dw, sums, outer, outer_g))) return rc;
    }
    if (want_dw) {
        // bias gradients (FlashAttention form): column sums of the projection outputs' gradients
        sums->add(g.dq, true, any.HW, any.HW, t->dbq);
        sums->add(g.dk, true, any.HW, any.HW, t->dbk);
        sums->add(g.dv, true, any.HW, any.HW, t->dbv);
        sums->add(t->dy, false, t->E, t->E, t->dbo);
    }
    return LTCA_OK;
}

// Workspace of the TimeSelfAttention form (no input LayerNorm, no dropout), without the column-sum scratch.
int inner_workspace(const ltca_tsa_params* t, int which, Room room, size_t* bytes_out) {
    if (use_tensor(t, which != 0 || keeps_for_backward(t))) {
        return planned_bytes(t, which != 0 || keeps_for_backward(t), [&](const TPlan& tp) { return tensor_workspace(tp, which); },
                             bytes_out);
    }
    Plan pl;
    int rc = make_plan(t, &pl, room);
    if (rc) return rc;
    size_t n = 4 * pl.buf + pl.lse;                       // q, k, v, ctx, lse
    if (which == 0) {
        n += pl.y;                                        // y before residual / LayerNorm
        n += pl.attn_fwd;
    } else {
        n += 4 * pl.buf;                                  // dctx, dq, dk, dv
        n += pl.attn_fwd > pl.attn_bwd ? pl.attn_fwd : pl.attn_bwd;
    }
    *bytes_out = n;
    return LTCA_OK;
}

// The module without the FlashAttention-form steps: what the pre_norm wrappers run in the middle.
ltca_tsa_params core_form(const ltca_tsa_params* t) {
    ltca_tsa_params c = *t;
    c.pre_norm = 0;
    c.use_residual = 0;
    c.use_layer_norm = 0;
    c.dropout_prob = 0.f;
    c.dgamma = nullptr;
    c.dbeta = nullptr;
    return c;
}
size_t act_bytes(const ltca_tsa_params* t) {
    return align_up((size_t)t->B * t->S * t->E * sizeof(float), 256);
}

int workspace_bytes(const ltca_tsa_params* t, int which, Room room, size_t* bytes_out) {
    size_t n = 0;
    int rc;
    if (t->pre_norm) {
        const ltca_tsa_params c = core_form(t);
        if ((rc = inner_workspace(&c, which, room, &n))) return rc;
        n += (which == 0 ? 1 : 3) * act_bytes(t);         // LayerNorm(x); backward: + masked dy, gradient at LayerNorm(x)
    } else if ((rc = inner_workspace(t, which, room, &n))) {
        return rc;
    }
    if (which != 0) n += colsum_scratch_bytes(t);
    *bytes_out = n;
    return LTCA_OK;
}

}  // namespace
}  // namespace ltca

using namespace ltca;

extern "C" {

int ltca_tsa_saved_bytes(const ltca_tsa_params* t, size_t* bytes_out) {
    if (!t || !bytes_out) return LTCA_ERR_INVALID;
    if (t->pre_norm) return LTCA_ERR_UNSUPPORTED;
    ltca_tsa_params probe = *t;
    probe.saved = nullptr;
    if (use_tensor(&probe, true)) {
        return planned_bytes(&probe, true, [&](const TPlan& tp) { return kept_word_bytes(&probe) + tensor_saved_bytes(tp); }, bytes_out);
    }
    Plan pl;
    int rc = make_plan(&probe, &pl);
    if (rc) return rc;
    *bytes_out = 4 * pl.buf + pl.lse;
    return LTCA_OK;
}

int ltca_tsa_weight_cache_bytes(const ltca_tsa_params* t, size_t* bytes_out) {
    if (!t || !bytes_out) return LTCA_ERR_INVALID;
    *bytes_out = 0;
    // the cache serves the pipeline that the backward takes, which a forward with a cache takes too
    if (!use_tensor(t, true)) return LTCA_OK;
    TPlan tp;
    int rc = make_tplan(t, &tp, true);
    if (rc) return rc;
    *bytes_out = 3 * tp.w_in + tp.w_out + (tp.wide ? 2 * tp.w_in : 0) + (composed_weights(t) ? tp.w_in + tp.w_out : 0);
    return LTCA_OK;
}

int ltca_tsa_workspace_bytes(const ltca_tsa_params* t, int which, size_t* bytes_out) {
    if (!t || !bytes_out || which < 0 || which > 3) return LTCA_ERR_INVALID;
    return workspace_bytes(t, which, kFullRoom, bytes_out);
}

static int tsa_forward(ltca_ctx* ctx, const ltca_tsa_params* t, const ltca_tsa_params* outer, bool fused);
static int tsa_backward(ltca_ctx* ctx, const ltca_tsa_params* t, bool want_dx, bool want_dw, ColSum* sums,
                        const ltca_tsa_params* outer, float* outer_g);

// Whether the core of the module takes the raw rows and runs the first steps of the FlashAttention form itself: the
// streaming tensor pipeline, whose operands are bf16.  (The exact pipeline and the written-out-score path, which keeps a
// second term of x, read fp32 rows.)
static bool fuses_prenorm(const ltca_tsa_params* c, bool backward) {
    return use_tensor(c, backward) && !use_wide(c, backward);
}

// FlashAttention form, forward: LayerNorm on the input, the core module, residual with the raw input, dropout.
static int prenorm_forward(ltca_ctx* ctx, const ltca_tsa_params* t) {
    size_t need = 0;
    const ltca_tsa_params layout = laid_out(t, 0);
    int rc = ltca_tsa_workspace_bytes(&layout, 0, &need);
    if (rc) return rc;
    if (!t->workspace || t->workspace_bytes < need)
        return fail(ctx, LTCA_ERR_WORKSPACE, "forward needs %zu bytes of workspace", need);
    char* w = reinterpret_cast<char*>(t->workspace);
    float* xin = reinterpret_cast<float*>(w);
    w += act_bytes(t);
    ltca_tsa_params c = core_form(t);
    const bool fused = fuses_prenorm(&c, keeps_for_backward(&c));
    if (!fused && t->use_layer_norm) {
        const RowOut xo{xin, nullptr, t->E, 0};
        if ((rc = prenorm_prepare(ctx, t, xo, nullptr, nullptr))) return rc;
        c.x = xin;
    }
    c.workspace = w;
    c.workspace_bytes = t->workspace_bytes - act_bytes(t);
    return tsa_forward(ctx, &c, t, fused);
}

// FlashAttention form, backward (an extension: the reference class has no backward pass).
static int prenorm_backward(ltca_ctx* ctx, const ltca_tsa_params* t, bool want_dx, bool want_dw) {
    const Layout layout = lay_out(t, 1);
    const size_t need = layout.need;
    int rc = layout.rc;
    if (rc) return rc;
    if (!t->workspace || t->workspace_bytes < need)
        return fail(ctx, LTCA_ERR_WORKSPACE, "backward needs %zu bytes of workspace", need);
    if (t->use_layer_norm && !t->ln_gamma) return fail(ctx, LTCA_ERR_INVALID, "LayerNorm needs gamma");
    const int64_t rows = (int64_t)t->B * t->S;
    const int64_t n = rows * t->E;
    const size_t act = act_bytes(t);
    char* w = reinterpret_cast<char*>(t->workspace);
    float* xin = reinterpret_cast<float*>(w);   w += act;
    float* gbuf = reinterpret_cast<float*>(w);  w += act;
    float* dxin = reinterpret_cast<float*>(w);  w += act;
    float* colsum_scratch = reinterpret_cast<float*>(reinterpret_cast<char*>(t->workspace) + need - colsum_scratch_bytes(t));
    ltca_tsa_params c = core_form(t);
    const bool fused = fuses_prenorm(&c, true);
    const bool drops = t->dropout_prob > 0.f;
    const float* g = drops ? gbuf : t->dy;       // gradient behind the dropout
    if (!fused) {
        const RowOut xo{t->use_layer_norm ? xin : nullptr, nullptr, t->E, 0}, go{drops ? gbuf : nullptr, nullptr, t->E, 0};
        if ((rc = prenorm_prepare(ctx, t, xo, &go, nullptr))) return rc;
        if (t->use_layer_norm) c.x = xin;
    }
    const bool want_ln_params = want_dw && t->use_layer_norm && (t->dgamma || t->dbeta);
    const bool need_dxin = want_dx || want_ln_params;
    c.dy = g;
    c.dx = dxin;
    c.workspace = w;
    c.workspace_bytes = t->workspace_bytes - 3 * act;
    ColSum sums;
    memset(&sums, 0, sizeof(sums));
    const bool vec = row_pieces(t->E) == 0 || aligned16(dxin, t->x, t->ln_gamma, g, t->dx);
    sums.tail = need_dxin && t->use_layer_norm && tail_width(t->E) && vec;
    if ((rc = tsa_backward(ctx, &c, need_dxin, want_dw, &sums, fused ? t : nullptr, drops ? gbuf : nullptr))) return rc;
    if (need_dxin && !t->use_layer_norm) {
        if (want_dx && t->use_residual) {
            if ((rc = ltca_add_tensors(ctx, dxin, g, t->dx, (size_t)n))) return rc;
        } else if (want_dx) {
            LTCA_CUDA_OK(ctx, cudaMemcpyAsync(t->dx, dxin, (size_t)n * sizeof(float), cudaMemcpyDeviceToDevice, ctx->stream));
        }
    } else if (sums.tail) {
        sums.ln_g = dxin; sums.ln_x = t->x; sums.ln_gamma = t->ln_gamma;
        sums.ln_res = want_dx && t->use_residual ? g : nullptr;
        sums.ln_dx = want_dx ? t->dx : nullptr;
        sums.ln_dgamma = want_ln_params ? t->dgamma : nullptr;
        sums.ln_dbeta = want_ln_params ? t->dbeta : nullptr;
        sums.E = t->E;
        sums.eps = 1e-5f;
        return module_tail(ctx, sums, rows, colsum_scratch);
    } else if (need_dxin) {
        // LayerNorm(x) is no longer needed: its buffer takes dxin * xhat, whose column sums are dgamma
        float* prod = (want_ln_params && t->dgamma) ? xin : nullptr;
        const int wpb = 8;
        auto kern = layer_norm_bwd_kernel<0>;
        switch (row_pieces(t->E)) {
            case 1: kern = layer_norm_bwd_kernel<1>; break;
            case 2: kern = layer_norm_bwd_kernel<2>; break;
            case 3: kern = layer_norm_bwd_kernel<3>; break;
            case 4: kern = layer_norm_bwd_kernel<4>; break;
            case 5: kern = layer_norm_bwd_kernel<5>; break;
            case 6: kern = layer_norm_bwd_kernel<6>; break;
            case 7: kern = layer_norm_bwd_kernel<7>; break;
            case 8: kern = layer_norm_bwd_kernel<8>; break;
        }
        LTCA_CUDA_OK(ctx, launch_dependent(kern, dim3((unsigned)((rows + wpb - 1) / wpb)), dim3(wpb * 32), 0, ctx->stream,
                                           (const float*)dxin, t->x, t->ln_gamma, (want_dx && t->use_residual) ? g : nullptr,
                                           want_dx ? t->dx : nullptr, prod, rows, t->E, 1e-5f));
        if (want_ln_params) {
            sums.add(dxin, false, t->E, t->E, t->dbeta);
            sums.add(prod, false, t->E, t->E, t->dgamma);
        }
    }
    return column_sums(ctx, sums, rows, colsum_scratch);
}

// `outer` (or null): the FlashAttention form around this module; see tensor_forward.
static int tsa_forward(ltca_ctx* ctx, const ltca_tsa_params* t, const ltca_tsa_params* outer, bool fused) {
    int rc = check(ctx, t);
    if (rc) return rc;
    LTCA_CUDA_OK(ctx, cudaSetDevice(ctx->device));
    if (!t->out) return fail(ctx, LTCA_ERR_INVALID, "out must be non-null");
    if (t->use_layer_norm && (!t->ln_gamma || !t->ln_beta))
        return fail(ctx, LTCA_ERR_INVALID, "LayerNorm needs gamma and beta");
    if (t->dropout_prob < 0.f || t->dropout_prob >= 1.f)
        return fail(ctx, LTCA_ERR_INVALID, "dropout_prob must be in [0, 1)");
    if (t->pre_norm) return prenorm_forward(ctx, t);
    if (use_tensor(t, keeps_for_backward(t))) return tensor_forward(ctx, t, outer, fused);
    Plan pl;
    const ltca_tsa_params layout = laid_out(t, 0);
    if ((rc = make_plan(&layout, &pl))) return rc;
    size_t need = 0;
    ltca_tsa_workspace_bytes(&layout, 0, &need);
    if (!t->workspace || t->workspace_bytes < need)
        return fail(ctx, LTCA_ERR_WORKSPACE, "forward needs %zu bytes of workspace", need);
    char* w = reinterpret_cast<char*>(t->workspace);
    float* y = reinterpret_cast<float*>(w);
    w += pl.y;
    FwdBufs fb;
    if ((rc = forward_core(ctx, t, pl, w, &fb, pl.attn_fwd))) return rc;
    if (!outer && projects_and_norms(t, pl.rows, pl.HW)) return project_norm(ctx, t, fb.ctx, pl.rows, pl.HW);
    const int rows = (int)pl.rows;
    const Gemm32Problem proj = {fb.ctx, t->wo, t->bo, y, rows, t->E, pl.HW, pl.HW, t->E, t->E};
    if ((rc = gemm_fp32(ctx, &proj, 1, 0, 0, false, true))) return rc;
    return outer ? prenorm_finish(ctx, outer, y) : residual_layer_norm(ctx, t, y, pl.rows);
}

int ltca_tsa_fwd(ltca_ctx* ctx, const ltca_tsa_params* t) { return tsa_forward(ctx, t, nullptr, false); }

// `sums` (or null): the FlashAttention form around this module collects the bias gradients' column sums and runs them.
static int tsa_backward(ltca_ctx* ctx, const ltca_tsa_params* t, bool want_dx, bool want_dw, ColSum* sums,
                        const ltca_tsa_params* outer, float* outer_g) {
    int rc = check(ctx, t);
    if (rc) return rc;
    LTCA_CUDA_OK(ctx, cudaSetDevice(ctx->device));
    if (!t->dy) return fail(ctx, LTCA_ERR_INVALID, "dy must be non-null");
    if (want_dx && !t->dx) return fail(ctx, LTCA_ERR_INVALID, "dx must be non-null");
    if (want_dw && (!t->dwq || !t->dwk || !t->dwv || !t->dwo))
        return fail(ctx, LTCA_ERR_INVALID, "dwq, dwk, dwv, dwo must be non-null");
    if (t->dropout_prob < 0.f || t->dropout_prob >= 1.f)
        return fail(ctx, LTCA_ERR_INVALID, "dropout_prob must be in [0, 1)");
    if (t->pre_norm) return prenorm_backward(ctx, t, want_dx, want_dw);
    const Layout layout = lay_out(t, 1);
    const size_t need = layout.need;
    if (!t->workspace || t->workspace_bytes < need)
        return fail(ctx, LTCA_ERR_WORKSPACE, "backward needs %zu bytes of workspace", need);
    float* colsum_scratch =
        reinterpret_cast<float*>(reinterpret_cast<char*>(t->workspace) + need - colsum_scratch_bytes(t));
    ColSum own;
    memset(&own, 0, sizeof(own));
    ColSum* jobs = sums ? sums : &own;
    if (use_tensor(t, true)) {
        if ((rc = tensor_backward(ctx, t, want_dx, want_dw, jobs, outer, outer_g))) return rc;
        return column_sums(ctx, own, (int64_t)t->B * t->S, colsum_scratch);
    }
    Plan pl;
    if ((rc = make_plan(&layout.t, &pl, layout.room))) return rc;
    char* w = reinterpret_cast<char*>(t->workspace);
    float* dctx = reinterpret_cast<float*>(w); w += pl.buf;
    float* dq = reinterpret_cast<float*>(w);   w += pl.buf;
    float* dk = reinterpret_cast<float*>(w);   w += pl.buf;
    float* dv = reinterpret_cast<float*>(w);   w += pl.buf;
    FwdBufs fb;
    // the forward is recomputed, as the reference's caller does before each backward
    // (src/ml/ml_liquid_net.cu:715-721)
    if ((rc = forward_core(ctx, t, pl, w, &fb, pl.attn_fwd))) return rc;
    const int rows = (int)pl.rows, E = t->E, HW = pl.HW;
    ltca_attn_params a;
    fill_attn(t, &a);
    a.q = fb.q; a.k = fb.k; a.v = fb.v; a.o = fb.ctx; a.lse = fb.lse;
    a.dout = dctx; a.dq = dq; a.dk = dk; a.dv = dv;
    a.workspace = pl.attn_bwd ? fb.rest : nullptr;
    a.workspace_bytes = pl.attn_bwd;
    // dctx = dy Wo^T
    const ltca_strides dys = x_strides(t, E);
    const FromOutput from = {t->dy, t->wo, E, dys.batch, dys.seq};
    if (attn_bwd_exact(&a) && attn_bwd_fp32_forms_dout(ctx, &a, from)) {
        if ((rc = launch_attn_bwd_fp32(ctx, &a, &from))) return rc;
    } else {
        const Gemm32Problem back = {t->dy, t->wo, nullptr, dctx, rows, HW, E, E, E, HW};
        if ((rc = gemm_fp32(ctx, &back, 1, 0, 1, false, false))) return rc;
        if ((rc = ltca_attn_bwd(ctx, &a))) return rc;
    }
    if (want_dw) {
        // bias gradients (FlashAttention form): column sums of the projection outputs' gradients
        jobs->add(dq, false, HW, HW, t->dbq);
        jobs->add(dk, false, HW, HW, t->dbk);
        jobs->add(dv, false, HW, HW, t->dbv);
        jobs->add(t->dy, false, E, E, t->dbo);
    }
    const Gemm32Problem terms[3] = {{dq, t->wq, nullptr, t->dx, rows, E, HW, HW, HW, E},
                                    {dk, t->wk, nullptr, t->dx, rows, E, HW, HW, HW, E},
                                    {dv, t->wv, nullptr, t->dx, rows, E, HW, HW, HW, E}};
    // dW = x^T dQ  ([E, rows] x [rows, HW]),  dWo = ctx^T dy  ([HW, rows] x [rows, E])
    // dctx is dead once the attention backward has run: it holds the contraction slices
    const Gemm32Problem dw[4] = {{t->x, dq, nullptr, t->dwq, E, HW, rows, E, HW, HW},
                                 {t->x, dk, nullptr, t->dwk, E, HW, rows, E, HW, HW},
                                 {t->x, dv, nullptr, t->dwv, E, HW, rows, E, HW, HW},
                                 {fb.ctx, t->dy, nullptr, t->dwo, HW, E, rows, HW, E, E}};
    if (want_dx && want_dw) rc = gemm_fp32_grads(ctx, terms, 3, dw, 4, dctx, pl.buf);
    else if (want_dx) rc = gemm_fp32(ctx, terms, 3, 0, 1, true, true);
    else if (want_dw) rc = gemm_fp32(ctx, dw, 4, 1, 0, false, true, dctx, pl.buf);
    if (rc) return rc;
    return column_sums(ctx, own, pl.rows, colsum_scratch);
}

int ltca_tsa_bwd_data(ltca_ctx* ctx, const ltca_tsa_params* t) {
    return tsa_backward(ctx, t, true, false, nullptr, nullptr, nullptr);
}
int ltca_tsa_bwd_weights(ltca_ctx* ctx, const ltca_tsa_params* t) {
    return tsa_backward(ctx, t, false, true, nullptr, nullptr, nullptr);
}
int ltca_tsa_bwd(ltca_ctx* ctx, const ltca_tsa_params* t) {
    return tsa_backward(ctx, t, true, true, nullptr, nullptr, nullptr);
}

}  // extern "C"
