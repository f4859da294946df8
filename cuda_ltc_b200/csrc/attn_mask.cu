// Packs a dense fp32 keep-mask into the words the attention kernels read (attn_mask.cuh).
#include "attn_mask.cuh"

namespace ltca {

namespace {

// One warp per block of 32 queries x 32 keys: lane l reads key l of each query (coalesced); the vote over a query's 32
// values is its row word, the values a lane has seen are its key's column word.
__global__ void __launch_bounds__(256) mask_words_kernel(const float* __restrict__ mask, uint32_t* __restrict__ by_query,
                                                         uint32_t* __restrict__ by_key, int64_t blocks, int Sq, int Sk, int nq, int nk) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int lane = threadIdx.x & 31;
    for (int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); w < blocks; w += (int64_t)gridDim.x * 8) {
        const int kw = (int)(w % nk), qw = (int)(w / nk % nq);
        const int64_t b = w / ((int64_t)nk * nq);
        const int q0 = qw * 32, k = kw * 32 + lane;
        const float* src = mask + (b * Sq + q0) * Sk + k;
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = (k < Sk && q0 + i < Sq) ? __ldg(src + (int64_t)i * Sk) : 0.f;
        uint32_t row = 0, col = 0;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const bool keep = v[i] != 0.f;
            const uint32_t bits = __ballot_sync(0xffffffffu, keep);
            if (lane == i) row = bits;
            col |= (keep ? 1u : 0u) << i;
        }
        if (q0 + lane < Sq) by_query[(b * Sq + q0 + lane) * nk + kw] = row;
        if (k < Sk) by_key[(b * Sk + k) * nq + qw] = col;
    }
}

}  // namespace

int pack_mask_words(ltca_ctx* ctx, const ltca_attn_params* p, void* words) {
    const MaskArgs m = mask_args(p, words);
    const int64_t blocks = (int64_t)p->B * m.nq * m.nk, ctas = (blocks + 7) / 8;
    const int64_t most = 8ll * (ctx->sm_device > 0 ? ctx->sm_device : kPlanSms);
    LTCA_CUDA_OK(ctx, launch_dependent(mask_words_kernel, dim3((unsigned)(ctas < most ? ctas : most)), dim3(256), 0, ctx->stream,
                                       p->keep_mask, const_cast<uint32_t*>(m.by_query), const_cast<uint32_t*>(m.by_key), blocks, p->Sq,
                                       p->Sk, m.nq, m.nk));
    return LTCA_OK;
}

int mask_words_of(ltca_ctx* ctx, const ltca_attn_params* p, size_t used, const void** words) {
    *words = nullptr;
    if (!p->keep_mask) return LTCA_OK;
    if (ctx->mask_packed == p->keep_mask && ctx->mask_words) {
        *words = ctx->mask_words;
        return LTCA_OK;
    }
    if (!p->workspace || (reinterpret_cast<uintptr_t>(p->workspace) & 255) || p->workspace_bytes < used + mask_words_bytes(p))
        return LTCA_OK;
    void* w = reinterpret_cast<char*>(p->workspace) + used;
    *words = w;
    return pack_mask_words(ctx, p, w);
}

}  // namespace ltca
