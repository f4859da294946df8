// Packs a dense fp32 keep-mask into the words the attention kernels read (attn_mask.cuh).
#include "attn_mask.cuh"

namespace ltca {

namespace {

__global__ void __launch_bounds__(256) mask_words_kernel(const MaskArgs m, int B) {
    grid_dependency_wait();
    write_mask_words(m, B, (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5), (int64_t)gridDim.x * 8);
}

}  // namespace

int pack_mask_words(ltca_ctx* ctx, const ltca_attn_params* p, void* words) {
    const MaskArgs m = mask_args(p, words);
    const int64_t blocks = (int64_t)p->B * m.nq * m.nk, ctas = (blocks + 7) / 8;
    const int64_t most = 8ll * (ctx->sm_device > 0 ? ctx->sm_device : kPlanSms);
    LTCA_CUDA_OK(ctx, launch_dependent(mask_words_kernel, dim3((unsigned)(ctas < most ? ctas : most)), dim3(256), 0, ctx->stream, m, p->B));
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
