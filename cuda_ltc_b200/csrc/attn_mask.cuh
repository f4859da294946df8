// Dense keep-masks in the tensor-pipe kernels.  A thread owns one row of a score tile (one query, or one key of the
// transposed tiles) and needs the mask value of each of its columns.  Read column by column from the caller's fp32 mask,
// every load of a warp touches 32 different lines, and every head and every pass reads the mask again: 17 of the 25 us
// of a B16 H4 S200 forward.  So a call packs the mask once into bits (attn_mask.cu), row words and column words, and a
// thread needs one word per 32 columns, loaded before the wait for the step's scores.  A call whose workspace has no
// room for the words (they are part of what ltca_attn_workspace_bytes asks for) votes them together step by step.
#pragma once

#include "host_common.h"
#include "sm100_ptx.cuh"

namespace ltca {

struct MaskArgs {
    const float* dense;            // [B, Sq, Sk], or null: no mask
    const uint32_t* by_query;      // [B, Sq, nk]: bit c of word w = key 32 w + c; null: not packed
    const uint32_t* by_key;        // [B, Sk, nq]: bit c of word w = query 32 w + c
    int Sq, Sk, nk, nq;
};

// Bytes of both forms for a call with a dense mask, and the launch that fills them.
inline size_t mask_words_bytes(const ltca_attn_params* p) {
    if (!p->keep_mask) return 0;
    const size_t nk = (size_t)(p->Sk + 31) / 32, nq = (size_t)(p->Sq + 31) / 32;
    return align_up((size_t)p->B * ((size_t)p->Sq * nk + (size_t)p->Sk * nq) * 4, 256);
}
int pack_mask_words(ltca_ctx* ctx, const ltca_attn_params* p, void* words);
// The words for this call: the context's, where a module call has packed the mask for all its kernels; else packed now
// into the workspace behind its first `used` bytes; null without a mask or without room.
int mask_words_of(ltca_ctx* ctx, const ltca_attn_params* p, size_t used, const void** words);
inline MaskArgs mask_args(const ltca_attn_params* p, const void* words) {
    MaskArgs m;
    m.dense = p->keep_mask;
    m.Sq = p->Sq; m.Sk = p->Sk;
    m.nk = (p->Sk + 31) / 32; m.nq = (p->Sq + 31) / 32;
    m.by_query = p->keep_mask ? static_cast<const uint32_t*>(words) : nullptr;
    m.by_key = m.by_query ? m.by_query + (size_t)p->B * p->Sq * m.nk : nullptr;
    return m;
}

// Packs the dense mask into m's words: one warp per block of 32 queries x 32 keys, blocks first, first + step, ...  Lane l
// reads key l of each query (coalesced); the vote over a query's 32 values is its row word, the values a lane has seen are
// its key's column word.
__device__ __forceinline__ void write_mask_words(const MaskArgs& m, int B, int64_t first, int64_t step) {
    const int lane = threadIdx.x & 31, Sq = m.Sq, Sk = m.Sk, nq = m.nq, nk = m.nk;
    uint32_t* by_query = const_cast<uint32_t*>(m.by_query);
    uint32_t* by_key = const_cast<uint32_t*>(m.by_key);
    for (int64_t w = first; w < (int64_t)B * nq * nk; w += step) {
        const int kw = (int)(w % nk), qw = (int)(w / nk % nq);
        const int64_t b = w / ((int64_t)nk * nq);
        const int q0 = qw * 32, k = kw * 32 + lane;
        const float* src = m.dense + (b * Sq + q0) * Sk + k;
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

// Bit c of the result: key k + c is kept for query q0 + lane (k a multiple of 32).  Whole-warp call.
__device__ __forceinline__ uint32_t mask_bits_of_queries(const MaskArgs& m, int b, int q0, int k) {
    if (!m.dense) return ~0u;
    const int lane = threadIdx.x & 31;
    if (m.by_query) {
        const int q = q0 + lane;
        return (q < m.Sq && k < m.Sk) ? __ldg(m.by_query + ((int64_t)b * m.Sq + q) * m.nk + (k >> 5)) : 0u;
    }
    const float* mask = m.dense + (int64_t)b * m.Sq * m.Sk + k + lane;
    const bool in = k + lane < m.Sk;
    uint32_t mine = 0;
#pragma unroll 1
    for (int r0 = 0; r0 < 32; r0 += 8) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = (in && q0 + r0 + i < m.Sq) ? __ldg(mask + (int64_t)(q0 + r0 + i) * m.Sk) : 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t bits = __ballot_sync(0xffffffffu, v[i] != 0.f);
            if (lane == r0 + i) mine = bits;
        }
    }
    return mine;
}

// Bit c of the result: key kj (this lane's) is kept for query q0 + c (q0 a multiple of 32).
__device__ __forceinline__ uint32_t mask_bits_of_key(const MaskArgs& m, int b, int q0, int kj) {
    if (!m.dense) return ~0u;
    if (kj >= m.Sk || q0 >= m.Sq) return 0u;
    if (m.by_key) return __ldg(m.by_key + ((int64_t)b * m.Sk + kj) * m.nq + (q0 >> 5));
    const float* mask = m.dense + (int64_t)b * m.Sq * m.Sk + kj;
    uint32_t mine = 0;
#pragma unroll 1
    for (int c0 = 0; c0 < 32; c0 += 8)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int q = q0 + c0 + i;
            mine |= (q < m.Sq && __ldg(mask + (int64_t)q * m.Sk) != 0.f ? 1u : 0u) << (c0 + i);
        }
    return mine;
}

}  // namespace ltca
