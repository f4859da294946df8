// Attention forward on the sm_100a tensor pipe.
//
//   O = softmax(mask(scale * Q K^T)) V,   lse = log sum exp of the masked, scaled scores
//
// replaces flashAttentionKernel of the reference (src/ml/flash_attention.cu:18-272): the same
// contract (scale, keep-mask with 0 = hidden, optional score clamp), plus a causal flag and
// per-sequence key lengths, computed as a true online softmax.
//
// Two kernels: attn_fwd_tile_sm100_kernel, a CTA per 128-row query tile (further down), and, for calls of few tiles with
// long keys at head_dim 64, attn_fwd_sm100_kernel:
//   - one CTA per (256 query rows, head, batch): two 128-row query tiles share every K/V tile
//     that TMA brings in, which halves the L2 -> shared traffic per FLOP;
//   - 16 softmax warps: a query row belongs to TWO threads, each owning half of the step's key
//     columns (warps w and w + 8 read the same 32 tensor-memory lanes), so that every scheduler
//     holds four softmax warps and the special-function unit stays busy while other warps load,
//     reduce or wait.  The two threads of a row agree on the row maximum through shared memory;
//     row sums stay private until the epilogue.  Warps 0-3 / 8-11: tile 0, 4-7 / 12-15: tile 1;
//   - warps 16 / 17 issue the tcgen05.mma of tile 0 / 1 (one thread each), warp 18 is the TMA
//     producer.  The control warps give registers up for the softmax warps (setmaxnreg);
//   - S = Q K^T accumulates in tensor memory; the softmax warps read it with tcgen05.ld and
//     release it at once, so the next step's S is computed while this step's exponentials
//     run; P goes back to its OWN tensor-memory columns as packed bf16 (tcgen05.st) and the
//     second contraction O += P V takes it from there; O never leaves tensor memory until the
//     epilogue;
//   - K and V tiles travel through one ring of shared-memory slots in the order
//     K0 V0 K1 V1 ..., each slot guarded by a full/empty mbarrier pair.
// Its keys per step: 128 for a bf16 result, else 64 (the split-P variant), chosen so that everything fits the 512
// tensor-memory columns: S0 S1 (kBN each) | O0 O1 (D each) | P0 P1 (kBN/2 each) | split-P only: Plo0 Plo1 (kBN/2 each)
#include <type_traits>

#include "host_common.h"
#include "attn_mask.cuh"
#include "sm100_ptx.cuh"
#include "trace.cuh"


namespace ltca {

namespace {

constexpr int kBlockM = 128;        // query rows per tile
// Two threads share one query row (each owns half of the step's key columns): 16 softmax warps, four per
// scheduler, row maxima exchanged through shared memory.  (One thread per row, 8 warps, hid no latency.)
constexpr int kRowSplit = 2;
constexpr int kMathWarps = 8 * kRowSplit;
constexpr int kFwdThreads = 32 * (kMathWarps + 4);   // + one warpgroup of control warps
constexpr int kMmaWarp0 = kMathWarps;                // issues the contractions of tile 0 (tile 1: the next warp)
constexpr int kTmaWarp = kMathWarps + 2;
constexpr int kLaunchRegs = 96;     // registers per thread at launch (65536 / threads, rounded down to 8)
constexpr int kCtrlRegs = 32;
constexpr int kMathRegs = 112;
// setmaxnreg can only redistribute what the CTA was launched with; asking for more never returns
static_assert(32 * kMathWarps * kMathRegs + 128 * kCtrlRegs <= kFwdThreads * kLaunchRegs, "register budget");
constexpr uint32_t kTmemCols = 512;

struct FwdArgs {
    int B, H, Sq, Sk;
    int causal, causal_off;
    float scale;            // score scale
    float scale_log2;       // scale * log2(e)
    float clamp_raw;        // score clamp divided by scale (raw QK^T units); +inf when unused
    int use_clamp;
    void* o;
    int64_t o_sb, o_sh, o_ss;
    float* lse;
    MaskArgs mask;
    const int32_t* kv_len;
    uint32_t* status;
};

// The two-tile kernel, head_dim 64.
constexpr int kPairD = 64;
template <bool kSplitP>
struct FwdCfg {
    static constexpr int D = kPairD;
    static constexpr int kBN = kSplitP ? 64 : 128;                 // keys per step
    static constexpr int kQTileBytes = kBlockM * D * 2;
    static constexpr int kKvTileBytes = kBN * D * 2;
    static constexpr int kStages = 8;                              // ring slots
    // tensor-memory columns
    static constexpr int kColS = 0;
    static constexpr int kColO = 2 * kBN;
    static constexpr int kColP = kColO + 2 * D;
    static constexpr int kColPlo = kColP + kBN;
    static_assert(kColPlo + (kSplitP ? kBN : 0) <= 512, "tensor memory overflow");
    // shared memory
    static constexpr int kQOff = 0;
    static constexpr int kRingOff = 2 * kQTileBytes;
    static constexpr int kXchgOff = kRingOff + kStages * kKvTileBytes;   // float [3][2 tiles][2 halves][128]
    static constexpr int kBarOff = kXchgOff + 3 * 2 * 2 * kBlockM * 4;
    // barriers: q_full, kv_full[kStages], kv_empty[kStages], s_full[2], s_free[2], p_full[2], o_done[2],
    // pair[8] (one per pair of warps that share rows), turn[2]
    static constexpr int kNumBars = 1 + 2 * kStages + 8 + 8 + 2;
    static constexpr int kMiscOff = kBarOff + kNumBars * 8;        // tmem base, abort flag
    static constexpr int kBytes = kMiscOff + 16;
    static constexpr int kDynBytes = kBytes + 1024;                // room to align to 1024 B
};

__device__ __forceinline__ float neg_inf() { return __int_as_float(0xff800000); }

// kSplitP: P is written as two bf16 terms (p = hi + lo, 16 mantissa bits in total) and the
// second contraction runs once per term; used when the output is stored as fp32, where the
// 2^-9 rounding of a single bf16 P would be the largest error left.
template <bool kSplitP, bool kMask>
__global__ void __launch_bounds__(kFwdThreads, 1)
attn_fwd_sm100_kernel(const __grid_constant__ CUtensorMap tmap_q,
                      const __grid_constant__ CUtensorMap tmap_k,
                      const __grid_constant__ CUtensorMap tmap_v, const FwdArgs a) {
    using L = FwdCfg<kSplitP>;
    using OutT = typename std::conditional<kSplitP, float, __nv_bfloat16>::type;
    constexpr int D = kPairD, kBN = L::kBN;
    constexpr int kH = kBN / kRowSplit;  // key columns per thread and step
    constexpr int kDH = D / kRowSplit;   // output columns per thread
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));

    const uint32_t q_smem = smem_base + L::kQOff;
    const uint32_t ring_smem = smem_base + L::kRingOff;
    const uint32_t bar_base = smem_base + L::kBarOff;
    auto bar_q_full = [&]() { return bar_base; };
    auto bar_kv_full = [&](int s) { return bar_base + 8u * (1 + s); };
    auto bar_kv_empty = [&](int s) { return bar_base + 8u * (1 + L::kStages + s); };
    auto bar_s_full = [&](int t) { return bar_base + 8u * (1 + 2 * L::kStages + t); };
    auto bar_s_free = [&](int t) { return bar_base + 8u * (3 + 2 * L::kStages + t); };
    auto bar_p_full = [&](int t) { return bar_base + 8u * (5 + 2 * L::kStages + t); };
    auto bar_o_done = [&](int t) { return bar_base + 8u * (7 + 2 * L::kStages + t); };
    auto bar_pair = [&](int t, int wq) { return bar_base + 8u * (9 + 2 * L::kStages + t * 4 + wq); };
    auto bar_turn = [&](int t) { return bar_base + 8u * (17 + 2 * L::kStages + t); };
    float* xchg = reinterpret_cast<float*>(smem_gen + L::kXchgOff);
    volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(smem_gen + L::kMiscOff);
    // misc[0] = tensor-memory base address, misc[1] = abort flag

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int m_block = gridDim.x - 1 - blockIdx.x;     // heavy (late) causal blocks first
    const int h = blockIdx.y;
    const int b = blockIdx.z;

    int kvlen = a.Sk;
    if (a.kv_len) {
        grid_dependency_wait();                // the lengths may come from the kernel before this one
        kvlen = min(max(a.kv_len[b], 0), a.Sk);
    }
    int n_tiles[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        const int q0 = m_block * 2 * kBlockM + t * kBlockM;
        int lim = 0;
        if (q0 < a.Sq) {
            lim = kvlen;
            if (a.causal) lim = min(lim, min(q0 + kBlockM - 1, a.Sq - 1) + a.causal_off + 1);
        }
        n_tiles[t] = lim > 0 ? (lim + kBN - 1) / kBN : 0;
    }
    const int n_max = max(n_tiles[0], n_tiles[1]);

    if (threadIdx.x == 0) {
        mbar_init(bar_q_full(), 1);
        for (int s = 0; s < L::kStages; ++s) {
            mbar_init(bar_kv_full(s), 1);
            mbar_init(bar_kv_empty(s), 2);     // both MMA issuers release a slot
        }
        for (int t = 0; t < 2; ++t) {
            mbar_init(bar_s_full(t), 1);
            mbar_init(bar_s_free(t), 4 * kRowSplit);   // one arrival per softmax warp of the tile
            mbar_init(bar_p_full(t), 4 * kRowSplit);
            mbar_init(bar_o_done(t), 1);
            for (int wq = 0; wq < 4; ++wq) mbar_init(bar_pair(t, wq), 2);
            mbar_init(bar_turn(t), 4 * kRowSplit);
        }
        misc[1] = 0u;
        mbar_fence_init();
    }
    if (warp == kMmaWarp0) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(&misc[0])), kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = misc[0];
    const WaitCtx wc{&misc[1], a.status};
    LTCA_TRACE_DECL(blockIdx.x == 0 && blockIdx.y == 5 && blockIdx.z == 0);
    LTCA_TRACE_EVT(0x01);
    grid_dependency_wait();                    // q, k, v are complete once the kernel before this one has ended

    if (warp >= kMathWarps) {
        reg_dealloc<kCtrlRegs>();
        auto slot_of = [&](int item) { return item % L::kStages; };
        auto phase_of = [&](int item) { return (uint32_t)((item / L::kStages) & 1); };
        if (warp == kTmaWarp) {
            // ------------------------------ TMA producer --------------------------------------
            if (lane == 0 && n_max > 0) {
                tma_prefetch_desc(&tmap_q);
                tma_prefetch_desc(&tmap_k);
                tma_prefetch_desc(&tmap_v);
                mbar_arrive_expect_tx(bar_q_full(), 2u * L::kQTileBytes);
                for (int t = 0; t < 2; ++t)
                    tma_load_4d(q_smem + t * L::kQTileBytes, &tmap_q, bar_q_full(), 0, m_block * 2 * kBlockM + t * kBlockM, h, b);
                bool ok = true;
                for (int j = 0; j < n_max && ok; ++j) {
#pragma unroll
                    for (int which = 0; which < 2; ++which) {     // 0: K_j, 1: V_j
                        const int item = 2 * j + which;
                        const int slot = slot_of(item);
                        ok = ok && mbar_wait(bar_kv_empty(slot), phase_of(item) ^ 1u, wc, 0x10 + which);
                        if (!ok) break;
                        mbar_arrive_expect_tx(bar_kv_full(slot), (uint32_t)L::kKvTileBytes);
                        tma_load_4d(ring_smem + slot * L::kKvTileBytes, which == 0 ? &tmap_k : &tmap_v, bar_kv_full(slot), 0,
                                    j * kBN, h, b);
                    }
                }
            }
        } else if (warp == kMmaWarp0 || warp == kMmaWarp0 + 1) {
            // ------------------------------ MMA issuer of tile t ------------------------------
            const int t = warp - kMmaWarp0;
            if (lane == 0 && n_max > 0) {
                const int n_t = n_tiles[t];
                constexpr uint32_t idesc_qk = make_idesc_bf16(kBlockM, kBN, 0, 0);
                constexpr uint32_t idesc_pv = make_idesc_bf16(kBlockM, D, 0, 1);
                // descriptors are built once; a byte offset inside shared memory adds offset >> 4
                const uint64_t q_desc = make_smem_desc_sw128(q_smem + t * L::kQTileBytes, 16, 1024);
                const uint64_t k_desc = make_smem_desc_sw128(ring_smem, 16, 1024);
                const uint64_t v_desc = make_smem_desc_sw128(ring_smem, kBN * 128, 1024);
                const uint32_t s_tmem = tmem_base + L::kColS + t * kBN;
                const uint32_t o_tmem = tmem_base + L::kColO + t * D;
                const uint32_t p_tmem = tmem_base + L::kColP + t * (kBN / 2);
                const uint32_t plo_tmem = tmem_base + L::kColPlo + t * (kBN / 2);
                auto issue_qk = [&](int slot) {
                    const uint64_t kd = k_desc + (uint64_t)((slot * L::kKvTileBytes) >> 4);
#pragma unroll
                    for (int k = 0; k < D / 16; ++k)
                        mma_ss(s_tmem, q_desc + 2 * k, kd + 2 * k, idesc_qk, k > 0 ? 1u : 0u);
                };
                auto issue_pv = [&](int slot, bool acc) {
                    const uint64_t vd = v_desc + (uint64_t)((slot * L::kKvTileBytes) >> 4);
#pragma unroll
                    for (int k = 0; k < kBN / 16; ++k)
                        mma_ts(o_tmem, p_tmem + k * 8, vd + ((k * 2048) >> 4), idesc_pv,
                               (acc || k > 0) ? 1u : 0u);
                    if constexpr (kSplitP) {
#pragma unroll
                        for (int k = 0; k < kBN / 16; ++k)
                            mma_ts(o_tmem, plo_tmem + k * 8, vd + ((k * 2048) >> 4), idesc_pv, 1u);
                    }
                };

                bool ok = mbar_wait(bar_q_full(), 0, wc, 0x20);
                ok = ok && mbar_wait(bar_kv_full(slot_of(0)), phase_of(0), wc, 0x21);
                if (ok) {
                    tc_fence_after_sync();
                    if (n_t > 0) {
                        issue_qk(slot_of(0));
                        mma_commit(bar_s_full(t));
                    }
                    mma_commit(bar_kv_empty(slot_of(0)));
                }
                for (int j = 0; j < n_max && ok; ++j) {
                    const int item_v = 2 * j + 1, item_k = 2 * j + 2;
                    // S of step j+1 as soon as the softmax warps have taken S of step j
                    if (j + 1 < n_max) {
                        ok = mbar_wait(bar_kv_full(slot_of(item_k)), phase_of(item_k), wc, 0x23);
                        if (ok && j + 1 < n_t) {
                            ok = mbar_wait(bar_s_free(t), (uint32_t)(j & 1), wc, 0x26 + t);
                            if (!ok) break;
                            tc_fence_after_sync();
                            LTCA_TRACE_EVT(0x20 + (j << 8));
                            issue_qk(slot_of(item_k));
                            mma_commit(bar_s_full(t));
                            LTCA_TRACE_EVT(0x22 + (j << 8));
                        }
                        if (!ok) break;
                        mma_commit(bar_kv_empty(slot_of(item_k)));
                    }
                    ok = mbar_wait(bar_kv_full(slot_of(item_v)), phase_of(item_v), wc, 0x22);
                    if (ok && j < n_t) {
                        ok = mbar_wait(bar_p_full(t), (uint32_t)(j & 1), wc, 0x24 + t);
                        if (!ok) break;
                        tc_fence_after_sync();
                        LTCA_TRACE_EVT(0x24 + (j << 8));
                        issue_pv(slot_of(item_v), j > 0);
                        mma_commit(bar_o_done(t));
                        LTCA_TRACE_EVT(0x26 + (j << 8));
                    }
                    if (!ok) break;
                    mma_commit(bar_kv_empty(slot_of(item_v)));
                }
                // everything this thread issued has to be complete before tensor memory is released
                if (ok && n_t > 0) ok = mbar_wait(bar_o_done(t), (uint32_t)((n_t - 1) & 1), wc, 0x28 + t);
            }
        }
    } else {
        // ------------------------------ softmax / correction / epilogue ------------------------
        reg_alloc<kMathRegs>();
        const int t = (warp >> 2) & 1;
        const int half = warp >> 3;          // which part of the key columns (and of the output columns)
        const int wq = warp & 3;
        const int row = wq * 32 + lane;
        const int q0 = m_block * 2 * kBlockM + t * kBlockM;
        const int qi = q0 + row;
        const int n_t = n_tiles[t];
        const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
        const uint32_t tS = tmem_base + lane_base + L::kColS + t * kBN + half * kH;
        const uint32_t tO = tmem_base + lane_base + L::kColO + t * D + half * kDH;
        const uint32_t tP = tmem_base + lane_base + L::kColP + t * (kBN / 2) + half * (kH / 2);
        const uint32_t tPlo = tmem_base + lane_base + L::kColPlo + t * (kBN / 2) + half * (kH / 2);
        const float c2 = a.scale_log2;
        const bool general = kMask || (a.use_clamp != 0);
        // exchange slots: [buffer][tile][half][row]
        auto xslot = [&](int buf, int hf) { return xchg + ((buf * 2 + t) * 2 + hf) * kBlockM + row; };
        uint32_t pair_phase = 0;

        float m_run = neg_inf();
        float l_run = 0.f;
        bool ok = true;
        for (int j = 0; j < n_t; ++j) {
            uint32_t keep[kH / 32];              // dense mask of this thread's columns
#pragma unroll
            for (int w = 0; w < kH / 32; ++w)
                keep[w] = kMask ? mask_bits_of_queries(a.mask, b, q0 + wq * 32, j * kBN + half * kH + 32 * w) : ~0u;
            ok = mbar_wait_warp(bar_s_full(t), (uint32_t)(j & 1), wc, 0x30 + t);
            if (!ok) break;
            tc_fence_after_sync();
            LTCA_TRACE_EVT(0x10 + (j << 8));
            uint32_t su[kH];
#pragma unroll
            for (int c0 = 0; c0 < kH; c0 += 32)
                tmem_ld32(tS + c0, reinterpret_cast<uint32_t(&)[32]>(su[c0]));
            tmem_wait_ld();
            // S is in registers: the next step's Q K^T may overwrite it
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_s_free(t));
            LTCA_TRACE_EVT(0x11 + (j << 8));
#define S_(c) __uint_as_float(su[(c)])
            const int k0 = j * kBN;
            const bool edge = (k0 + kBN > kvlen) || (a.causal && (k0 + kBN - 1 > q0 + a.causal_off));
            if (general) {
                int lim = kvlen;
                if (a.causal) lim = min(lim, qi + a.causal_off + 1);
                lim -= k0 + half * kH;                  // own columns c < lim are visible
#pragma unroll
                for (int c = 0; c < kH; ++c) {
                    float v = S_(c);
                    if (a.use_clamp) v = fminf(v, a.clamp_raw);
                    const bool vis = c < lim && (keep[c / 32] >> (c % 32) & 1u);
                    su[c] = __float_as_uint(vis ? v : neg_inf());
                }
            } else if (edge) {
                // causal diagonal or end of the keys, no dense mask: a select per column, no branches
                int lim = kvlen;
                if (a.causal) lim = min(lim, qi + a.causal_off + 1);
                lim -= k0 + half * kH;
#pragma unroll
                for (int c = 0; c < kH; ++c) su[c] = (c < lim) ? su[c] : 0xff800000u;
            }
            float mx[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) mx[i] = fmaxf(S_(2 * i), S_(2 * i + 1));
#pragma unroll
            for (int c = 8; c < kH; c += 8)
#pragma unroll
                for (int i = 0; i < 4; ++i) mx[i] = fmax3(mx[i], S_(c + 2 * i), S_(c + 2 * i + 1));
            float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            {
                // the row's other half: both threads publish, meet, and read each other's maximum
                *xslot(j & 1, half) = mt;
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_pair(t, wq));
                ok = mbar_wait_warp(bar_pair(t, wq), pair_phase, wc, 0x3a);
                pair_phase ^= 1u;
                if (!ok) break;
                mt = fmaxf(mt, *xslot(j & 1, half ^ 1));
            }
            LTCA_TRACE_EVT(0x12 + (j << 8));

            // Lazy rescale: keep the stale maximum while the new one exceeds it by less than
            // 2^8 in the exponent; P stays below 256 and fp32 sums keep their accuracy.
            float factor = 1.0f;
            bool need = false;
            if (j == 0) {
                m_run = mt;
            } else if ((mt - m_run) * c2 > 8.0f) {
                factor = fast_exp2((m_run - mt) * c2);
                m_run = mt;
                need = true;
            }
            bool o_waited = (j == 0);
            if (j > 0 && __any_sync(0xffffffffu, need)) {
                ok = mbar_wait_warp(bar_o_done(t), (uint32_t)((j - 1) & 1), wc, 0x32 + t);
                if (!ok) break;
                o_waited = true;
                tc_fence_after_sync();
#pragma unroll
                for (int c0 = 0; c0 < kDH; c0 += 32) {
                    uint32_t o[32];
                    tmem_ld32(tO + c0, o);
                    tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * factor);
                    tmem_st32(tO + c0, o);
                }
                l_run *= factor;
            }
            // One-time delay: tile 1 starts its first exponentials when tile 0 has finished its own, so that from
            // then on one tile exponentiates while the other loads its scores, finds its maxima and talks to the
            // barriers.  (Strict turn-taking at every step was slower.)
            if (t == 1 && j == 0 && n_tiles[0] > 0) {
                ok = mbar_wait_warp(bar_turn(0), 0, wc, 0x3e);
                if (!ok) break;
            }
            LTCA_TRACE_EVT(0x15 + (j << 8));
            const float m_safe = (m_run == neg_inf()) ? 0.f : m_run;
            const float mneg = -m_safe * c2;
            float sum0 = 0.f, sum1 = 0.f, sum2 = 0.f, sum3 = 0.f;
#pragma unroll
            for (int ch = 0; ch < kH / 32; ++ch) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int cc = 0; cc < 32; cc += 4) {
                    const int c = ch * 32 + cc;
                    const float p0 = fast_exp2(fmaf(S_(c), c2, mneg));
                    const float p1 = fast_exp2(fmaf(S_(c + 1), c2, mneg));
                    const float p2 = fast_exp2(fmaf(S_(c + 2), c2, mneg));
                    const float p3 = fast_exp2(fmaf(S_(c + 3), c2, mneg));
                    sum0 += p0; sum1 += p1; sum2 += p2; sum3 += p3;
                    const uint32_t h01 = pack_bf16x2(p0, p1), h23 = pack_bf16x2(p2, p3);
                    hi[cc / 2] = h01;
                    hi[cc / 2 + 1] = h23;
                    if constexpr (kSplitP) {
                        lo[cc / 2] = pack_bf16x2(p0 - __uint_as_float(h01 << 16),
                                                 p1 - __uint_as_float(h01 & 0xffff0000u));
                        lo[cc / 2 + 1] = pack_bf16x2(p2 - __uint_as_float(h23 << 16),
                                                     p3 - __uint_as_float(h23 & 0xffff0000u));
                    }
                }
                if (ch == 0 && !o_waited) {
                    // P of the previous step must have been consumed before it is overwritten
                    ok = mbar_wait_warp(bar_o_done(t), (uint32_t)((j - 1) & 1), wc, 0x36 + t);
                    if (!ok) break;
                }
                tmem_st16(tP + ch * 16, hi);
                if constexpr (kSplitP) tmem_st16(tPlo + ch * 16, lo);
            }
            if (!ok) break;
            if (t == 0 && j == 0) {
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_turn(t));
            }
            l_run += (sum0 + sum1) + (sum2 + sum3);
            LTCA_TRACE_EVT(0x13 + (j << 8));
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_p_full(t));
            LTCA_TRACE_EVT(0x14 + (j << 8));
#undef S_
        }

        // epilogue: O / l and lse; the row sum is the total of the two halves
        if (ok && q0 < a.Sq) {
            float inv = 0.f;
            float lse = neg_inf();
            if (n_t > 0) {
                {
                    *xslot(2, half) = l_run;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_pair(t, wq));
                    ok = mbar_wait_warp(bar_pair(t, wq), pair_phase, wc, 0x3b);
                    if (ok) l_run += *xslot(2, half ^ 1);
                }
                ok = ok && mbar_wait_warp(bar_o_done(t), (uint32_t)((n_t - 1) & 1), wc, 0x34 + t);
                tc_fence_after_sync();
                if (l_run > 0.f) {
                    inv = 1.0f / l_run;
                    lse = m_run * a.scale + __logf(l_run);
                }
            }
            OutT* orow = reinterpret_cast<OutT*>(a.o) + b * a.o_sb + h * a.o_sh + (int64_t)qi * a.o_ss +
                         half * kDH;
#pragma unroll
            for (int c0 = 0; c0 < kDH; c0 += 32) {
                uint32_t o[32];
                if (n_t > 0 && ok) {
                    tmem_ld32(tO + c0, o);
                    tmem_wait_ld();
                } else {
#pragma unroll
                    for (int c = 0; c < 32; ++c) o[c] = 0u;
                }
                if (qi < a.Sq) {
                    if constexpr (sizeof(OutT) == 2) {
                        uint4* dst = reinterpret_cast<uint4*>(orow + c0);
#pragma unroll
                        for (int v = 0; v < 4; ++v) {
                            uint4 w;
                            w.x = pack_bf16x2(__uint_as_float(o[8 * v + 0]) * inv, __uint_as_float(o[8 * v + 1]) * inv);
                            w.y = pack_bf16x2(__uint_as_float(o[8 * v + 2]) * inv, __uint_as_float(o[8 * v + 3]) * inv);
                            w.z = pack_bf16x2(__uint_as_float(o[8 * v + 4]) * inv, __uint_as_float(o[8 * v + 5]) * inv);
                            w.w = pack_bf16x2(__uint_as_float(o[8 * v + 6]) * inv, __uint_as_float(o[8 * v + 7]) * inv);
                            dst[v] = w;
                        }
                    } else {
                        float4* dst = reinterpret_cast<float4*>(orow + c0);
#pragma unroll
                        for (int v = 0; v < 8; ++v)
                            dst[v] = make_float4(__uint_as_float(o[4 * v + 0]) * inv,
                                                 __uint_as_float(o[4 * v + 1]) * inv,
                                                 __uint_as_float(o[4 * v + 2]) * inv,
                                                 __uint_as_float(o[4 * v + 3]) * inv);
                    }
                }
            }
            if (half == 0 && a.lse && qi < a.Sq) a.lse[((int64_t)b * a.H + h) * a.Sq + qi] = lse;
        }
    }

    // ------------------------------ tear-down -------------------------------------------------
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kMmaWarp0) {
        __syncwarp();
        if (misc[1]) __nanosleep(200000);    // aborted: give copies and MMAs in flight time to land
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// ---------------------------------------------------------------------------------------------
// One-tile kernel: a CTA is ONE 128-row query tile, four CTAs to an SM at head_dim 64, two at 128.
//
// Softmax warps of several tiles share every scheduler, as latencies between the two contractions of a step need (a step
// leaves a tile's warps idle for about 1300 cycles while P is multiplied and the next scores are formed), and the tiles
// are independent work: a causal tile of two key steps leaves after two and the next takes its place, and a call is
// dealt out in pieces of 128 rows.  A persistent kernel with four tiles on one key stream, which this replaces, made the
// early tiles of 512 causal rows wait for the late ones' keys: B64 H8 S512 causal 68 us against 46 now, B8 H16 S4096 causal
// 440 against 365.  What it pays is a set-up per tile and a K/V read per tile from L2 (20 bytes per clock and SM).
//   - warps 0-3 softmax, one row per thread, head_dim keys per step; tensor memory S [0, D), O [D, 2 D).  At head_dim 128 a
//     thread so holds 128 scores in its 216 registers and two warps share a scheduler; two threads per row, 64 scores each,
//     had four of them but met once a step to agree on the row's maximum (B8 H16 S4096 causal 568 us, one per row 525).
//     Two score buffers and 64 keys a step there overlap a step's products with the softmax before it (ragged causal B4 H16 S1500
//     40.5 -> 37.0 us), but take P relative to a maximum over half as many keys: the error against 64 bits grows by 1 % at inputs
//     of unit variance, and B16 H8 S256 causal takes 8.5 us and not 8.2.
//     fp32 results at head_dim 128 have two threads per row (warps 0-7), which share the work of P's second term, and the
//     halves of P below are one thread's each (B8 H16 S2048 causal 325 -> 319 us).  Not with a mask, whose words no longer fit
//     their 104 registers: what is spilled goes out to L2, since the tiles leave an SM next to no L1 (masked B64 H8 S200 126 us
//     with two threads per row, 97 with one; B4 H16 S1500 298 and 247);
//   - P overwrites the first half of S, its second bf16 term (kSplitP: results stored as fp32) the other half.  It is handed
//     to the contraction in two halves of the keys, so that the first products run under the second half's exponentials
//     (B8 H16 S4096 D64, not causal: one hand-over 721 us, two 698);
//   - a step's V slot is returned before the next S is issued: with two slots at head_dim 128 the next V then arrives a
//     contraction earlier (B1 H8 S4096 76 -> 65);
//   - of the last four warps one issues the contractions and one is the TMA producer (the others complete the
//     warpgroup that gives registers up);
//   - the result leaves through the Q slot (fp32: and the ring) and a TMA store.
//
// kTeams > 1 is the form for a context whose SMs are limited (ltca_ctx_set_sm_limit): CTAs of a tile each settle on every
// SM that has room, so there one CTA per SM holds the same number of tiles side by side, a team of warps each with its own
// ring, barriers and accumulators, and the teams take tiles from a counter until there are none left.  A tile's
// arithmetic, and with it every bit of the result, is that of the plain form; a team waits for its slowest warp between
// tiles and loads nothing of the next tile before that.  On 16 SMs B8 H16 S4096 causal takes 3.72 ms, 402 us scaled to 148,
// where the plain form takes 365 there (four tiles that start together stay in step); on 132 SMs 473 us, B8 H16 S1024
// causal 43, B64 H8 S512 causal 56.
// ---------------------------------------------------------------------------------------------
template <int D, bool kSplitP, bool kMask>
struct TileCfg {
    static constexpr int kBN = D;                                  // keys per step
    static constexpr int kRowSplit = D == 128 && kSplitP && !kMask ? 2 : 1;    // threads per row
    static constexpr int kCols = kBN / kRowSplit;                  // score columns of a thread
    static constexpr int kMathWarps = 4 * kRowSplit;
    static constexpr int kThreads = 32 * (kMathWarps + 4);
    static constexpr int kCtas = D == 64 ? 4 : 2;                  // per SM
    static constexpr int kLaunchRegs = 65536 / (kCtas * kThreads) / 8 * 8;
    static constexpr int kMathRegs = kCols == 64 ? 104 : 216, kCtrlRegs = D == 64 ? 24 : kCols == 64 ? 32 : 40;
    static_assert(32 * kMathWarps * kMathRegs + 128 * kCtrlRegs <= kThreads * kLaunchRegs, "register budget");
    static constexpr int kBlocks = D / 64;                         // 128-byte column blocks of a row
    static constexpr int kQBytes = kBlockM * D * 2;
    static constexpr int kKvBytes = kBN * D * 2;
    static constexpr int kStages = D == 64 ? 4 : 2;                // ring slots: K0 V0 K1 V1 ...
    static constexpr int kRingOff = kQBytes;
    static constexpr int kXchgOff = kRingOff + kStages * kKvBytes; // row maxima [2 buffers][2 halves][128], row sums [2][128]
    static constexpr int kBarOff = kXchgOff + (kRowSplit > 1 ? 3 * 2 * kBlockM * 4 : 0);
    static constexpr int kNumBars = 1 + 2 * kStages + 4 + 4;       // q_full, kv_full[], kv_empty[], s_full, p_full[2], staged, pair[4]
    static constexpr int kMiscOff = kBarOff + kNumBars * 8;        // tmem base, abort flag, a team's next tile
    static constexpr int kDynBytes = kMiscOff + 32 + 1024;
    static_assert(kCtas * (kDynBytes + 1024) <= 228 * 1024, "shared memory");
    static constexpr int kTeamBytes = (kMiscOff + 32 + 1023) / 1024 * 1024;
    static constexpr int kTeamsDynBytes = kCtas * kTeamBytes + 1024;
    static_assert(kTeamsDynBytes <= 227 * 1024, "shared memory");
    static constexpr uint32_t kTmemCols = 2 * D;
};

template <int D, bool kSplitP, bool kMask, int kTeams>
__global__ void __launch_bounds__(TileCfg<D, kSplitP, kMask>::kThreads * kTeams, kTeams > 1 ? 1 : TileCfg<D, kSplitP, kMask>::kCtas)
attn_fwd_tile_sm100_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                           const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_o, const FwdArgs a,
                           const ItemGrid items) {
    using L = TileCfg<D, kSplitP, kMask>;
    // (the teams share the registers and the tensor memory that as many CTAs of the plain form have on an SM)
    static_assert(kTeams == 1 || kTeams == L::kCtas, "one CTA or an SM's worth of them");
    constexpr int kBN = L::kBN, kRS = L::kRowSplit, kC = L::kCols, kMmaWarp = L::kMathWarps, kTmaWarp = L::kMathWarps + 1;
    extern __shared__ uint8_t smem_raw[];
    // (through a shuffle: what follows from it is then known to be the same in a whole warp, which the operands of the
    // tensor-core instructions have to be)
    const int team = kTeams > 1 ? __shfl_sync(0xffffffffu, (int)threadIdx.x / L::kThreads, 0) : 0, tid = threadIdx.x - team * L::kThreads;
    const uint32_t smem_cta = (smem_u32(smem_raw) + 1023u) & ~1023u, smem_base = smem_cta + team * L::kTeamBytes;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t ring = smem_base + L::kRingOff;
    const uint32_t bar_base = smem_base + L::kBarOff;
    auto bar_kv_full = [&](int s) { return bar_base + 8u * (1 + s); };
    auto bar_kv_empty = [&](int s) { return bar_base + 8u * (1 + L::kStages + s); };
    const uint32_t bar_q_full = bar_base, bar_s_full = bar_base + 8u * (1 + 2 * L::kStages), bar_p_full = bar_s_full + 8,
                   bar_staged = bar_s_full + 24, bar_pair0 = bar_s_full + 32;
    volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(smem_gen + L::kMiscOff);
    volatile uint32_t* misc_cta = reinterpret_cast<volatile uint32_t*>(smem_raw + (smem_cta - smem_u32(smem_raw)) + L::kMiscOff);
    const int warp = kTeams > 1 ? __shfl_sync(0xffffffffu, tid >> 5, 0) : tid >> 5, lane = tid & 31;

    if (tid == 0) {
        mbar_init(bar_q_full, 1);
        for (int s = 0; s < L::kStages; ++s) { mbar_init(bar_kv_full(s), 1); mbar_init(bar_kv_empty(s), 1); }
        mbar_init(bar_s_full, 1);
        mbar_init(bar_p_full, L::kMathWarps);  // the first half of P, and O at its scale in all columns
        mbar_init(bar_p_full + 8u, 4);
        mbar_init(bar_staged, L::kMathWarps);
        for (int i = 0; i < 4; ++i) mbar_init(bar_pair0 + 8u * i, 2);
        misc[1] = 0u;
        mbar_fence_init();
    }
    if (warp == kMmaWarp && team == 0) { tmem_alloc(smem_u32(const_cast<uint32_t*>(&misc[0])), kTeams * L::kTmemCols); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = misc_cta[0] + team * L::kTmemCols;
    const WaitCtx wc{&misc[1], a.status};
    grid_dependency_wait();                    // the operands are complete once the kernel before this one has ended

    // The tile at hand, and what of this team's barriers and ring went before it: key steps, and tiles with any.
    int h, b, q0, kvlen, n_t = 0, steps = 0, tiles = 0;
    bool started = false;
    auto slot_of = [](int e) { return e % L::kStages; };
    auto phase_of = [](int e) { return (uint32_t)((e / L::kStages) & 1); };
    auto take = [&](int rank, int nblk) {
        q0 = (nblk - 1 - rank) * kBlockM;      // heavy (late) causal tiles first
        kvlen = a.Sk;
        if (a.kv_len) kvlen = min(max(a.kv_len[b], 0), a.Sk);
        int lim = kvlen;
        if (a.causal) lim = min(lim, min(q0 + kBlockM - 1, a.Sq - 1) + a.causal_off + 1);
        n_t = lim > 0 ? (lim + kBN - 1) / kBN : 0;
    };
    // Whole-team call: false when there is no further tile (or a wait of this team gave up).
    auto next_tile = [&]() {
        int rank;
        if constexpr (kTeams > 1) {
            auto team_sync = [&]() {
                __syncwarp();
                asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(L::kThreads) : "memory");
            };
            steps = (steps + n_t) & 1023;      // (only their place in the ring and their parities matter)
            tiles = (tiles + (n_t > 0 ? 1 : 0)) & 1;
            tc_fence_before_sync();
            team_sync();                       // every warp is done with the tile before
            if (tid == 0) {
                // The first tiles are dealt out there and back, so that a CTA gets heavy and light ones; then the counter.
                const int dealt = team * gridDim.x + ((team & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
                int item = items.n_items;
                if (!misc[1]) item = started ? (int)(kTeams * gridDim.x) + atomicAdd(items.counters, 1) : dealt;
                started = true;
                if (item < items.n_items) {
                    sched_item(items, item, rank, h, b);
                    take(rank, items.nblk);
                    misc[3] = (uint32_t)q0; misc[4] = (uint32_t)h; misc[5] = (uint32_t)b;
                    misc[6] = (uint32_t)kvlen; misc[7] = (uint32_t)n_t;
                }
                misc[2] = item < items.n_items ? 1u : 0u;
            }
            team_sync();
            tc_fence_after_sync();
            if (!misc[2]) return false;
            q0 = (int)misc[3]; h = (int)misc[4]; b = (int)misc[5]; kvlen = (int)misc[6]; n_t = (int)misc[7];
        } else {
            sched_block(rank, h, b, items.group);
            take(rank, (int)gridDim.x);
        }
        return true;
    };

    if (warp >= L::kMathWarps) {
        reg_dealloc<L::kCtrlRegs>();
        do {
            if (!next_tile()) break;
            const int e0 = 2 * steps;                                  // ring entries that went before
            if (warp == kTmaWarp && lane == 0 && n_t > 0) {
                mbar_arrive_expect_tx(bar_q_full, (uint32_t)L::kQBytes);
                for (int kb = 0; kb < L::kBlocks; ++kb) tma_load_4d(smem_base + kb * (kBlockM * 128), &tmap_q, bar_q_full, kb * 64, q0, h, b);
                bool ok = true;
                for (int e = 0; e < 2 * n_t && ok; ++e) {              // K0 V0 K1 V1 ...
                    const int s = slot_of(e0 + e);
                    ok = mbar_wait(bar_kv_empty(s), phase_of(e0 + e) ^ 1u, wc, 0x50);
                    if (!ok) break;
                    mbar_arrive_expect_tx(bar_kv_full(s), (uint32_t)L::kKvBytes);
                    for (int kb = 0; kb < L::kBlocks; ++kb)
                        tma_load_4d(ring + s * L::kKvBytes + kb * (kBN * 128), (e & 1) ? &tmap_v : &tmap_k, bar_kv_full(s), kb * 64,
                                    (e >> 1) * kBN, h, b);
                }
            } else if (warp == kMmaWarp && lane == 0 && n_t > 0) {
                constexpr uint32_t idesc_qk = make_idesc_bf16(kBlockM, kBN, 0, 0);
                constexpr uint32_t idesc_pv = make_idesc_bf16(kBlockM, D, 0, 1);
                const uint32_t q_lo = smem_desc_lo(smem_base, 16), k_lo = smem_desc_lo(ring, 16), v_lo = smem_desc_lo(ring, kBN * 128);
                auto issue_qk = [&](int s) {
    #pragma unroll
                    for (int k = 0; k < D / 16; ++k)
                        mma_ss_lo(tmem_base, q_lo + (k / 4) * (kBlockM * 8) + (k % 4) * 2,
                                  k_lo + ((s * L::kKvBytes) >> 4) + (k / 4) * (kBN * 8) + (k % 4) * 2, idesc_qk, k > 0 ? 1u : 0u);
                };
                auto issue_pv = [&](int s, int part, bool first) {     // one half of the step's keys
                    constexpr int kSteps = kBN / 32;
                    const uint32_t vd = v_lo + ((s * L::kKvBytes) >> 4);
    #pragma unroll
                    for (int t = 0; t < (kSplitP ? 2 : 1); ++t)
    #pragma unroll
                        for (int k = 0; k < kSteps; ++k)
                            mma_ts_lo(tmem_base + kBN, tmem_base + (kBN / 2) * t + (part * kSteps + k) * 8, vd + 128 * (part * kSteps + k),
                                      idesc_pv, (!first || t > 0 || k > 0) ? 1u : 0u);
                };
                bool ok = mbar_wait(bar_q_full, (uint32_t)(tiles & 1), wc, 0x51) && mbar_wait(bar_kv_full(slot_of(e0)), phase_of(e0), wc, 0x52);
                if (ok) {
                    tc_fence_after_sync();
                    issue_qk(slot_of(e0));
                    mma_commit(bar_kv_empty(slot_of(e0)));
                    mma_commit(bar_s_full);
                }
                for (int j = 0; j < n_t && ok; ++j) {
                    const int e_v = e0 + 2 * j + 1, e_k = e0 + 2 * j + 2;
                    const bool more = j + 1 < n_t;
                    ok = mbar_wait(bar_kv_full(slot_of(e_v)), phase_of(e_v), wc, 0x53);
                    if (more) ok = ok && mbar_wait(bar_kv_full(slot_of(e_k)), phase_of(e_k), wc, 0x54);
                    for (int part = 0; part < 2 && ok; ++part) {
                        ok = mbar_wait(bar_p_full + 8u * part, (uint32_t)((steps + j) & 1), wc, 0x55);
                        if (!ok) break;
                        tc_fence_after_sync();
                        issue_pv(slot_of(e_v), part, j == 0 && part == 0);
                    }
                    if (!ok) break;
                    mma_commit(bar_kv_empty(slot_of(e_v)));
                    if (more) {
                        issue_qk(slot_of(e_k));
                        mma_commit(bar_kv_empty(slot_of(e_k)));
                    }
                    mma_commit(bar_s_full);                            // S of step j + 1 ready, O holds steps 0 .. j
                }
            }
        } while (kTeams > 1);
    } else {
        reg_alloc<L::kMathRegs>();
        const int wq = warp & 3, half = kRS > 1 ? warp >> 2 : 0;
        const int row = wq * 32 + lane;
        const uint32_t lane_base = (uint32_t)(wq * 32) << 16;
        const uint32_t tS = tmem_base + lane_base + half * kC, tO = tmem_base + lane_base + kBN + half * (D / kRS);
        const uint32_t tP = tmem_base + lane_base + half * (kC / 2), tPlo = tP + kBN / 2;
        float* xchg = reinterpret_cast<float*>(smem_gen + L::kXchgOff);
        auto xslot = [&](int buf, int hf) { return xchg + (buf * 2 + hf) * kBlockM + row; };
        // the row's other thread has published its value too
        uint32_t pair_phase = 0;
        auto meet = [&]() {
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_pair0 + 8u * wq);
            const bool met = mbar_wait_warp(bar_pair0 + 8u * wq, pair_phase, wc, 0x59);
            pair_phase ^= 1u;
            return met;
        };
        const float c2 = a.scale_log2;
        const bool general = kMask || (a.use_clamp != 0);
        do {
            if (!next_tile()) break;
            const int s_full0 = steps + tiles;                         // score tiles that went before (one more than steps each)
            // per row: number of visible keys; per tile: the first step that needs masking at all
            int lim_row = kvlen, je = n_t;
            if (a.causal) lim_row = min(lim_row, q0 + row + a.causal_off + 1);
            if (kvlen % kBN) je = min(je, kvlen / kBN);
            if (a.causal) {
                const int v = q0 + a.causal_off - (kBN - 1);           // step j is cut by the diagonal when j * kBN > v
                je = min(je, v < 0 ? 0 : v / kBN + 1);
            }
            float m_run = neg_inf(), l_run = 0.f;
            bool ok = true;
            for (int j = 0; j < n_t; ++j) {
                uint32_t keep[kC / 32];                                // dense mask of this thread's columns
    #pragma unroll
                for (int w = 0; w < kC / 32; ++w)
                    keep[w] = kMask ? mask_bits_of_queries(a.mask, b, q0 + wq * 32, j * kBN + half * kC + 32 * w) : ~0u;
                ok = mbar_wait_warp(bar_s_full, (uint32_t)((s_full0 + j) & 1), wc, 0x56);
                if (!ok) break;
                tc_fence_after_sync();
                uint32_t su[kC];
    #pragma unroll
                for (int c = 0; c < kC; c += 32) tmem_ld32(tS + c, reinterpret_cast<uint32_t(&)[32]>(su[c]));
                tmem_wait_ld();
    #pragma unroll
                for (int c = 0; c < kC; c += 32) tmem_ld_fence(reinterpret_cast<uint32_t(&)[32]>(su[c]));
    #define S_(c) __uint_as_float(su[(c)])
                const int lim_c = lim_row - j * kBN - half * kC;       // own columns c < lim_c are visible
                if (general) {
    #pragma unroll
                    for (int c = 0; c < kC; ++c) {
                        float v = S_(c);
                        if (a.use_clamp) v = fminf(v, a.clamp_raw);
                        const bool vis = c < lim_c && (keep[c / 32] >> (c % 32) & 1u);
                        su[c] = __float_as_uint(vis ? v : neg_inf());
                    }
                } else if (j >= je) {
    #pragma unroll
                    for (int c = 0; c < kC; ++c) su[c] = (c < lim_c) ? su[c] : 0xff800000u;
                }
                float mx[4];
    #pragma unroll
                for (int i = 0; i < 4; ++i) mx[i] = fmaxf(S_(2 * i), S_(2 * i + 1));
    #pragma unroll
                for (int c = 8; c < kC; c += 8)
    #pragma unroll
                    for (int i = 0; i < 4; ++i) mx[i] = fmax3(mx[i], S_(c + 2 * i), S_(c + 2 * i + 1));
                float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
                if constexpr (kRS > 1) {
                    // Behind this meeting both halves of S are in registers: P may overwrite them.  The columns that this warp
                    // writes were read by the row's other warp, hence the fences of a hand-over of tensor memory.
                    *xslot(j & 1, half) = mt;
                    tc_fence_before_sync();
                    ok = meet();
                    if (!ok) break;
                    tc_fence_after_sync();
                    mt = fmaxf(mt, *xslot(j & 1, half ^ 1));
                }
                // lazy rescale, as in the kernels above
                float factor = 1.0f;
                bool need = false;
                if (j == 0) {
                    m_run = mt;
                } else if ((mt - m_run) * c2 > 8.0f) {
                    factor = fast_exp2((m_run - mt) * c2);
                    m_run = mt;
                    need = true;
                }
                if (j > 0 && __any_sync(0xffffffffu, need)) {
    #pragma unroll 1
                    for (int c0 = 0; c0 < D / kRS; c0 += 16) {
                        uint32_t o[16];
                        tmem_ld16(tO + c0, o);
                        tmem_wait_ld();
    #pragma unroll
                        for (int c = 0; c < 16; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * factor);
                        tmem_st16(tO + c0, o);
                    }
                    l_run *= factor;
                }
                if constexpr (kRS > 1) {
                    // The product of P's first half adds to every column of O, so it waits for the warps that hold the
                    // second half of P and of O's columns too.
                    if (half == 1) {
                        tmem_wait_st();
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_p_full);
                    }
                }
                const float m_safe = (m_run == neg_inf()) ? 0.f : m_run;
                const f32x2 c2_2 = pair(c2, c2), mneg_2 = pair(-m_safe * c2, -m_safe * c2);
                f32x2 sum01 = pair(0.f, 0.f), sum23 = sum01;
    #pragma unroll
                for (int ch = 0; ch < kC / 32; ++ch) {
                    uint32_t hi[16], lo[16];
    #pragma unroll
                    for (int cc = 0; cc < 32; cc += 4) {
                        const int c = ch * 32 + cc;
                        const float2 x01 = halves(fma2(pair(S_(c), S_(c + 1)), c2_2, mneg_2));
                        const float2 x23 = halves(fma2(pair(S_(c + 2), S_(c + 3)), c2_2, mneg_2));
                        const float p0 = fast_exp2(x01.x), p1 = fast_exp2(x01.y), p2 = fast_exp2(x23.x), p3 = fast_exp2(x23.y);
                        sum01 = add2(sum01, pair(p0, p1));
                        sum23 = add2(sum23, pair(p2, p3));
                        const uint32_t h01 = pack_bf16x2(p0, p1), h23 = pack_bf16x2(p2, p3);
                        hi[cc / 2] = h01;
                        hi[cc / 2 + 1] = h23;
                        if constexpr (kSplitP) {
                            lo[cc / 2] = pack_bf16x2(p0 - __uint_as_float(h01 << 16), p1 - __uint_as_float(h01 & 0xffff0000u));
                            lo[cc / 2 + 1] = pack_bf16x2(p2 - __uint_as_float(h23 << 16), p3 - __uint_as_float(h23 & 0xffff0000u));
                        }
                    }
                    tmem_st16(tP + ch * 16, hi);                       // P over S (all of S is in registers)
                    if constexpr (kSplitP) tmem_st16(tPlo + ch * 16, lo);
                    constexpr int kHalf = kBN / 64;                    // pieces in one half of the step's keys
                    if (ch % kHalf == kHalf - 1) {                     // their contraction may begin
                        tmem_wait_st();
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(bar_p_full + 8u * (half + ch / kHalf));
                    }
                }
                const float2 s01 = halves(sum01), s23 = halves(sum23);
                l_run += (s01.x + s01.y) + (s23.x + s23.y);
    #undef S_
            }
            const int qi = q0 + row;
            const int64_t stat = ((int64_t)b * a.H + h) * a.Sq + qi;
            if (n_t > 0) {
                if constexpr (kRS > 1) {
                    *xslot(2, half) = l_run;
                    ok = ok && meet();
                    if (ok) l_run += *xslot(2, half ^ 1);
                }
                ok = ok && mbar_wait_warp(bar_s_full, (uint32_t)((s_full0 + n_t) & 1), wc, 0x57);
                tc_fence_after_sync();
                float inv = 0.f, lse = neg_inf();
                if (l_run > 0.f) {
                    inv = 1.0f / l_run;
                    lse = m_run * a.scale + __logf(l_run);
                }
                if (ok) {
                    // every operand has been read: Q's slot (and the ring) take the result as 128-byte-swizzled boxes
    #pragma unroll
                    for (int ob = 0; ob < D / 64 / kRS; ++ob) {
                        uint32_t o[64];
                        tmem_ld32(tO + ob * 64, reinterpret_cast<uint32_t(&)[32]>(o[0]));
                        tmem_ld32(tO + ob * 64 + 32, reinterpret_cast<uint32_t(&)[32]>(o[32]));
                        tmem_wait_ld();
                        tmem_ld_fence(reinterpret_cast<uint32_t(&)[32]>(o[0]));
                        tmem_ld_fence(reinterpret_cast<uint32_t(&)[32]>(o[32]));
    #pragma unroll
                        for (int v = 0; v < (kSplitP ? 16 : 8); ++v) {
                            uint4 w;
                            if constexpr (kSplitP) {
                                w = make_uint4(__float_as_uint(__uint_as_float(o[4 * v]) * inv),
                                               __float_as_uint(__uint_as_float(o[4 * v + 1]) * inv),
                                               __float_as_uint(__uint_as_float(o[4 * v + 2]) * inv),
                                               __float_as_uint(__uint_as_float(o[4 * v + 3]) * inv));
                            } else {
                                w.x = pack_bf16x2(__uint_as_float(o[8 * v + 0]) * inv, __uint_as_float(o[8 * v + 1]) * inv);
                                w.y = pack_bf16x2(__uint_as_float(o[8 * v + 2]) * inv, __uint_as_float(o[8 * v + 3]) * inv);
                                w.z = pack_bf16x2(__uint_as_float(o[8 * v + 4]) * inv, __uint_as_float(o[8 * v + 5]) * inv);
                                w.w = pack_bf16x2(__uint_as_float(o[8 * v + 6]) * inv, __uint_as_float(o[8 * v + 7]) * inv);
                            }
                            const int box = (half + ob) * (kSplitP ? 2 : 1) + v / 8;
                            *reinterpret_cast<uint4*>(smem_gen + box * (kBlockM * 128) + row * 128 + (((v % 8) ^ (row & 7)) << 4)) = w;
                        }
                    }
                    fence_proxy_async_smem();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_staged);
                if (half == 0 && a.lse && qi < a.Sq) a.lse[stat] = lse;
                if (warp == 0 && lane == 0 && ok && mbar_wait(bar_staged, (uint32_t)(tiles & 1), wc, 0x58)) {
                    constexpr int kCols = kSplitP ? 32 : 64;           // of a 128-byte box
                    for (int i = 0; i < D / kCols; ++i) tma_store_4d(&tmap_o, smem_base + i * (kBlockM * 128), i * kCols, q0, h, b);
                    tma_store_commit();
                    tma_store_wait_read<0>();
                }
            } else if (qi < a.Sq) {
                // no key is visible to these rows: zeros and -inf
                using OutT = typename std::conditional<kSplitP, float, __nv_bfloat16>::type;
                uint4* dst = reinterpret_cast<uint4*>(reinterpret_cast<OutT*>(a.o) + b * a.o_sb + h * a.o_sh + (int64_t)qi * a.o_ss +
                                                      half * (D / kRS));
    #pragma unroll
                for (int v = 0; v < D / kRS * (int)sizeof(OutT) / 16; ++v) dst[v] = make_uint4(0u, 0u, 0u, 0u);
                if (half == 0 && a.lse) a.lse[stat] = neg_inf();
            }
        } while (kTeams > 1);
    }
    tc_fence_before_sync();
    bool gave_up;
    if constexpr (kTeams > 1) {
        gave_up = __syncthreads_or(misc[1] != 0);
        if (threadIdx.x == 0) item_counters_release(items.counters);
    } else {
        __syncthreads();
        gave_up = misc[1] != 0;
    }
    if (warp == kMmaWarp && team == 0) {
        __syncwarp();
        if (gave_up) __nanosleep(200000);    // aborted: give copies and MMAs in flight time to land
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTeams * L::kTmemCols);
    }
}

template <int D, bool kSplitP, bool kMask>
int launch_fwd_tile(ltca_ctx* ctx, const ltca_attn_params* p, const void* q, const void* k, const void* v, const ltca_strides& qs,
                    const ltca_strides& ks, const ltca_strides& vs, const FwdArgs& a) {
    using L = TileCfg<D, kSplitP, kMask>;
    CUtensorMap tq, tk, tv, to;
    int rc;
    if ((rc = make_tmap_bhsd(ctx, &tq, q, 2, p->B, p->H, p->Sq, D, qs, 64, kBlockM))) return rc;
    if ((rc = make_tmap_bhsd(ctx, &tk, k, 2, p->B, p->H, p->Sk, D, ks, 64, L::kBN))) return rc;
    if ((rc = make_tmap_bhsd(ctx, &tv, v, 2, p->B, p->H, p->Sk, D, vs, 64, L::kBN))) return rc;
    if ((rc = make_tmap_bhsd(ctx, &to, p->o, kSplitP ? 4 : 2, p->B, p->H, p->Sq, D, p->o_strides, kSplitP ? 32 : 64, kBlockM))) return rc;
    ItemGrid items;
    memset(&items, 0, sizeof(items));
    items.group = sched_group((int64_t)p->B * p->H, 4ll * p->Sk * D);
    // bf16 results at head_dim 64 keep to the SMs that the context allows: what a sequence-sharded run computes while slices
    // are on their way between the GPUs.
    if constexpr (D == 64 && !kSplitP) {
        items.nblk = (p->Sq + kBlockM - 1) / kBlockM;
        items.H = p->H;
        items.BH = p->B * p->H;
        const int64_t n = (int64_t)items.nblk * items.BH, ctas = (n + L::kCtas - 1) / L::kCtas;
        if (ctx->sm_count < ctx->sm_device && n <= 0x7fffffff - 2ll * L::kCtas * ctx->sm_device) {
            items.n_items = (int)n;
            items.counters = ctx->d_sched + 6;        // ints 6,7: the forward's
            auto kern = attn_fwd_tile_sm100_kernel<D, kSplitP, kMask, L::kCtas>;
            static SmemOptIn opt_in;
            LTCA_CUDA_OK(ctx, opt_in_dynamic_smem(opt_in, ctx->device, kern, L::kTeamsDynBytes));
            LTCA_CUDA_OK(ctx, launch_dependent_if(small_attention_call(p), kern, dim3((unsigned)(ctas < ctx->sm_count ? ctas : ctx->sm_count)),
                                                  dim3(L::kThreads * L::kCtas), L::kTeamsDynBytes, ctx->stream, tq, tk, tv, to, a, items));
            return LTCA_OK;
        }
    }
    auto kern = attn_fwd_tile_sm100_kernel<D, kSplitP, kMask, 1>;
    static SmemOptIn opt_in;
    LTCA_CUDA_OK(ctx, opt_in_dynamic_smem(opt_in, ctx->device, kern, L::kDynBytes));
    dim3 grid((p->Sq + kBlockM - 1) / kBlockM, p->H, p->B);
    LTCA_CUDA_OK(ctx, launch_dependent_if(small_attention_call(p), kern, grid, dim3(L::kThreads), L::kDynBytes, ctx->stream, tq, tk, tv, to, a, items));
    return LTCA_OK;
}

template <int D, typename OutT>
int launch_fwd(ltca_ctx* ctx, const ltca_attn_params* p, const void* mask_words, const void* q, const void* k,
               const void* v, const ltca_strides& qs, const ltca_strides& ks,
               const ltca_strides& vs) {
    constexpr bool kSplitP = sizeof(OutT) == 4;
    FwdArgs a;
    a.B = p->B; a.H = p->H; a.Sq = p->Sq; a.Sk = p->Sk;
    a.causal = p->causal ? 1 : 0;
    a.causal_off = p->Sk - p->Sq;
    a.scale = p->scale;
    a.scale_log2 = p->scale * 1.4426950408889634f;
    a.use_clamp = (p->score_clamp > 0.f) ? 1 : 0;
    a.clamp_raw = a.use_clamp ? p->score_clamp / p->scale : __builtin_inff();
    a.o = p->o;
    a.o_sb = p->o_strides.batch; a.o_sh = p->o_strides.head; a.o_ss = p->o_strides.seq;
    a.lse = p->lse;
    a.mask = mask_args(p, mask_words);
    a.kv_len = p->kv_len;
    a.status = ctx->d_status;

    // The one-tile kernel, except where head_dim is 64 and the call has so few tiles that two-tile CTAs run in one wave and
    // keys enough that a tile's own step time decides: there two threads per row shorten the step (two-tile kernel against
    // one-tile, us: bf16 B=1 H=8 S=4096 causal 60 and 61, B=4 H=16 Sq=512 Sk=4096 63 and 76, B=16 H=8 Sq=128 Sk=1024 15 and
    // 17; at S=512 the one-tile kernel is the faster one, 10.4 for B=4 H=8).  The line is older than the one-tile kernel's
    // hand-over of P in halves: with few pairs and long keys that kernel has since become the faster one for fp32 results (B=1
    // H=8 S=4096 causal 91 and 85; but B=4 H=16 Sq=512 Sk=4096 119 and 131) and is 1 to 13 % faster at some bf16 shapes
    // (B=2 H=8 S=1024 18.1 and 17.3, B=1 H=8 S=700 15.0 and 13.0; but S=2048 causal B=2 31.6 and 32.4).  The device's SM count decides, not a limit set on the context: the choice, and with it
    // the bits of the result, does not move with the launch width.
    const int64_t ctas2 = (int64_t)p->B * p->H * ((p->Sq + 2 * kBlockM - 1) / (2 * kBlockM));
    const int64_t sms = ctx->sm_device > 0 ? ctx->sm_device : kPlanSms;
    // Module calls with a key bias (ctx->fwd_pairs) keep it for short queries too.
    const bool few = ctas2 <= sms && p->Sk > 512;
    const bool ordered = ctx->fwd_pairs && (ctas2 <= sms || p->Sq <= 2 * kBlockM);
    if (D != 64 || !(few || ordered))
        return p->keep_mask ? launch_fwd_tile<D, kSplitP, true>(ctx, p, q, k, v, qs, ks, vs, a)
                            : launch_fwd_tile<D, kSplitP, false>(ctx, p, q, k, v, qs, ks, vs, a);

    if constexpr (D == 64) {
        using L = FwdCfg<kSplitP>;
        CUtensorMap tq, tk, tv;
        int rc;
        if ((rc = make_tmap_bhsd(ctx, &tq, q, 2, p->B, p->H, p->Sq, D, qs, 64, kBlockM))) return rc;
        if ((rc = make_tmap_bhsd(ctx, &tk, k, 2, p->B, p->H, p->Sk, D, ks, 64, L::kBN))) return rc;
        if ((rc = make_tmap_bhsd(ctx, &tv, v, 2, p->B, p->H, p->Sk, D, vs, 64, L::kBN))) return rc;
        auto kern = p->keep_mask ? attn_fwd_sm100_kernel<kSplitP, true> : attn_fwd_sm100_kernel<kSplitP, false>;
        static SmemOptIn opt_in[2];               // one pair per template instantiation
        LTCA_CUDA_OK(ctx, opt_in_dynamic_smem(opt_in[p->keep_mask ? 1 : 0], ctx->device, kern, L::kDynBytes));
        dim3 grid((p->Sq + 2 * kBlockM - 1) / (2 * kBlockM), p->H, p->B);
        LTCA_CUDA_OK(ctx, launch_dependent(kern, grid, dim3(kFwdThreads), L::kDynBytes, ctx->stream, tq, tk, tv, a));
        LTCA_LAUNCH_OK(ctx, "attn_fwd_sm100_kernel");
    }
    return LTCA_OK;
}

}  // namespace

#ifdef LTCA_TRACE
extern "C" int ltca_trace_read_fwd(unsigned long long* events, unsigned int* counts) {
    if (cudaMemcpyFromSymbol(events, g_trace, sizeof(g_trace)) != cudaSuccess) return -1;
    if (cudaMemcpyFromSymbol(counts, g_trace_count, sizeof(g_trace_count)) != cudaSuccess) return -1;
    return 0;
}
#endif

bool attn_fwd_sm100_supported(const ltca_attn_params* p) {
    if (p->D != 64 && p->D != 128) return false;
    if (p->Sq < 1 || p->Sk < 1) return false;
    if (!(p->scale > 0.f)) return false;
    if (p->H > 65535 || p->B > 65535) return false;
    return true;
}

// Expects bf16 Q, K, V (already converted when the caller's storage is fp32).
int launch_attn_fwd_sm100_bf16in(ltca_ctx* ctx, const ltca_attn_params* p, const void* mask_words, const void* q,
                                 const void* k, const void* v, const ltca_strides& qs,
                                 const ltca_strides& ks, const ltca_strides& vs) {
    const int oes = elem_size(p->dtype);
    if ((reinterpret_cast<uintptr_t>(p->o) & 15) || ((p->o_strides.seq * oes) & 15) ||
        ((p->o_strides.head * oes) & 15) || ((p->o_strides.batch * oes) & 15))
        return fail(ctx, LTCA_ERR_INVALID, "output base and strides must be 16-byte aligned");
    if (p->D == 64) {
        return p->dtype == LTCA_BF16 ? launch_fwd<64, __nv_bfloat16>(ctx, p, mask_words, q, k, v, qs, ks, vs)
                                     : launch_fwd<64, float>(ctx, p, mask_words, q, k, v, qs, ks, vs);
    }
    return p->dtype == LTCA_BF16 ? launch_fwd<128, __nv_bfloat16>(ctx, p, mask_words, q, k, v, qs, ks, vs)
                                 : launch_fwd<128, float>(ctx, p, mask_words, q, k, v, qs, ks, vs);
}

}  // namespace ltca
