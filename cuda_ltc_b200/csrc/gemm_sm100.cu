// Projection GEMMs of the TimeSelfAttention module on the tcgen05 tensor pipe.
//
//   C[M,N] = sum over pairs p of op(A_p) op(B_p)  (+ bias[N]),   bf16 operands, fp32 accumulation
//
// replaces the reference's cublasSgemm + addBiasKernel calls
// (reference src/ml/flash_attention.cu:866-958, 1075-1104) and the projections that cuDNN performs
// inside cudnnMultiHeadAttnForward / BackwardData / BackwardWeights (src/ml/cuDNN_ops.cu:203, 301, 366).
//
// Operand forms (all row-major in HBM):
//   A "K-major":  stored [M, K]  (activations x, ctx, dy, dq ...)      -> one 128 x 64 TMA box
//   A "M-major":  stored [K, M]  (x^T, ctx^T of the weight gradients)  -> two 64 x 64 boxes
//   B "K-major":  stored [N, K]  (a weight matrix used transposed)     -> one 128 x 64 box
//   B "N-major":  stored [K, N]  (a weight matrix used as stored; dq of the weight gradients)
// so no operand is ever transposed in memory: the instruction descriptor's major bits select the
// form and the shared-memory descriptors follow the layout the TMA boxes produce.
//
// Persistent CTAs (one per SM) walk a list of tiles of C: warp 0 is the TMA producer (ring of (A, B) stages of 64 K
// values), warp 1 issues the MMAs (K16 steps) into one of two accumulators in tensor memory, warps 2-5 are the epilogue
// (one accumulator row per thread: tcgen05.ld, bias, convert; the tile is staged in shared memory as 128-byte-swizzled
// boxes and stored with TMA), which works on tile i while the MMAs of tile i+1 run.  Tiles are 128 x 256 (four stages of
// 48 KB), 128 x 128 (six of 32 KB) or, for two CTAs of a cluster, 256 x 256 (six of 32 KB: each CTA holds its 128 rows of A
// and half the columns of B); pick_tile says which.  Measured at the module's sizes: a ring stage of 48 KB arrives
// every 600 - 700 cycles (about 80 bytes per cycle and SM from L2: every 128-row block of A is re-read once per
// N tile and every weight matrix once per M tile) against 512 cycles of MMAs; the epilogue of a tile takes 4700 cycles
// (bf16) to 7200 (fp32) and is hidden behind the next tile's main loop except for the last tile of a CTA.  Without any
// epilogue M=32768, N=3 x 512, K=512 takes 41 of 51 us, without its stores 47; eight epilogue warps, stores of 32 bytes
// per thread straight from registers and stores of whole lines through shared memory all took as long or longer.
// The tile list runs over independent problems (Q, K and V projections share one launch) and/or splits of K
// (weight gradients: K = batch x time is long and M x N is small, so the K range is cut into
// slices whose partial tiles go to scratch and are summed in a fixed order by a second kernel).
// `n_sum` > 1 accumulates several operand pairs into one tile (dx = dq Wq^T + dk Wk^T + dv Wv^T).
#include <type_traits>

#include "host_common.h"
#include "gemm_sm100.h"
#include "attn_wide.h"
#include "sm100_ptx.cuh"
#include "trace.cuh"
#ifndef LTCA_TRACE_GEMM_Z
#define LTCA_TRACE_GEMM_Z 1   // which launch of a module call records: the one with this many problems
#endif

namespace ltca {

namespace {

constexpr int kBM = 128, kBK = 64;                 // rows of A per CTA, contraction per ring stage
constexpr int kATileBytes = kBM * kBK * 2;         // 16 KB
// The result tile leaves through two staging boxes of 128 rows x 128 bytes (64 bf16 or 32 fp32 columns) that
// alternate.  A tiled TMA store reads shared memory at 32 bytes per cycle (513 cycles per box, measured with one
// and with 148 CTAs storing, whatever the number of stores in flight), so a second pair of boxes buys nothing,
// and a fourth ring stage measured 3 - 6 % faster at the module's sizes than three stages with four or five boxes.
constexpr int kStageBoxes = 2;
constexpr int kStageOutBytes = kBM * 128 * kStageBoxes;
constexpr int kGemmThreads = 192;
template <int kBN, bool kPair>
struct GemmCfg {
    static constexpr int kTileM = kPair ? 2 * kBM : kBM;           // rows of C per work item
    static constexpr int kBRows = kPair ? kBN / 2 : kBN;           // columns of the tile whose B this CTA holds
    static constexpr int kStageBytes = kATileBytes + kBRows * kBK * 2;
    static constexpr int kStages = kStageBytes > 32768 ? 4 : 6;    // operand ring
    static constexpr int kOutOff = kStages * kStageBytes;
    static constexpr int kBarOff = kOutOff + kStageOutBytes;
    static constexpr int kNumBars = 2 * kStages + 4;               // full[S], empty[S], acc_full[2], acc_empty[2]
    static constexpr int kMiscOff = kBarOff + kNumBars * 8;
    static constexpr int kBiasOff = kMiscOff + 16;                 // this tile's kBN bias values
    static constexpr int kDynBytes = kBiasOff + kBN * 4 + 1024;
    static_assert(kDynBytes <= 227 * 1024, "shared memory");
    static constexpr uint32_t kAccCols = 2 * kBN;                  // two accumulators
};

struct GemmMaps { CUtensorMap a[kMaxGemmProblems], b[kMaxGemmProblems], c[kMaxGemmProblems]; };
// A group's: up to three terms a member (twelve in all), second terms of the results behind the first.
constexpr int kMaxGroupPairs = 12;
struct GemmGroupMaps {
    CUtensorMap a[kMaxGroupPairs], b[kMaxGroupPairs], c[2 * kMaxGemmGroup];
    int first[kMaxGemmGroup + 1];      // a member's pairs
    int form[kMaxGemmGroup];           // ... operand forms (bit 0: A stored [K, M], bit 1: B stored [K, N]), and whether its
                                       // result has a second term (bit 2; where any has one)
    int M[kMaxGemmGroup], N[kMaxGemmGroup], K[kMaxGemmGroup], ksplit[kMaxGemmGroup], tiles_x[kMaxGemmGroup], tiles_y[kMaxGemmGroup];
    int tile0[kMaxGemmGroup + 1];      // ... tiles: members one after the other
};

struct GemmKArgs {
    int M, N, K;
    int n_sum, ksplit;
    int tiles_x, tiles_y, tiles_z;   // N tiles, M tiles, problems x K slices (a group: all tiles, 1, 1)
    int batch_h, batch_b;            // independent products of the same shape (slowest index of the tile list)
    int sum_h;                       // heads whose products one tile sums up
    int a_head, b_head;              // 0: the heads share the operand
    int out_bf16;
    int tma_store;                   // results leave through shared memory and a TMA store (needs 16-byte aligned rows)
    int add_to_c;
    int64_t c_bs[2];                 // element strides of C over (h, b)
    int64_t ldc;
    void* C[kMaxGemmProblems];
    void* c_lo;                      // second bf16 term of the (single) result, or null; its tensor map is c[1]
    const float* bias[kMaxGemmProblems];
    float* partial;                  // [problem][slice][M][N] when ksplit > 1
    uint32_t* status;
    RunIf run_if;
};

// One tile of the work list of a CTA.
struct GemmTile {
    int m0, n0, problem, slice, kb_begin, kb_end, pair_begin, n_pairs, n_iters;
    int M, N, ksplit;                // of its problem
    int bh, bb;                      // batch entry
};
template <int kBN, int kTileM, typename Maps>
__device__ __forceinline__ GemmTile gemm_tile(const Maps& maps, const GemmKArgs& g, int sum_h, int linear, int rank) {
    GemmTile t;
    int K, tiles_x, tiles_y;
    if constexpr (std::is_same<Maps, GemmGroupMaps>::value) {
        t.problem = 0;
        while (linear >= maps.tile0[t.problem + 1]) ++t.problem;
        linear -= maps.tile0[t.problem];
        t.M = maps.M[t.problem]; t.N = maps.N[t.problem]; K = maps.K[t.problem]; t.ksplit = maps.ksplit[t.problem];
        tiles_x = maps.tiles_x[t.problem]; tiles_y = maps.tiles_y[t.problem];
    } else {
        t.M = g.M; t.N = g.N; K = g.K; t.ksplit = g.ksplit;
        tiles_x = g.tiles_x; tiles_y = g.tiles_y;
    }
    const int x = linear % tiles_x;
    const int yz = linear / tiles_x;
    const int y = yz % tiles_y, zw = yz / tiles_y;
    t.n0 = x * kBN;
    t.m0 = y * kTileM + rank * kBM;
    if constexpr (std::is_same<Maps, GemmGroupMaps>::value) {
        t.slice = zw % t.ksplit;
        t.bh = zw / t.ksplit;
        t.bb = 0;
        t.pair_begin = maps.first[t.problem];
        t.n_pairs = maps.first[t.problem + 1] - t.pair_begin;
    } else {
        const int z = zw % g.tiles_z, w = zw / g.tiles_z;
        t.bh = w % g.batch_h;
        t.bb = w / g.batch_h;
        t.problem = z / g.ksplit;
        t.slice = z % g.ksplit;
        t.pair_begin = g.n_sum > 1 ? 0 : t.problem;
        t.n_pairs = g.n_sum > 1 ? g.n_sum : 1;
    }
    const int nkb = (K + kBK - 1) / kBK;
    const int per = (nkb + t.ksplit - 1) / t.ksplit;
    t.kb_begin = min(t.slice * per, nkb);
    t.kb_end = min(t.kb_begin + per, nkb);
    t.n_iters = t.n_pairs * sum_h * (t.kb_end - t.kb_begin);
    return t;
}

__device__ __forceinline__ bool has_second_term(const GemmMaps&, int) { return true; }
__device__ __forceinline__ bool has_second_term(const GemmGroupMaps& maps, int problem) { return (maps.form[problem] & 4) != 0; }
template <bool kByMember, bool kMn, typename Maps>
__device__ __forceinline__ bool is_mn(const Maps& maps, int problem, int bit) {
    if constexpr (kByMember) return (maps.form[problem] & bit) != 0;
    return kMn;
}

// Persistent: CTA (or pair) c computes tiles c, c + their number, ... of the list (N tiles fastest, so neighbouring CTAs
// share their rows of A in L2).  The two accumulators alternate: while the epilogue warps read tile i out of
// tensor memory, convert it and hand it to the TMA store, the MMA thread is already accumulating tile i+1 and
// the producer is loading tile i+2's operands.
// kKind: kHeads has operands that heads share, sums over heads and results that are added to C (the plain kernel is free of
// them: they cost it 0.1 us a launch); the members of a kGroup differ in shape, split of K, operand forms (kAMn, kBMn do
// not count) and number of terms.  Four weight gradients of 8 x 512 x 512 x 512 with three and two terms: 55 us as four launches, 31 as
// one.
enum GemmKind { kPlain, kHeads, kGroup };
template <bool kAMn, bool kBMn, int kBN, bool kPair, int kKind>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_bf16_sm100_kernel(const __grid_constant__ typename std::conditional<kKind == kGroup, GemmGroupMaps, GemmMaps>::type maps,
                       const __grid_constant__ GemmKArgs g) {
    const int sum_h = kKind == kHeads ? g.sum_h : 1;
    const bool add_to_c = kKind == kHeads && g.add_to_c;
    if (skipped(g.run_if)) return;
    using L = GemmCfg<kBN, kPair>;
    static_assert(kKind != kGroup || !kPair, "groups run on single CTAs");
    constexpr int kStages = L::kStages, kStageBytes = L::kStageBytes;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const uint32_t bar_base = smem_base + L::kBarOff;
    auto a_smem = [&](int s) { return smem_base + (uint32_t)(s * kStageBytes); };
    auto b_smem = [&](int s) { return smem_base + (uint32_t)(s * kStageBytes + kATileBytes); };
    auto bar_full = [&](int s) { return bar_base + 8u * s; };
    auto bar_empty = [&](int s) { return bar_base + 8u * (kStages + s); };
    auto bar_acc_full = [&](int b) { return bar_base + 8u * (2 * kStages + b); };
    auto bar_acc_empty = [&](int b) { return bar_base + 8u * (2 * kStages + 2 + b); };
    volatile uint32_t* misc = reinterpret_cast<volatile uint32_t*>(smem_gen + L::kMiscOff);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int n_tiles;
    if constexpr (kKind == kGroup) n_tiles = g.tiles_x;
    else n_tiles = g.tiles_x * g.tiles_y * g.tiles_z * g.batch_h * g.batch_b;
    const int rank = kPair ? (int)cluster_rank() : 0;             // rank 0 issues the pair's MMAs
    LTCA_TRACE_DECL(blockIdx.x == 5 && g.tiles_z == LTCA_TRACE_GEMM_Z);
    LTCA_TRACE_EVT(0x01);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(bar_acc_full(b), 1); mbar_init(bar_acc_empty(b), kPair ? 8 : 4); }
        misc[1] = 0u;
        mbar_fence_init();
    }
    if (warp == 1) {
        if constexpr (kPair) { tmem_alloc_pair(smem_u32(const_cast<uint32_t*>(&misc[0])), L::kAccCols); tmem_relinquish_pair(); }
        else { tmem_alloc(smem_u32(const_cast<uint32_t*>(&misc[0])), L::kAccCols); tmem_relinquish(); }
    }
    tc_fence_before_sync();
    __syncthreads();
    if constexpr (kPair) cluster_sync();                          // the other CTA's barriers may be signalled
    tc_fence_after_sync();
    const uint32_t tmem_base = misc[0];
    const WaitCtx wc{&misc[1], g.status};
    LTCA_TRACE_EVT(0x02);
    // Two tiles or more for every CTA: the kernel after this one may place its CTAs as these leave one by one (8192 rows,
    // QKV and attention: 55.0 us of module forward against 56.0).  With less the SMs without a tile would take them all.
    // This kernel's operands are complete once the kernel before it has ended.
    if (n_tiles >= 2 * (int)(kPair ? gridDim.x >> 1 : gridDim.x)) grid_launch_dependents();
    grid_dependency_wait();

    if (warp == 0) {
        if (lane == 0) {
            tma_prefetch_desc(&maps.a[0]);
            tma_prefetch_desc(&maps.b[0]);
            bool ok = true;
            int it = 0;
            for (int lin = kPair ? blockIdx.x >> 1 : blockIdx.x; lin < n_tiles && ok; lin += kPair ? gridDim.x >> 1 : gridDim.x) {
                const GemmTile t = gemm_tile<kBN, L::kTileM>(maps, g, sum_h, lin, rank);
                const bool amn = is_mn<kKind == kGroup, kAMn>(maps, t.problem, 1), bmn = is_mn<kKind == kGroup, kBMn>(maps, t.problem, 2);
                for (int p = 0, head = t.bh; p < t.n_pairs && ok; ++head == t.bh + sum_h ? (++p, head = t.bh) : 0) {
                    const int pair = t.pair_begin + p;
                    const CUtensorMap* ta = &maps.a[pair];
                    const CUtensorMap* tb = &maps.b[pair];
                    const int ha = kKind == kHeads && !g.a_head ? 0 : head, hb = kKind == kHeads && !g.b_head ? 0 : head;
                    for (int kb = t.kb_begin; kb < t.kb_end; ++kb, ++it) {
                        const int s = it % kStages;
                        ok = mbar_wait(bar_empty(s), (uint32_t)(((it / kStages) & 1) ^ 1), wc, 0xd0);
                        if (!ok) break;
                        LTCA_TRACE_EVT(0x10 + (it << 8));
                        // a pair's loads all signal the issuing CTA's barrier
                        if (rank == 0) mbar_arrive_expect_tx(bar_full(s), (uint32_t)(kPair ? 2 : 1) * kStageBytes);
                        const uint32_t bar = kPair ? map_shared(bar_full(s), 0) : bar_full(s);
                        auto load = [&](uint32_t dst, const CUtensorMap* map, int c0, int c1, int h) {
                            if constexpr (kPair) tma_load_4d_pair(dst, map, bar, c0, c1, h, t.bb);
                            else tma_load_4d(dst, map, bar, c0, c1, h, t.bb);
                        };
                        const int k0 = kb * kBK, n0 = t.n0 + rank * L::kBRows;
                        if (amn) {
                            load(a_smem(s), ta, t.m0, k0, ha);
                            load(a_smem(s) + 8192, ta, t.m0 + 64, k0, ha);
                        } else {
                            load(a_smem(s), ta, k0, t.m0, ha);
                        }
                        if (bmn) {
#pragma unroll
                            for (int pn = 0; pn < L::kBRows / 64; ++pn)     // 64-column blocks of 64 K rows, 8 KB each
                                load(b_smem(s) + pn * 8192, tb, n0 + 64 * pn, k0, hb);
                        } else {
#pragma unroll
                            for (int pn = 0; pn < L::kBRows / 128; ++pn)    // boxes of 128 rows of 128 bytes
                                load(b_smem(s) + pn * 16384, tb, k0, n0 + 128 * pn, hb);
                        }
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // K-major tile: 128 rows of 128 bytes, 8-row groups 1024 bytes apart, 32 bytes per K step.
            // MN-major tile: two blocks of 64 columns, 8192 bytes apart, each 64 K rows of 128 bytes;
            // a K step of 16 rows advances 2048 bytes.
            bool ok = true;
            int it = 0, na = 0;                         // ring position; tiles that used an accumulator
            for (int lin = kPair ? blockIdx.x >> 1 : blockIdx.x; lin < n_tiles && ok; lin += kPair ? gridDim.x >> 1 : gridDim.x) {
                const GemmTile t = gemm_tile<kBN, L::kTileM>(maps, g, sum_h, lin, rank);
                if (t.n_iters == 0) continue;
                const int buf = na & 1;
                // the epilogue has read this accumulator's previous tile out
                ok = mbar_wait(bar_acc_empty(buf), (uint32_t)(((na >> 1) & 1) ^ 1), wc, 0xd3);
                if (!ok) break;
                LTCA_TRACE_EVT(0x20 + (na << 8));
                const uint32_t acc = tmem_base + (uint32_t)kBN * buf;
                const bool amn = is_mn<kKind == kGroup, kAMn>(maps, t.problem, 1), bmn = is_mn<kKind == kGroup, kBMn>(maps, t.problem, 2);
                const uint32_t idesc = make_idesc_bf16(L::kTileM, kBN, amn ? 1 : 0, bmn ? 1 : 0);
                const uint64_t a_desc0 = make_smem_desc_sw128(a_smem(0), amn ? 8192 : 16, 1024);
                const uint64_t b_desc0 = make_smem_desc_sw128(b_smem(0), bmn ? 8192 : 16, 1024);
                const uint64_t a_step = amn ? 128 : 2, b_step = bmn ? 128 : 2;
                for (int i = 0; i < t.n_iters && ok; ++i, ++it) {
                    const int s = it % kStages;
                    ok = mbar_wait(bar_full(s), (uint32_t)((it / kStages) & 1), wc, 0xd1);
                    if (!ok) break;
                    LTCA_TRACE_EVT(0x21 + (it << 8));
                    tc_fence_after_sync();
                    const uint64_t ad = a_desc0 + (uint64_t)((s * kStageBytes) >> 4);
                    const uint64_t bd = b_desc0 + (uint64_t)((s * kStageBytes) >> 4);
#pragma unroll
                    for (int k = 0; k < kBK / 16; ++k) {
                        const uint32_t more = (i > 0 || k > 0) ? 1u : 0u;
                        if constexpr (kPair) mma_ss_pair(acc, ad + a_step * k, bd + b_step * k, idesc, more);
                        else mma_ss(acc, ad + a_step * k, bd + b_step * k, idesc, more);
                    }
                    if constexpr (kPair) mma_commit_pair(bar_empty(s));
                    else mma_commit(bar_empty(s));
                }
                if constexpr (kPair) { if (ok) mma_commit_pair(bar_acc_full(buf)); }
                else { if (ok) mma_commit(bar_acc_full(buf)); }
                LTCA_TRACE_EVT(0x22 + (na << 8));
                ++na;
            }
        }
    } else {
        // epilogue: warp w reads the 32 accumulator rows of its lane quarter (w % 4)
        const int qd = warp & 3;
        const int row = qd * 32 + lane;
        uint8_t* stage = smem_gen + L::kOutOff;
        const uint32_t stage_addr = smem_base + L::kOutOff;
        const int box_cols = g.out_bf16 ? 64 : 32;
        auto release_acc = [&](int buf) {                    // the accumulator is in registers
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                if constexpr (kPair) mbar_arrive_cluster(map_shared(bar_acc_empty(buf), 0));
                else mbar_arrive(bar_acc_empty(buf));
            }
        };
        bool ok = true;
        int na = 0, pc = 0;                                 // accumulators used; boxes staged
        for (int lin = kPair ? blockIdx.x >> 1 : blockIdx.x; lin < n_tiles; lin += kPair ? gridDim.x >> 1 : gridDim.x) {
            const GemmTile t = gemm_tile<kBN, L::kTileM>(maps, g, sum_h, lin, rank);
            const int gm = t.m0 + row;
            const int buf = na & 1;
            const bool have = t.n_iters > 0;
            if (have) {
                if (ok) ok = mbar_wait_warp(bar_acc_full(buf), (uint32_t)((na >> 1) & 1), wc, 0xd2);
                tc_fence_after_sync();
                LTCA_TRACE_EVT(0x30 + (na << 8));
                ++na;
            }
            const uint32_t tacc = tmem_base + (uint32_t)kBN * buf + ((uint32_t)(qd * 32) << 16);
            const float* bias = kKind != kGroup && g.ksplit == 1 ? g.bias[t.problem] : nullptr;
            if (g.tma_store) {
                // The tile leaves box by box: 128 rows of 128 bytes (64 bf16 or 32 fp32 columns) go to shared memory
                // in the layout of a 128-byte swizzled TMA box and one thread stores the box; the tensor map clips
                // rows and columns past the end of C.  (Storing a row's 16-byte pieces straight from registers costs
                // 32 L1 wavefronts per instruction, about as many cycles per tile as its MMAs.)  The two boxes of the
                // staging area alternate, so a box is filled while the store of the one before it is still reading,
                // and the columns of the next box are on their way out of tensor memory while this one is converted.
                // With a second term the low-order part takes the second box and the boxes do not alternate.
                const int n_pieces = kBN / box_cols;
                const bool two = g.out_bf16 != 0;              // a bf16 box holds two 32-column loads
                uint32_t va0[32], va1[32], vb0[32], vb1[32];
                auto load_piece = [&](int pi, uint32_t (&x0)[32], uint32_t (&x1)[32]) {
                    if (have && ok) {
                        tmem_ld32(tacc + pi * box_cols, x0);
                        if (two) tmem_ld32(tacc + pi * box_cols + 32, x1);
                    } else {
#pragma unroll
                        for (int c = 0; c < 32; ++c) x0[c] = x1[c] = 0u;
                    }
                };
                auto put_bf16 = [&](uint8_t* box, int ch0, const uint32_t (&v)[32]) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint4 w;
                        w.x = pack_bf16x2(__uint_as_float(v[8 * c + 0]), __uint_as_float(v[8 * c + 1]));
                        w.y = pack_bf16x2(__uint_as_float(v[8 * c + 2]), __uint_as_float(v[8 * c + 3]));
                        w.z = pack_bf16x2(__uint_as_float(v[8 * c + 4]), __uint_as_float(v[8 * c + 5]));
                        w.w = pack_bf16x2(__uint_as_float(v[8 * c + 6]), __uint_as_float(v[8 * c + 7]));
                        *reinterpret_cast<uint4*>(box + (((ch0 + c) ^ (row & 7)) << 4)) = w;
                        if (g.c_lo) {
                            uint4 l;
                            l.x = pack_bf16x2(__uint_as_float(v[8 * c + 0]) - __uint_as_float(w.x << 16),
                                              __uint_as_float(v[8 * c + 1]) - __uint_as_float(w.x & 0xffff0000u));
                            l.y = pack_bf16x2(__uint_as_float(v[8 * c + 2]) - __uint_as_float(w.y << 16),
                                              __uint_as_float(v[8 * c + 3]) - __uint_as_float(w.y & 0xffff0000u));
                            l.z = pack_bf16x2(__uint_as_float(v[8 * c + 4]) - __uint_as_float(w.z << 16),
                                              __uint_as_float(v[8 * c + 5]) - __uint_as_float(w.z & 0xffff0000u));
                            l.w = pack_bf16x2(__uint_as_float(v[8 * c + 6]) - __uint_as_float(w.w << 16),
                                              __uint_as_float(v[8 * c + 7]) - __uint_as_float(w.w & 0xffff0000u));
                            *reinterpret_cast<uint4*>(box + kBM * 128 + (((ch0 + c) ^ (row & 7)) << 4)) = l;
                        }
                    }
                };
                // The tile's bias goes through shared memory once: read per row from global memory it was 32 uniform
                // loads per 32 columns and thread, 7 us of a product of 3200 x 256 x 256.
                float* bias_s = reinterpret_cast<float*>(smem_gen + L::kBiasOff);
                if (bias) {
                    // (the last reads of the tile before lie before that tile's last barrier)
                    for (int c = row; c < kBN; c += 128) bias_s[c] = t.n0 + c < t.N ? __ldg(bias + t.n0 + c) : 0.f;
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                }
                auto add_bias = [&](int gn0, uint32_t (&v)[32]) {
#pragma unroll
                    for (int c = 0; c < 32; c += 4) {
                        const float4 x = *reinterpret_cast<const float4*>(bias_s + gn0 - t.n0 + c);
                        v[c] = __float_as_uint(__uint_as_float(v[c]) + x.x);
                        v[c + 1] = __float_as_uint(__uint_as_float(v[c + 1]) + x.y);
                        v[c + 2] = __float_as_uint(__uint_as_float(v[c + 2]) + x.z);
                        v[c + 3] = __float_as_uint(__uint_as_float(v[c + 3]) + x.w);
                    }
                };
                auto put_piece = [&](int pi, uint32_t (&x0)[32], uint32_t (&x1)[32]) {
                    const int gn0 = t.n0 + pi * box_cols;
                    if (bias) {
                        add_bias(gn0, x0);
                        if (two) add_bias(gn0 + 32, x1);
                    }
                    const int hb = g.c_lo ? 2 * (pc % (kStageBoxes / 2)) : pc % kStageBoxes;
                    // the box is free: the storing thread waits for the store that last read it before it comes here
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    uint8_t* box = stage + hb * (kBM * 128) + row * 128;
                    if (two) {
                        put_bf16(box, 0, x0);
                        put_bf16(box, 4, x1);
                    } else {
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                            *reinterpret_cast<uint4*>(box + ((c ^ (row & 7)) << 4)) =
                                make_uint4(x0[4 * c], x0[4 * c + 1], x0[4 * c + 2], x0[4 * c + 3]);
                    }
                    LTCA_TRACE_EVT(0x31 + (pi << 8));
                    fence_proxy_async_smem();
                    asm volatile("bar.sync 1, 128;" ::: "memory");    // the four epilogue warps have staged their rows
                    if (warp == 2 && lane == 0) {
                        // (partial tiles are one [problem][slice][M][N] tensor)
                        const CUtensorMap* tc = &maps.c[kKind != kGroup && g.ksplit > 1 ? 0 : t.problem];
                        if (gn0 < t.N && t.m0 < t.M) {
                            if (add_to_c) tma_reduce_add_4d(tc, stage_addr + hb * (kBM * 128), gn0, t.m0, t.bh, t.bb);
                            else tma_store_4d(tc, stage_addr + hb * (kBM * 128), gn0, t.m0, t.ksplit > 1 ? t.slice : t.bh,
                                              t.ksplit > 1 ? (kKind == kGroup ? 0 : t.problem) : t.bb);
                            if (g.c_lo && has_second_term(maps, t.problem))
                                tma_store_4d(&maps.c[kKind == kGroup ? kMaxGemmGroup + t.problem : 1], stage_addr + (hb + 1) * (kBM * 128), gn0, t.m0, t.bh, t.bb);
                        }
                        tma_store_commit();
                        // the box that the next piece takes has been read
                        if (g.c_lo) tma_store_wait_read<kStageBoxes / 2 - 1>();
                        else tma_store_wait_read<kStageBoxes - 1>();
                        LTCA_TRACE_EVT(0x32 + (pi << 8));
                    }
                    ++pc;
                };
                load_piece(0, va0, va1);
#pragma unroll 1
                for (int pi = 0; pi < n_pieces; pi += 2) {
                    tmem_wait_ld();
                    tmem_ld_fence(va0);
                    tmem_ld_fence(va1);
                    load_piece(pi + 1, vb0, vb1);
                    put_piece(pi, va0, va1);
                    tmem_wait_ld();
                    tmem_ld_fence(vb0);
                    tmem_ld_fence(vb1);
                    if (pi + 2 < n_pieces) {
                        load_piece(pi + 2, va0, va1);
                    } else if (have) {
                        release_acc(buf);              // the MMA thread may start the tile after next in it
                    }
                    put_piece(pi + 1, vb0, vb1);
                }
                continue;
            }
            // Direct stores: split-K partials and results whose rows are not 16-byte aligned.
#pragma unroll 1
            for (int c0 = 0; c0 < kBN; c0 += 32) {
                uint32_t v[32];
                __syncwarp();
                if (have && ok) {
                    tmem_ld32(tacc + c0, v);
                    tmem_wait_ld();
                } else {
#pragma unroll
                    for (int c = 0; c < 32; ++c) v[c] = 0u;
                }
                if (have && c0 + 32 == kBN) release_acc(buf);
                const int gn0 = t.n0 + c0;
                if (bias) {
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (gn0 + c < g.N) v[c] = __float_as_uint(__uint_as_float(v[c]) + __ldg(bias + gn0 + c));
                }
                if (gm >= g.M || gn0 >= g.N) continue;
                const bool full = gn0 + 32 <= g.N;
                if (g.ksplit > 1) {
                    float* dst = g.partial + (((int64_t)t.problem * g.ksplit + t.slice) * g.M + gm) * g.N + gn0;
                    if (full && (g.N & 3) == 0) {
#pragma unroll
                        for (int c = 0; c < 32; c += 4)
                            *reinterpret_cast<uint4*>(dst + c) = make_uint4(v[c], v[c + 1], v[c + 2], v[c + 3]);
                    } else {
#pragma unroll
                        for (int c = 0; c < 32; ++c)
                            if (gn0 + c < g.N) dst[c] = __uint_as_float(v[c]);
                    }
                } else if (g.out_bf16) {
                    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(g.C[t.problem]) + t.bh * g.c_bs[0] +
                                         t.bb * g.c_bs[1] + (int64_t)gm * g.ldc + gn0;
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (gn0 + c < g.N) dst[c] = __float2bfloat16_rn(__uint_as_float(v[c]));
                    if (g.c_lo) {
                        __nv_bfloat16* lo = reinterpret_cast<__nv_bfloat16*>(g.c_lo) + (dst -
                                            reinterpret_cast<__nv_bfloat16*>(g.C[t.problem]));
#pragma unroll
                        for (int c = 0; c < 32; ++c)
                            if (gn0 + c < g.N)
                                lo[c] = __float2bfloat16_rn(__uint_as_float(v[c]) - __bfloat162float(dst[c]));
                    }
                } else {
                    float* dst = reinterpret_cast<float*>(g.C[t.problem]) + t.bh * g.c_bs[0] + t.bb * g.c_bs[1] +
                                 (int64_t)gm * g.ldc + gn0;
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        if (gn0 + c < g.N) dst[c] = (add_to_c ? dst[c] : 0.f) + __uint_as_float(v[c]);
                }
            }
        }
        if (warp == 2 && lane == 0) tma_store_wait_read<0>();    // the staging area outlives its last store
    }

    LTCA_TRACE_EVT(0x3e);
    tc_fence_before_sync();
    __syncthreads();
    LTCA_TRACE_EVT(0x3f);
    if (misc[1]) __nanosleep(200000);        // aborted: give copies and MMAs in flight time to land
    if constexpr (kPair) cluster_sync();     // nothing of the other CTA's is on its way here any more
    if (warp == 1) {
        __syncwarp();
        tc_fence_after_sync();
        if constexpr (kPair) tmem_dealloc_pair(tmem_base, L::kAccCols);
        else tmem_dealloc(tmem_base, L::kAccCols);
    }
}

#ifdef LTCA_TRACE
}  // namespace
}  // namespace ltca
extern "C" int ltca_trace_read_gemm(unsigned long long* events, unsigned int* counts) {
    if (cudaMemcpyFromSymbol(events, ltca::g_trace, sizeof(ltca::g_trace)) != cudaSuccess) return -1;
    if (cudaMemcpyFromSymbol(counts, ltca::g_trace_count, sizeof(ltca::g_trace_count)) != cudaSuccess) return -1;
    return 0;
}
namespace ltca {
namespace {
#endif

// C[problem][i] = sum over slices of partial[problem][slice][i], in slice order; kVec consecutive i per thread, the loads
// of four slices in flight at once: four values where that still leaves a thousand threads per SM (3 x 512 x 512 from four
// slices: 4.8 us with one value and one load at a time, 3.7 so), else one (512 x 512 from 16 slices: 7.6 us with four).
template <int kVec>
__global__ void __launch_bounds__(256) gemm_splitk_reduce_kernel(const float* __restrict__ partial, float* c0, float* c1, float* c2,
                                                                 float* c3, int64_t mn, int ksplit, const RunIf run_if) {
    if (skipped(run_if)) return;
    grid_dependency_wait();
    const int problem = blockIdx.y;
    float* c = problem == 0 ? c0 : (problem == 1 ? c1 : (problem == 2 ? c2 : c3));
    const int64_t i = ((int64_t)blockIdx.x * 256 + threadIdx.x) * kVec;
    if (i >= mn) return;
    const float* p = partial + (int64_t)problem * ksplit * mn + i;
    float acc[kVec] = {};
    for (int s = 0; s < ksplit; s += 4) {
        float v[4][kVec];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (s + e >= ksplit) continue;
            if constexpr (kVec == 4) *reinterpret_cast<float4*>(v[e]) = __ldg(reinterpret_cast<const float4*>(p + (int64_t)(s + e) * mn));
            else v[e][0] = __ldg(p + (int64_t)(s + e) * mn);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int j = 0; j < kVec; ++j)
                if (s + e < ksplit) acc[j] += v[e][j];
    }
    if constexpr (kVec == 4) *reinterpret_cast<float4*>(c + i) = make_float4(acc[0], acc[1], acc[2], acc[3]);
    else c[i] = acc[0];
}

__global__ void cvt_rows_bf16_kernel(const float* __restrict__ src, int64_t ld_src, __nv_bfloat16* __restrict__ dst,
                                     int64_t ld_dst, int64_t rows, int cols) {
    const int64_t n = rows * cols;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = i / cols;
        const int c = (int)(i - r * cols);
        dst[r * ld_dst + c] = __float2bfloat16_rn(src[r * ld_src + c]);
    }
}

constexpr int kCvtBatch = 4;                   // loads in flight per thread (67 MB to 34: 16.6 us with one, 15.9 so)
__global__ void cvt_rows_bf16_vec_kernel(const float4* __restrict__ src, uint2* __restrict__ dst, int64_t n4) {
    const int64_t first = (int64_t)blockIdx.x * (kCvtBatch * 256) + threadIdx.x;
    float4 v[kCvtBatch];
#pragma unroll
    for (int e = 0; e < kCvtBatch; ++e)
        if (first + e * 256 < n4) v[e] = __ldg(src + first + e * 256);
#pragma unroll
    for (int e = 0; e < kCvtBatch; ++e)
        if (first + e * 256 < n4) dst[first + e * 256] = make_uint2(pack_bf16x2(v[e].x, v[e].y), pack_bf16x2(v[e].z, v[e].w));
}

// Several matrices of any sizes in ONE launch (the activations and the weights of a module call).  Releases the projection
// behind it at its start: that kernel's CTAs are one to an SM and cannot settle unevenly (module forward B32 S256 E512 54.9
// us, 55.1 without; module step B64 S512 equal within 0.2 %).
__global__ void cvt_many_bf16_kernel(const __grid_constant__ CvtMany b) {
    grid_launch_dependents();
    grid_dependency_wait();
    cvt_many_pieces(b, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

int make_operand_map(ltca_ctx* ctx, CUtensorMap* map, const GemmOperand& o, int mn_extent, int k_extent,
                     int batch_h, int batch_b, const int64_t* bs, bool shared) {
    if (shared) batch_h = 1;
    ltca_strides st;
    st.batch = bs[1]; st.head = bs[0]; st.seq = o.ld;
    if (o.mn_major)   // stored [K, MN]: rows are K, 64 x 64 boxes
        return make_tmap_bhsd(ctx, map, o.ptr, 2, batch_b, batch_h, k_extent, mn_extent, st, 64, 64);
    return make_tmap_bhsd(ctx, map, o.ptr, 2, batch_b, batch_h, mn_extent, k_extent, st, 64, 128);
}

// Which tile a product takes.
//   - 128 x 128: all its tiles fit beside one another on the SMs.  One wave either way, and the smaller tile is spread over
//     twice as many SMs and has half the epilogue behind its last MMA (M=3200 N=256 K=256: 9.3 us with 128 x 256, 7.1 so;
//     three such products of K=3200 in four slices 12.0, 9.0).  With a second wave the traffic per MMA decides against it
//     (M=8192, N=3 x 512, K=512: 17.4 us against 22.4), unless the other tile's second half would be empty anyway.
//   - pairs: contractions of kPairMinBlocks ring stages or more whose tiles fill the pairs' waves as well.  The pair loads a
//     third less per MMA (M=8192 N=4096, three pairs of K=512: 87 us and 76; dW of 3 x 512 x 512, K=32768: 60 and 52).  A
//     short contraction spends its time on the results, and there the two CTAs only wait for one another (M=32768,
//     N=3 x 512, K=512: 51 us and 56; 256 products of 256 x 256 x 512: 29 and 37).
//   - 128 x 256 otherwise.
enum GemmTileKind { kTile128, kTile256, kTilePair };
constexpr int kPairMinBlocks = 16;
GemmTileKind pick_tile(int M, int N, int64_t blocks, int64_t z, int sms) {
    auto up = [](int64_t a, int64_t b) { return (a + b - 1) / b; };
    if (N <= 128 || up(M, 128) * up(N, 128) * z <= sms) return kTile128;
    if (sms < 2 || blocks < kPairMinBlocks) return kTile256;
    const int64_t waves_pair = up(up(M, 256) * up(N, 256) * z, sms / 2), waves_256 = up(up(M, 128) * up(N, 256) * z, sms);
    return waves_pair <= waves_256 ? kTilePair : kTile256;
}

template <int kBN, bool kPair, int kKind>
int launch_gemm(ltca_ctx* ctx, const GemmMaps& m, const GemmKArgs& g, bool amn, bool bmn, int64_t n_tiles, int sms) {
    using L = GemmCfg<kBN, kPair>;
    auto kern = !bmn ? gemm_bf16_sm100_kernel<false, false, kBN, kPair, kKind>
                     : (amn ? gemm_bf16_sm100_kernel<true, true, kBN, kPair, kKind> : gemm_bf16_sm100_kernel<false, true, kBN, kPair, kKind>);
    static SmemOptIn opt_in[3];
    LTCA_CUDA_OK(ctx, opt_in_dynamic_smem(opt_in[!bmn ? 0 : (amn ? 2 : 1)], ctx->device, kern, L::kDynBytes));
    const int64_t units = kPair ? sms / 2 : sms;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)((n_tiles < units ? n_tiles : units) * (kPair ? 2 : 1)));
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = L::kDynBytes;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 2; attr[1].val.clusterDim.y = 1; attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = kPair ? 2 : 1;
    LTCA_CUDA_OK(ctx, cudaLaunchKernelEx(&cfg, kern, m, g));
    LTCA_LAUNCH_OK(ctx, "gemm_bf16_sm100_kernel");
    return LTCA_OK;
}

}  // namespace

size_t gemm_sm100_partial_bytes(int M, int N, int n_problems, int ksplit) {
    if (ksplit <= 1) return 0;
    return align_up((size_t)n_problems * ksplit * M * N * sizeof(float), 256);
}

int gemm_sm100_pick_ksplit(int M, int N, int K, int n_problems, int sm_count) {
    const int tiles = ((M + kBM - 1) / kBM) * ((N + 255) / 256) * n_problems;
    const int nkb = (K + kBK - 1) / kBK;
    if (sm_count <= 0) sm_count = kPlanSms;
    int ks = 1;
    // split while the tiles alone leave most SMs idle and every slice keeps at least 8 K blocks
    while (tiles * ks * 2 <= sm_count && nkb / (ks * 2) >= 8 && ks < 16) ks *= 2;
    return ks;
}

int gemm_sm100(ltca_ctx* ctx, const GemmProblem& gp) {
    if (gp.n_problems < 1 || gp.n_problems > kMaxGemmProblems || gp.n_sum < 1 || gp.n_sum > 3 ||
        (gp.n_sum > 1 && gp.n_problems != 1))
        return fail(ctx, LTCA_ERR_INVALID, "gemm: between 1 and 4 problems, or one problem of up to 3 summed pairs");
    if (gp.M < 1 || gp.N < 1 || gp.K < 1) return fail(ctx, LTCA_ERR_INVALID, "gemm: empty problem");
    const bool batched = gp.batch_h > 1 || gp.batch_b > 1;
    if (gp.sum_h < 1 || (gp.sum_h > 1 && (gp.batch_h != 1 || gp.n_problems != 1 || gp.ksplit > 1)))
        return fail(ctx, LTCA_ERR_INVALID, "gemm: a sum over heads takes one problem, no batch of heads and no split of K");
    if (gp.add_to_c && (gp.out_bf16 || gp.ksplit > 1)) return fail(ctx, LTCA_ERR_INVALID, "gemm: adding to C needs fp32 results, no split of K");
    const int heads = gp.sum_h > 1 ? gp.sum_h : gp.batch_h;
    if (gp.batch_h < 1 || gp.batch_b < 1 || (batched && (gp.n_problems != 1 || gp.ksplit > 1)))
        return fail(ctx, LTCA_ERR_INVALID, "gemm: a batch takes one problem (or one sum of pairs) and no split of K");
    const int n_pairs = gp.n_sum > 1 ? gp.n_sum : gp.n_problems;
    GemmMaps maps;
    int rc;
    for (int i = 0; i < n_pairs; ++i) {
        if (gp.a[i].mn_major != gp.a[0].mn_major || gp.b[i].mn_major != gp.b[0].mn_major)
            return fail(ctx, LTCA_ERR_INVALID, "gemm: all pairs of one launch share the operand forms");
        if ((rc = make_operand_map(ctx, &maps.a[i], gp.a[i], gp.M, gp.K, heads, gp.batch_b, gp.a_bs, gp.a_shared != 0))) return rc;
        if ((rc = make_operand_map(ctx, &maps.b[i], gp.b[i], gp.N, gp.K, heads, gp.batch_b, gp.b_bs, gp.b_shared != 0))) return rc;
    }
    GemmKArgs g;
    g.M = gp.M; g.N = gp.N; g.K = gp.K;
    g.n_sum = gp.n_sum;
    g.ksplit = gp.ksplit > 1 ? gp.ksplit : 1;
    g.ldc = gp.ldc;
    g.out_bf16 = gp.out_bf16;
    g.c_lo = gp.c_lo;
    if (gp.c_lo && (!gp.out_bf16 || gp.n_problems != 1 || gp.ksplit > 1))
        return fail(ctx, LTCA_ERR_INVALID, "gemm: a second result term needs one bf16 problem and no split of K");
    for (int i = 0; i < kMaxGemmProblems; ++i) { g.C[i] = gp.c[i < gp.n_problems ? i : 0]; g.bias[i] = i < gp.n_problems ? gp.bias[i] : nullptr; }
    g.partial = gp.partial;
    g.status = ctx->d_status;
    g.run_if = ctx->run_if;
    g.batch_h = gp.batch_h; g.batch_b = gp.batch_b;
    g.sum_h = gp.sum_h;
    g.a_head = gp.a_shared ? 0 : 1; g.b_head = gp.b_shared ? 0 : 1;
    g.add_to_c = gp.add_to_c;
    g.c_bs[0] = gp.c_bs[0]; g.c_bs[1] = gp.c_bs[1];
    const int ces = gp.out_bf16 ? 2 : 4;
    if (g.ksplit > 1) {
        const int64_t mn = (int64_t)gp.M * gp.N;
        const ltca_strides ps{mn * g.ksplit, mn, gp.N};
        g.tma_store = (gp.N & 3) == 0 && (reinterpret_cast<uintptr_t>(gp.partial) & 15) == 0;
        if (g.tma_store && (rc = make_tmap_bhsd(ctx, &maps.c[0], gp.partial, 4, gp.n_problems, g.ksplit, gp.M, gp.N, ps, 32, kBM))) return rc;
    } else {
        g.tma_store = ((gp.ldc * ces) % 16) == 0 && ((gp.c_bs[0] * ces) % 16) == 0 && ((gp.c_bs[1] * ces) % 16) == 0 &&
                      (reinterpret_cast<uintptr_t>(gp.c_lo) & 15) == 0;
        for (int i = 0; i < gp.n_problems; ++i)
            if (reinterpret_cast<uintptr_t>(gp.c[i]) & 15) g.tma_store = 0;
        const ltca_strides cs{gp.c_bs[1], gp.c_bs[0], gp.ldc};
        for (int i = 0; i < (gp.c_lo ? 2 : gp.n_problems) && g.tma_store; ++i) {
            void* dst = (i == 1 && gp.c_lo) ? gp.c_lo : gp.c[i];
            if ((rc = make_tmap_bhsd(ctx, &maps.c[i], dst, ces, gp.batch_b, gp.batch_h, gp.M, gp.N, cs,
                                     gp.out_bf16 ? 64 : 32, kBM))) return rc;
        }
    }
    if (g.ksplit > 1) {
        if (!gp.partial) return fail(ctx, LTCA_ERR_WORKSPACE, "gemm: split K needs scratch");
        if (gp.out_bf16) return fail(ctx, LTCA_ERR_INVALID, "gemm: split K writes fp32 results");
        for (int i = 0; i < gp.n_problems; ++i)
            if (gp.bias[i]) return fail(ctx, LTCA_ERR_INVALID, "gemm: split K takes no bias");
    }
    const int sms = ctx->sm_count > 0 ? ctx->sm_count : kPlanSms;
    const int64_t z = (int64_t)gp.n_problems * g.ksplit * gp.batch_h * gp.batch_b;
    const GemmTileKind kind = pick_tile(gp.M, gp.N, (int64_t)((gp.K + kBK - 1) / kBK) / g.ksplit * g.n_sum * g.sum_h, z, sms);
    const int tile_m = kind == kTilePair ? 2 * kBM : kBM, tile_n = kind == kTile128 ? 128 : 256;
    g.tiles_x = (gp.N + tile_n - 1) / tile_n;
    g.tiles_y = (gp.M + tile_m - 1) / tile_m;
    g.tiles_z = gp.n_problems * g.ksplit;
    const int64_t n_tiles = g.tiles_x * (g.tiles_y * z);
    if (n_tiles > 0x7fffffff) return fail(ctx, LTCA_ERR_UNSUPPORTED, "gemm: too many tiles");
    const bool amn = gp.a[0].mn_major != 0, bmn = gp.b[0].mn_major != 0;
    if (amn && !bmn) return fail(ctx, LTCA_ERR_UNSUPPORTED, "gemm: A stored [K, M] with B stored [N, K] is not built");
    auto launch = kind == kTilePair ? launch_gemm<256, true, kPlain> : kind == kTile256 ? launch_gemm<256, false, kPlain> : launch_gemm<128, false, kPlain>;
    if (g.sum_h > 1 || g.add_to_c || !g.a_head || !g.b_head)
        launch = kind == kTilePair ? launch_gemm<256, true, kHeads> : kind == kTile256 ? launch_gemm<256, false, kHeads> : launch_gemm<128, false, kHeads>;
    rc = launch(ctx, maps, g, amn, bmn, n_tiles, sms);
    if (rc) return rc;
    return g.ksplit > 1 ? sum_splits(ctx, gp.partial, gp.c, gp.n_problems, (int64_t)gp.M * gp.N, g.ksplit) : LTCA_OK;
}

int sum_splits(ltca_ctx* ctx, const float* partial, void* const* dst, int n, int64_t mn, int ksplit) {
    float* c[kMaxGemmProblems];
    bool vec = (mn & 3) == 0 && (reinterpret_cast<uintptr_t>(partial) & 15) == 0 && mn / 4 * n >= (int64_t)kPlanSms * 1024;
    for (int i = 0; i < kMaxGemmProblems; ++i) {
        c[i] = reinterpret_cast<float*>(dst[i < n ? i : 0]);
        vec = vec && (reinterpret_cast<uintptr_t>(c[i]) & 15) == 0;
    }
    const int64_t per = vec ? 1024 : 256;
    const dim3 rg((unsigned)((mn + per - 1) / per), n);
    auto kern = vec ? gemm_splitk_reduce_kernel<4> : gemm_splitk_reduce_kernel<1>;
    LTCA_CUDA_OK(ctx, launch_dependent(kern, rg, dim3(256), 0, ctx->stream, partial, c[0], c[1], c[2], c[3], mn, ksplit, ctx->run_if));
    LTCA_LAUNCH_OK(ctx, "gemm_splitk_reduce_kernel");
    return LTCA_OK;
}

bool gemm_group_aligned(const GemmGroup& gg) {
    const int ces = gg.out_bf16 ? 2 : 4;
    for (int i = 0; i < gg.n; ++i) {
        const GemmGroup::Member& m = gg.m[i];
        if (m.ksplit > 1 && ((m.N & 3) || gg.heads > 1 || gg.out_bf16)) return false;
        if (((m.ldc * ces) & 15) || (gg.heads > 1 && ((m.c_hs * ces) & 15)) || (reinterpret_cast<uintptr_t>(m.c) & 15) ||
            (reinterpret_cast<uintptr_t>(m.c_lo) & 15))
            return false;
    }
    return true;
}

template <int kBN>
static int launch_group(ltca_ctx* ctx, const GemmGroupMaps& m, const GemmKArgs& g, int64_t n_tiles, int sms) {
    using L = GemmCfg<kBN, false>;
    auto kern = gemm_bf16_sm100_kernel<false, false, kBN, false, kGroup>;
    static SmemOptIn opt_in;
    LTCA_CUDA_OK(ctx, opt_in_dynamic_smem(opt_in, ctx->device, kern, L::kDynBytes));
    LTCA_CUDA_OK(ctx, launch_dependent(kern, dim3((unsigned)(n_tiles < sms ? n_tiles : sms)), dim3(kGemmThreads), L::kDynBytes, ctx->stream,
                                       m, g));
    LTCA_LAUNCH_OK(ctx, "gemm_bf16_sm100_kernel");
    return LTCA_OK;
}

int gemm_sm100_group(ltca_ctx* ctx, const GemmGroup& gg) {
    if (gg.heads < 1 || gg.n < 1 || gg.n > kMaxGemmGroup || !gemm_group_aligned(gg))
        return fail(ctx, LTCA_ERR_INVALID, "gemm: between 1 and %d members with 16-byte aligned results", kMaxGemmGroup);
    GemmGroupMaps maps;
    GemmKArgs g;
    memset(&maps, 0, sizeof(maps));
    memset(&g, 0, sizeof(g));
    g.n_sum = 1; g.ksplit = 1; g.sum_h = 1;
    g.batch_h = gg.heads; g.batch_b = 1;
    g.a_head = g.b_head = 1;
    g.out_bf16 = gg.out_bf16;
    g.tma_store = 1;
    for (int i = 0; i < gg.n; ++i)
        if (gg.m[i].c_lo) g.c_lo = gg.m[i].c_lo;       // (whether any is there: the stores go by the members' tensor maps)
    g.status = ctx->d_status;
    g.run_if = ctx->run_if;
    const int sms = ctx->sm_count > 0 ? ctx->sm_count : kPlanSms;
    bool wide = false;
    for (int i = 0; i < gg.n; ++i) wide = wide || gg.m[i].N > 128;
    wide = wide && !gemm_group_one_wave(ctx, gg);      // (pick_tile's rule, for all members alike)
    int64_t n_tiles = 0;
    int rc;
    for (int i = 0; i < gg.n; ++i) {
        const GemmGroup::Member& m = gg.m[i];
        if (m.M < 1 || m.N < 1 || m.K < 1 || m.ksplit < 1) return fail(ctx, LTCA_ERR_INVALID, "gemm: empty member");
        if (m.terms < 1 || m.terms > 3 || maps.first[i] + m.terms > kMaxGroupPairs || (m.c_lo && !gg.out_bf16))
            return fail(ctx, LTCA_ERR_INVALID, "gemm: a member has one to three terms, and a second term of its result in bf16 only");
        const int64_t as[2] = {m.a_hs, 0}, bs[2] = {m.b_hs, 0};
        maps.first[i + 1] = maps.first[i] + m.terms;
        maps.form[i] = (m.a[0].mn_major ? 1 : 0) | (m.b[0].mn_major ? 2 : 0) | (m.c_lo ? 4 : 0);
        for (int t = 0; t < m.terms; ++t) {
            if (m.a[t].mn_major != m.a[0].mn_major || m.b[t].mn_major != m.b[0].mn_major)
                return fail(ctx, LTCA_ERR_INVALID, "gemm: the terms of a member share the operand forms");
            if ((rc = make_operand_map(ctx, &maps.a[maps.first[i] + t], m.a[t], m.M, m.K, gg.heads, 1, as, false))) return rc;
            if ((rc = make_operand_map(ctx, &maps.b[maps.first[i] + t], m.b[t], m.N, m.K, gg.heads, 1, bs, false))) return rc;
        }
        const bool split = m.ksplit > 1;               // the slices stand where the heads' results do
        const ltca_strides cs{0, split ? (int64_t)m.M * m.N : m.c_hs, split ? m.N : m.ldc};
        for (int l = 0; l < (m.c_lo ? 2 : 1); ++l)
            if ((rc = make_tmap_bhsd(ctx, &maps.c[l * kMaxGemmGroup + i], l ? m.c_lo : m.c, gg.out_bf16 ? 2 : 4, 1, split ? m.ksplit : gg.heads,
                                     m.M, m.N, cs, gg.out_bf16 ? 64 : 32, kBM))) return rc;
        maps.M[i] = m.M; maps.N[i] = m.N; maps.K[i] = m.K; maps.ksplit[i] = m.ksplit;
        maps.tiles_x[i] = (m.N + (wide ? 255 : 127)) / (wide ? 256 : 128);
        maps.tiles_y[i] = (m.M + kBM - 1) / kBM;
        n_tiles += (int64_t)maps.tiles_x[i] * maps.tiles_y[i] * m.ksplit * gg.heads;
        if (n_tiles > 0x7fffffff) return fail(ctx, LTCA_ERR_UNSUPPORTED, "gemm: too many tiles");
        maps.tile0[i + 1] = (int)n_tiles;
    }
    g.tiles_x = (int)n_tiles; g.tiles_y = g.tiles_z = 1;
    return wide ? launch_group<256>(ctx, maps, g, n_tiles, sms) : launch_group<128>(ctx, maps, g, n_tiles, sms);
}

bool gemm_group_one_wave(const ltca_ctx* ctx, const GemmGroup& gg) {
    int64_t n = 0;
    for (int i = 0; i < gg.n; ++i)
        n += (int64_t)((gg.m[i].M + 127) / 128) * ((gg.m[i].N + 127) / 128) * gg.m[i].ksplit * gg.heads;
    return n <= (ctx->sm_count > 0 ? ctx->sm_count : kPlanSms);
}

int convert_rows_bf16(ltca_ctx* ctx, const float* src, int64_t ld_src, void* dst, int64_t ld_dst, int64_t rows,
                      int cols) {
    if (rows < 1 || cols < 1) return LTCA_OK;
    const int64_t n = rows * cols;
    if (ld_src == cols && ld_dst == cols && (n & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0 &&
        (reinterpret_cast<uintptr_t>(dst) & 7) == 0) {
        const int64_t n4 = n / 4;
        const unsigned blocks = (unsigned)((n4 + kCvtBatch * 256 - 1) / (kCvtBatch * 256));
        cvt_rows_bf16_vec_kernel<<<blocks, 256, 0, ctx->stream>>>(reinterpret_cast<const float4*>(src),
                                                                  reinterpret_cast<uint2*>(dst), n4);
    } else {
        const unsigned blocks = (unsigned)((n + 255) / 256 < 2368 ? (n + 255) / 256 : 2368);
        cvt_rows_bf16_kernel<<<blocks, 256, 0, ctx->stream>>>(src, ld_src, reinterpret_cast<__nv_bfloat16*>(dst),
                                                              ld_dst, rows, cols);
    }
    LTCA_LAUNCH_OK(ctx, "cvt_rows_bf16_kernel");
    return LTCA_OK;
}


bool make_cvt_many(CvtMany* b, int n, const float* const* src, const int64_t* ld_src, void* const* dst, const int64_t* ld_dst,
                   const int64_t* rows, const int* cols, void* const* lo) {
    memset(b, 0, sizeof(*b));
    uint64_t total = 0;
    for (int i = 0; i < n; ++i) {
        if (rows[i] < 1 || cols[i] < 1) continue;
        if ((lo && lo[i] && (reinterpret_cast<uintptr_t>(lo[i]) & 7)) || (cols[i] & 3) || (ld_src[i] & 3) || (ld_dst[i] & 3) ||
            (reinterpret_cast<uintptr_t>(src[i]) & 15) || (reinterpret_cast<uintptr_t>(dst[i]) & 7))
            return false;
        const int m = b->n++;
        b->src[m] = src[i]; b->dst[m] = reinterpret_cast<__nv_bfloat16*>(dst[i]);
        b->lo[m] = lo ? reinterpret_cast<__nv_bfloat16*>(lo[i]) : nullptr;
        b->ld_src[m] = ld_src[i]; b->ld_dst[m] = ld_dst[i];
        b->cols4[m] = (uint32_t)(cols[i] / 4);
        b->start4[m] = (uint32_t)total;
        total += (uint64_t)rows[i] * (uint64_t)(cols[i] / 4);
    }
    b->start4[b->n] = (uint32_t)total;
    return total < (1ull << 31);
}

int convert_many_bf16(ltca_ctx* ctx, int n, const float* const* src, const int64_t* ld_src, void* const* dst,
                      const int64_t* ld_dst, const int64_t* rows, const int* cols, void* const* lo) {
    if (n < 1 || n > kMaxCvtMany) return fail(ctx, LTCA_ERR_INVALID, "convert_many_bf16 takes 1 to %d matrices", kMaxCvtMany);
    CvtMany b;
    if (!make_cvt_many(&b, n, src, ld_src, dst, ld_dst, rows, cols, lo)) {
        // odd shapes or alignments: one matrix at a time
        for (int i = 0; i < n; ++i) {
            int rc;
            if (lo && lo[i]) rc = wide_split_bf16(ctx, src[i], ld_src[i], dst[i], lo[i], ld_dst[i], rows[i], cols[i]);
            else rc = convert_rows_bf16(ctx, src[i], ld_src[i], dst[i], ld_dst[i], rows[i], cols[i]);
            if (rc) return rc;
        }
        return LTCA_OK;
    }
    if (b.n == 0) return LTCA_OK;
    const uint32_t total = b.start4[b.n];
    const unsigned blocks = (unsigned)((total + 255) / 256 < 2368 ? (total + 255) / 256 : 2368);
    LTCA_CUDA_OK(ctx, launch_dependent(cvt_many_bf16_kernel, dim3(blocks), dim3(256), 0, ctx->stream, b));
    LTCA_LAUNCH_OK(ctx, "cvt_many_bf16_kernel");
    return LTCA_OK;
}

}  // namespace ltca
