// Products of the module's exact pipeline: fp32 operands, fp32 FMA arithmetic (that of the reference's cublasSgemm with
// tensor cores off, src/ml/flash_attention.cu:531-536).  The sums run in ascending order of the contraction, but for
// sliced contractions (slice by slice) and the small products that may run in any order (eight interleaved shares).
//
// What bounds them: the small modules this pipeline serves (model widths of 32 to 256, up to a few thousand rows) are
// launches and latency, the larger ones the FMA pipe.  So the products of one step (Q, K and V; the four weight gradients;
// the three terms of dx) share a launch, the tile shrinks until the tiles occupy the SMs, and operands arrive by
// 16-byte cp.async some steps ahead in whatever order they are stored: an operand whose rows run along the contraction is
// read as vectors of four contraction steps, one whose rows run across it as vectors of four rows or columns, so
// nothing is transposed on the way.
// Measured at B8 S32 E32 with 4 heads of 32: 21 launches of one 128 x 128 tile kernel took 8 to 24 us each and 241 us a
// training step; see pick_tile for the tiles.
#include "gemm_fp32.h"
#include "sm100_ptx.cuh"

namespace ltca {

namespace {

constexpr int kPad = 4;

struct Gemm32Args {
    Gemm32Problem p[kMaxGemm32];
    int n, sum;
    int kper, slices;      // contraction extent and number of slices (blockIdx.z = problem * slices + slice)
    float* partial;        // slice results: problem after problem, slice after slice, [M][N] each; null when unsliced
    int64_t part_off[kMaxGemm32];
    int vec;               // every operand row starts on a 16-byte boundary
};

__device__ __forceinline__ void cp_async16(float* dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

// Rows [r0, r0 + R) x columns [c0, c0 + C) of a row-major matrix into shared [R][C + kPad], zeros beyond it.
template <int R, int C, int NT>
__device__ __forceinline__ void load_block(float* dst, const float* base, int ld, int r0, int rows, int c0, int cols, bool vec) {
    constexpr int LD = C + kPad;
    if (vec) {
        constexpr int C4 = C / 4;
#pragma unroll
        for (int e0 = 0; e0 < R * C4; e0 += NT) {
            const int e = e0 + threadIdx.x;
            if (R * C4 % NT != 0 && e >= R * C4) break;
            const int r = e / C4, c = (e % C4) * 4;
            const int left = r0 + r < rows ? min(16, 4 * (cols - c0 - c)) : 0;
            cp_async16(dst + r * LD + c, left > 0 ? base + (int64_t)(r0 + r) * ld + c0 + c : base, left > 0 ? left : 0);
        }
    } else {
        for (int e = threadIdx.x; e < R * C; e += NT) {
            const int r = e / C, c = e % C;
            const bool in = r0 + r < rows && c0 + c < cols;
            cp_async4(dst + r * LD + c, in ? base + (int64_t)(r0 + r) * ld + c0 + c : base, in ? 4 : 0);
        }
    }
}

// N values of one contraction step e (0..3) or four steps of N rows, as the operand is stored.
template <bool kAlongK, int N, int V, int STRIDE>
struct Frag {
    float v[4][N];
    // along the contraction: rows x0 + STRIDE i (pitch LD), columns k .. k + 3
    // across it: row k + e, columns x0 + (i / V) * STRIDE + i % V
    template <int LD>
    __device__ __forceinline__ void load(const float* tile, int x0, int k) {
        if constexpr (kAlongK) {
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const float4 t = *reinterpret_cast<const float4*>(tile + (x0 + (i / V) * STRIDE + i % V) * LD + k);
                v[0][i] = t.x; v[1][i] = t.y; v[2][i] = t.z; v[3][i] = t.w;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < N; i += V) {
                    const float* p = tile + (k + e) * LD + x0 + (i / V) * STRIDE;
                    if constexpr (V == 4) {
                        const float4 t = *reinterpret_cast<const float4*>(p);
                        v[e][i] = t.x; v[e][i + 1] = t.y; v[e][i + 2] = t.z; v[e][i + 3] = t.w;
                    } else if constexpr (V == 2) {
                        const float2 t = *reinterpret_cast<const float2*>(p);
                        v[e][i] = t.x; v[e][i + 1] = t.y;
                    } else {
                        v[e][i] = *p;
                    }
                }
        }
    }
};

template <int TM, int TN, int NT>
struct Gemm32Tile {
    static constexpr int KC = TM >= 128 ? 16 : 32;
    // A 32 x 32 tile multiplies a step in a fraction of the latency of its loads and nothing else runs beside it (such
    // launches have few CTAs): five steps in flight instead of two.
    static constexpr int kStages = TM <= 32 ? 6 : 3;
    static constexpr int TY = NT / 16, RM = TM / TY, CN = TN / 16;
    static constexpr int VM = RM < 4 ? RM : 4, VN = CN < 4 ? CN : 4;
    template <bool TA> static constexpr int a_floats() { return TA ? KC * (TM + kPad) : TM * (KC + kPad); }
    template <bool TB> static constexpr int b_floats() { return TB ? TN * (KC + kPad) : KC * (TN + kPad); }
};

template <bool TA, bool TB, int TM, int TN, int NT>
__global__ void __launch_bounds__(NT) gemm_fp32_kernel(const __grid_constant__ Gemm32Args g) {
    grid_dependency_wait();
    using G = Gemm32Tile<TM, TN, NT>;
    constexpr int KC = G::KC, RM = G::RM, CN = G::CN, kStages = G::kStages;
    constexpr int kA = G::template a_floats<TA>(), kB = G::template b_floats<TB>();
    extern __shared__ __align__(16) float sm[];
    // the row at lane bit 0: both operands' 16-byte reads then meet their like at lane ^ 1 or ^ 2, two wavefronts instead of four
    const int tx = (threadIdx.x >> 1) & 15, ty = 2 * (threadIdx.x >> 5) + (threadIdx.x & 1);
    const int slice = blockIdx.z % g.slices, first = g.sum ? 0 : blockIdx.z / g.slices;
    const int terms = g.sum ? g.n : 1;
    const int M = g.p[first].M, N = g.p[first].N, K = g.p[first].K;
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    if (m0 >= M || n0 >= N) return;
    const int kbeg = slice * g.kper, kend = min(K, kbeg + g.kper);
    const int steps = (kend - kbeg + KC - 1) / KC, all = steps * terms;
    const bool vec = g.vec != 0;

    auto fetch = [&](int it) {
        if (it < all) {
            const Gemm32Problem& p = g.p[first + it / steps];
            const int k0 = kbeg + (it % steps) * KC;
            float* as = sm + (it % kStages) * (kA + kB);
            if constexpr (TA) load_block<KC, TM, NT>(as, p.A, p.lda, k0, kend, m0, M, vec);
            else load_block<TM, KC, NT>(as, p.A, p.lda, m0, M, k0, kend, vec);
            if constexpr (TB) load_block<TN, KC, NT>(as + kA, p.B, p.ldb, n0, N, k0, kend, vec);
            else load_block<KC, TN, NT>(as + kA, p.B, p.ldb, k0, kend, n0, N, vec);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // rows of this thread: VM neighbouring ones per group, groups VM * TY apart; columns: VN neighbouring ones, or (B
    // along the contraction, where neighbouring rows of the tile would meet in one bank) 16 apart
    constexpr int VN = TB ? 1 : G::VN;
    const int mr = G::VM * ty, nc = VN * tx;
    float acc[RM][CN], total[RM][CN];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < CN; ++j) { acc[i][j] = 0.f; total[i][j] = 0.f; }
#pragma unroll 1
    for (int s = 0; s < kStages - 1; ++s) fetch(s);
    for (int it = 0; it < all; ++it) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();
        fetch(it + kStages - 1);
        const float* as = sm + (it % kStages) * (kA + kB);
        const float* bs = as + kA;
#pragma unroll(TM <= 32 ? 1 : KC / 4)
        for (int k = 0; k < KC; k += 4) {
            Frag<!TA, RM, G::VM, G::VM * G::TY> a;
            Frag<TB, CN, VN, VN * 16> b;
            a.template load<TA ? TM + kPad : KC + kPad>(as, mr, k);
            b.template load<TB ? KC + kPad : TN + kPad>(bs, nc, k);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < RM; ++i)
#pragma unroll
                    for (int j = 0; j < CN; ++j) acc[i][j] = fmaf(a.v[e][i], b.v[e][j], acc[i][j]);
        }
        if (terms > 1 && (it + 1) % steps == 0) {
            const bool only = it + 1 == steps;
#pragma unroll
            for (int i = 0; i < RM; ++i)
#pragma unroll
                for (int j = 0; j < CN; ++j) {
                    total[i][j] = only ? acc[i][j] : total[i][j] + acc[i][j];
                    acc[i][j] = 0.f;
                }
        }
    }
    const Gemm32Problem& p = g.p[first];
    float* out = g.partial ? g.partial + g.part_off[first] + (int64_t)slice * M * N : p.C;
    const int ldo = g.partial ? N : p.ldc;
    const bool vec_out = !TB && G::VN == 4 && (ldo % 4) == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int gm = m0 + mr + (i / G::VM) * (G::VM * G::TY) + i % G::VM;
        if (gm >= M) continue;
        float v[CN];
#pragma unroll
        for (int j = 0; j < CN; ++j) {
            const int gn = n0 + nc + (j / VN) * (VN * 16) + j % VN;
            v[j] = terms > 1 ? total[i][j] : acc[i][j];
            if (p.bias && !g.partial && gn < N) v[j] += __ldg(p.bias + gn);
        }
        float* row = out + (int64_t)gm * ldo;
#pragma unroll
        for (int j = 0; j < CN; j += VN) {
            const int gn = n0 + nc + (j / VN) * (VN * 16);
            if (VN == 4 && vec_out && gn + 3 < N) {
                *reinterpret_cast<float4*>(row + gn) = make_float4(v[j], v[j + 1 < CN ? j + 1 : j], v[j + 2 < CN ? j + 2 : j], v[j + 3 < CN ? j + 3 : j]);
            } else {
#pragma unroll
                for (int e = 0; e < VN; ++e)
                    if (gn + e < N) row[gn + e] = v[j + e];
            }
        }
    }
}

// Small products whose sums may run in any order (gradients with respect to x and to the weights, the output projection):
// 32 x 32 tiles whose eight warps split every step of the contraction between them, each holding the whole tile (8 x 4
// outputs per thread), and add their shares at the end: a launch of a few such tiles is one chain of steps per CTA, and
// this makes the chain eight times shorter.  The loops are not unrolled: such a launch meets a cold instruction cache,
// and fetching straight-line code took longer than running it (B8 S32 E32 with 4 heads of 32: dx and the weight gradients
// 24 us as launches of their own, 11.5 unrolled with four warps, 10 rolled).  Two groups of products, of different operand
// forms, share a launch (the steps behind the attention backward).
constexpr int kSmallStages = 6, kSmallK = 32, kSmallWarps = 8, kSmallThreads = 32 * kSmallWarps;
struct Gemm32Pair {
    Gemm32Args g[2];
    int tiles_x[2], tiles_y[2], blocks[2];      // blocks[i] = tiles x products of group i
    int form[2];                                // 0: A [M,K] B [K,N];  1: A [M,K] B [N,K];  2: A [K,M] B [K,N]
};
constexpr int kSmallFloats = kSmallStages * 2 * 32 * (32 + kPad);

template <bool TA, bool TB>
__device__ __forceinline__ void small_product(const Gemm32Args& g, int tx0, int ty0, int z, float* sm) {
    constexpr int KC = kSmallK, KW = KC / kSmallWarps, LD = 32 + kPad, kTile = 32 * LD, S = kSmallStages;
    const int warp = threadIdx.x >> 5, tx = (threadIdx.x >> 1) & 7, ty = (threadIdx.x & 1) + 2 * ((threadIdx.x >> 4) & 1);
    const int first = g.sum ? 0 : z, terms = g.sum ? g.n : 1;
    const int M = g.p[first].M, N = g.p[first].N, K = g.p[first].K;
    const int m0 = ty0 * 32, n0 = tx0 * 32;
    if (m0 >= M || n0 >= N) return;
    const int steps = (K + KC - 1) / KC, all = steps * terms;
    const bool vec = g.vec != 0;
    auto fetch = [&](int it) {
        if (it < all) {
            const Gemm32Problem& p = g.p[first + it / steps];
            const int k0 = (it % steps) * KC;
            float* as = sm + (it % S) * 2 * kTile;
            if constexpr (TA) load_block<KC, 32, kSmallThreads>(as, p.A, p.lda, k0, K, m0, M, vec);
            else load_block<32, KC, kSmallThreads>(as, p.A, p.lda, m0, M, k0, K, vec);
            if constexpr (TB) load_block<32, KC, kSmallThreads>(as + kTile, p.B, p.ldb, n0, N, k0, K, vec);
            else load_block<KC, 32, kSmallThreads>(as + kTile, p.B, p.ldb, k0, K, n0, N, vec);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 1
    for (int s = 0; s < S - 1; ++s) fetch(s);
    for (int it = 0; it < all; ++it) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S - 2) : "memory");
        __syncthreads();
        fetch(it + S - 1);
        const float* as = sm + (it % S) * 2 * kTile;
#pragma unroll 1
        for (int k = 0; k < KW; k += 4) {
            Frag<!TA, 8, TA ? 4 : 1, TA ? 16 : 4> a;
            Frag<TB, 4, TB ? 1 : 4, TB ? 8 : 32> b;
            a.template load<LD>(as, TA ? 4 * ty : ty, warp * KW + k);
            b.template load<LD>(as + kTile, TB ? tx : 4 * tx, warp * KW + k);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a.v[e][i], b.v[e][j], acc[i][j]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = TA ? (i / 4) * 16 + 4 * ty + i % 4 : ty + 4 * i, c = TB ? tx + 8 * j : 4 * tx + j;
            sm[warp * kTile + r * LD + c] = acc[i][j];
        }
    __syncthreads();
    const Gemm32Problem& p = g.p[first];
    for (int e = threadIdx.x; e < 32 * 32; e += kSmallThreads) {
        const int r = e / 32, c = e % 32, gm = m0 + r, gn = n0 + c;
        if (gm >= M || gn >= N) continue;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < kSmallWarps; ++w) v += sm[w * kTile + r * LD + c];
        if (p.bias) v += __ldg(p.bias + gn);
        p.C[(int64_t)gm * p.ldc + gn] = v;
    }
}
__global__ void __launch_bounds__(kSmallThreads) gemm_fp32_small_kernel(const __grid_constant__ Gemm32Pair a) {
    grid_dependency_wait();
    extern __shared__ __align__(16) float sm[];
    const int grp = (int)blockIdx.x < a.blocks[0] ? 0 : 1;
    const int block = blockIdx.x - (grp ? a.blocks[0] : 0);
    const int x = block % a.tiles_x[grp], y = block / a.tiles_x[grp] % a.tiles_y[grp], z = block / (a.tiles_x[grp] * a.tiles_y[grp]);
    if (a.form[grp] == 0) small_product<false, false>(a.g[grp], x, y, z, sm);
    else if (a.form[grp] == 1) small_product<false, true>(a.g[grp], x, y, z, sm);
    else small_product<true, false>(a.g[grp], x, y, z, sm);
}

// C[m][n] = sum over slices, in slice order, of the partial results; blockIdx.y picks the product.
__global__ void __launch_bounds__(256) gemm_fp32_reduce_kernel(const __grid_constant__ Gemm32Args g) {
    grid_dependency_wait();
    const Gemm32Problem& p = g.p[blockIdx.y];
    const int64_t mn = (int64_t)p.M * p.N;
    const float* src = g.partial + g.part_off[blockIdx.y];
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < mn; i += (int64_t)gridDim.x * 256) {
        float v = 0.f;
        for (int z = 0; z < g.slices; ++z) v += src[(int64_t)z * mn + i];
        p.C[(i / p.N) * p.ldc + (i % p.N)] = v;
    }
}

template <bool TA, bool TB, int TM, int TN, int NT>
int launch(ltca_ctx* ctx, const Gemm32Args& g, int max_m, int max_n) {
    using G = Gemm32Tile<TM, TN, NT>;
    constexpr int smem = G::kStages * (G::template a_floats<TA>() + G::template b_floats<TB>()) * (int)sizeof(float);
    static SmemOptIn once;
    if (smem > 48 * 1024) LTCA_CUDA_OK(ctx, opt_in_dynamic_smem(once, ctx->device, gemm_fp32_kernel<TA, TB, TM, TN, NT>, smem));
    dim3 grid((max_n + TN - 1) / TN, (max_m + TM - 1) / TM, (g.sum ? 1 : g.n) * g.slices);
    LTCA_CUDA_OK(ctx, launch_dependent(gemm_fp32_kernel<TA, TB, TM, TN, NT>, grid, dim3(NT), smem, ctx->stream, g));
    return LTCA_OK;
}

template <bool TA, bool TB>
int launch_tile(ltca_ctx* ctx, const Gemm32Args& g, int tile, int max_m, int max_n) {
    if (tile == 128) return launch<TA, TB, 128, 128, 256>(ctx, g, max_m, max_n);
    if (tile == 64) return launch<TA, TB, 64, 64, 128>(ctx, g, max_m, max_n);
    return launch<TA, TB, 32, 32, 128>(ctx, g, max_m, max_n);
}

// Tile, slices and operand checks of one group of products.
struct Plan32 {
    Gemm32Args g;
    int tile, max_m, max_n;
    int64_t tiles32;        // 32 x 32 tiles of the launch
};
int plan_gemm(ltca_ctx* ctx, Plan32* pl, const Gemm32Problem* p, int n, bool sum, float* scratch, size_t scratch_bytes) {
    if (n < 1 || n > kMaxGemm32) return fail(ctx, LTCA_ERR_INVALID, "gemm_fp32 takes 1 to %d products", kMaxGemm32);
    Gemm32Args& g = pl->g;
    memset(&g, 0, sizeof(g));
    g.n = n;
    g.sum = sum && n > 1 ? 1 : 0;
    g.slices = 1;
    g.kper = p[0].K;
    bool vec = true;
    int max_m = 0, max_n = 0;
    int64_t cells = 0;
    for (int i = 0; i < n; ++i) {
        g.p[i] = p[i];
        vec = vec && !(p[i].lda % 4) && !(p[i].ldb % 4) && !((reinterpret_cast<uintptr_t>(p[i].A) | reinterpret_cast<uintptr_t>(p[i].B)) & 15);
        if (p[i].M > max_m) max_m = p[i].M;
        if (p[i].N > max_n) max_n = p[i].N;
        cells += (int64_t)p[i].M * p[i].N;
        if (p[i].K != p[0].K) return fail(ctx, LTCA_ERR_INVALID, "gemm_fp32: one contraction length per launch");
    }
    g.vec = vec ? 1 : 0;
    const int K = p[0].K, sms = ctx->sm_device > 0 ? ctx->sm_device : kPlanSms;
    auto tiles = [&](int t) {
        int64_t c = 0;
        for (int i = 0; i < (g.sum ? 1 : n); ++i) c += (int64_t)((p[i].M + t - 1) / t) * ((p[i].N + t - 1) / t);
        return c;
    };
    // The largest tile whose CTAs occupy the SMs: reuse grows with the tile (8 x 8 outputs per thread at 128, 4 x 2 at
    // 32), but a launch of fewer CTAs than SMs lasts as long as one CTA.  A product that may be sliced counts its
    // slices of at least 256 contraction steps as CTAs.
    const int64_t most = scratch ? (int64_t)(scratch_bytes / sizeof(float)) / (cells > 0 ? cells : 1) : 1;
    auto slices_for = [&](int t) {
        int64_t s = (2 * sms + tiles(t) - 1) / tiles(t);
        if (s > K / 256) s = K / 256;
        if (s > most) s = most;
        return s < 1 ? (int64_t)1 : s;
    };
    int tile = 32;
    if (tiles(128) * slices_for(128) * 4 >= 3 * sms) tile = 128;
    else if (tiles(64) * slices_for(64) * 4 >= 3 * sms) tile = 64;
    if (scratch && !g.sum) {
        const int64_t s = slices_for(tile);
        if (s > 1) {
            g.kper = (int)(((K + s - 1) / s + 31) / 32 * 32);
            g.slices = (K + g.kper - 1) / g.kper;
            if (g.slices > 1) {
                for (int i = 0; i < n; ++i)
                    if (p[i].bias) return fail(ctx, LTCA_ERR_INVALID, "gemm_fp32: a sliced contraction takes no bias");
                g.partial = scratch;
                int64_t off = 0;
                for (int i = 0; i < n; ++i) { g.part_off[i] = off; off += (int64_t)g.slices * p[i].M * p[i].N; }
            }
        }
    }
    pl->tile = tile;
    pl->max_m = max_m;
    pl->max_n = max_n;
    pl->tiles32 = tiles(32);
    return LTCA_OK;
}

int launch_plan(ltca_ctx* ctx, const Plan32& pl, int ta, int tb) {
    const Gemm32Args& g = pl.g;
    int rc;
    if (!ta && !tb) rc = launch_tile<false, false>(ctx, g, pl.tile, pl.max_m, pl.max_n);
    else if (!ta && tb) rc = launch_tile<false, true>(ctx, g, pl.tile, pl.max_m, pl.max_n);
    else if (ta && !tb) rc = launch_tile<true, false>(ctx, g, pl.tile, pl.max_m, pl.max_n);
    else return fail(ctx, LTCA_ERR_UNSUPPORTED, "gemm_fp32: A stored [K, M] with B stored [N, K] is not built");
    if (rc || !g.partial) return rc;
    int64_t mn = 0;
    for (int i = 0; i < g.n; ++i) if ((int64_t)g.p[i].M * g.p[i].N > mn) mn = (int64_t)g.p[i].M * g.p[i].N;
    const int64_t blocks = (mn + 255) / 256, most = 8 * (ctx->sm_device > 0 ? ctx->sm_device : kPlanSms);
    LTCA_CUDA_OK(ctx, launch_dependent(gemm_fp32_reduce_kernel, dim3((unsigned)(blocks < most ? blocks : most), g.n), dim3(256), 0,
                                       ctx->stream, g));
    return LTCA_OK;
}

// Launches one or two groups of small products (see gemm_fp32_small_kernel).
int launch_small(ltca_ctx* ctx, const Plan32* pl, const int* form, int groups) {
    Gemm32Pair a;
    memset(&a, 0, sizeof(a));
    for (int i = 0; i < groups; ++i) {
        a.g[i] = pl[i].g;
        a.tiles_x[i] = (pl[i].max_n + 31) / 32;
        a.tiles_y[i] = (pl[i].max_m + 31) / 32;
        a.blocks[i] = a.tiles_x[i] * a.tiles_y[i] * (a.g[i].sum ? 1 : a.g[i].n);
        a.form[i] = form[i];
    }
    constexpr int smem = kSmallFloats * (int)sizeof(float);
    static SmemOptIn once;
    LTCA_CUDA_OK(ctx, opt_in_dynamic_smem(once, ctx->device, gemm_fp32_small_kernel, smem));
    LTCA_CUDA_OK(ctx, launch_dependent(gemm_fp32_small_kernel, dim3((unsigned)(a.blocks[0] + a.blocks[1])), dim3(kSmallThreads), smem, ctx->stream, a));
    return LTCA_OK;
}
// 32-wide tiles and an unsliced contraction: the launch is a chain of latencies.
bool small_plan(const Plan32& pl) { return pl.tile == 32 && pl.g.slices == 1; }

}  // namespace

int gemm_fp32(ltca_ctx* ctx, const Gemm32Problem* p, int n, int ta, int tb, bool sum, bool any_order, float* scratch,
              size_t scratch_bytes) {
    Plan32 pl;
    if (int rc = plan_gemm(ctx, &pl, p, n, sum, scratch, scratch_bytes)) return rc;
    const int form = ta ? 2 : tb ? 1 : 0;
    if (any_order && small_plan(pl) && !(ta && tb)) return launch_small(ctx, &pl, &form, 1);
    return launch_plan(ctx, pl, ta, tb);
}

int gemm_fp32_grads(ltca_ctx* ctx, const Gemm32Problem* dx, int n_dx, const Gemm32Problem* dw, int n_dw, float* scratch,
                    size_t scratch_bytes) {
    Plan32 pl[2];
    int rc;
    if ((rc = plan_gemm(ctx, &pl[0], dx, n_dx, true, nullptr, 0))) return rc;
    if ((rc = plan_gemm(ctx, &pl[1], dw, n_dw, false, scratch, scratch_bytes))) return rc;
    if (small_plan(pl[0]) && small_plan(pl[1])) {
        const int form[2] = {1, 2};
        return launch_small(ctx, pl, form, 2);
    }
    if ((rc = gemm_fp32(ctx, dx, n_dx, 0, 1, true, true))) return rc;
    return gemm_fp32(ctx, dw, n_dw, 1, 0, false, true, scratch, scratch_bytes);
}

}  // namespace ltca
