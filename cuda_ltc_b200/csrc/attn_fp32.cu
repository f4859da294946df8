// fp32 attention: the exact arithmetic mode (fp32 FMA, accurate expf) and the path for every
// shape the tensor-pipe kernels do not take (any head_dim up to 512, dense keep-masks, tiny
// sequences).  Forward and backward (one pass over the scores or two, no atomics, bit-reproducible).
//
// Replaces flashAttentionKernel (reference src/ml/flash_attention.cu:18-272) on its own valid
// domain (head_dim <= 16, one key tile) and extends it to a true online softmax for longer
// sequences; the score tiles keep one query row inside sixteen lanes so that row maxima
// and row sums are shuffle reductions.
#include <math.h>

#include "attn_mask.cuh"
#include "host_common.h"
#include "sm100_ptx.cuh"

namespace ltca {

namespace {

constexpr float kNegInf = -INFINITY;

__device__ __forceinline__ float ld_elem(const float* p) { return __ldg(p); }
__device__ __forceinline__ float ld_elem(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ void st_elem(float* p, float v) { *p = v; }
__device__ __forceinline__ void st_elem(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

struct CoreArgs {
    int B, H, Sq, Sk, D;
    int causal, causal_off;
    float scale, clamp;
    int use_clamp;
    const void *q, *k, *v, *o_in, *dout;
    void *o, *dq, *dk, *dv;
    ltca_strides qs, ks, vs, os, dos, dqs, dks, dvs;
    float* lse;
    const float* lse_in;
    float* delta;
    const float* keep_mask;
    const int32_t* kv_len;
    const uint32_t* mask_bits;  // backward: the dense mask packed, [B, Sq, mask_nw]; null: no room for it
    int mask_nw;
    float* dq_part;             // one-pass backward: dQ of every key block, [key blocks][pairs of the launch][Sq][part_ld]
    int part_ld, pair0, pairs;  // (batch, head) pairs of the launch: pair0 .. pair0 + pairs
    // dO is not there yet, it is dy Wo_h^T (see FromOutput); the two-kernel backward's first kernel writes dO's rows for the second
    const float *dy, *wo;
    int64_t dy_batch, dy_seq;
    int E;
    int vec;            // every row starts on a 16-byte (fp32) or 8-byte (bf16) boundary and holds a multiple of 4 elements
};

// The products of these kernels take packed fp32 pairs: they are bound by issue slots (loads, masks and exponentials share
// them with the multiply-adds), so halving the number of multiply-add instructions is worth the second accumulator.

// 16-byte asynchronous copy global -> shared; nothing is read and zeros are written when `bytes` is 0.
__device__ __forceinline__ void cp_async16(float* dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float4 ld4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 ld4(const __nv_bfloat16* p) {
    const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
    const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
    const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    return make_float4(x.x, x.y, y.x, y.y);
}
// Four elements of a row from column d on; zeros beyond D.
template <typename T>
__device__ __forceinline__ float4 row4(const T* row, int d, int D, bool vec) {
    if (vec) return d < D ? ld4(row + d) : make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(d < D ? ld_elem(row + d) : 0.f, d + 1 < D ? ld_elem(row + d + 1) : 0.f,
                       d + 2 < D ? ld_elem(row + d + 2) : 0.f, d + 3 < D ? ld_elem(row + d + 3) : 0.f);
}
template <typename T>
__device__ __forceinline__ void store4(T* row, int d, int D, float4 v, bool vec) {
    if (vec) {
        if (d >= D) return;
        if constexpr (sizeof(T) == 4) {
            *reinterpret_cast<float4*>(row + d) = v;
        } else {
            const __nv_bfloat162 x = __floats2bfloat162_rn(v.x, v.y), y = __floats2bfloat162_rn(v.z, v.w);
            *reinterpret_cast<uint2*>(row + d) =
                make_uint2(*reinterpret_cast<const uint32_t*>(&x), *reinterpret_cast<const uint32_t*>(&y));
        }
    } else {
        if (d < D) st_elem(row + d, v.x);
        if (d + 1 < D) st_elem(row + d + 1, v.y);
        if (d + 2 < D) st_elem(row + d + 2, v.z);
        if (d + 3 < D) st_elem(row + d + 3, v.w);
    }
}

// How the backward kernels meet a dense mask: not at all, as packed words, or as it is (a workspace sized without the mask has no
// room for the words; short one-pass calls).
constexpr int kNoMask = 0, kWords = 1, kDense = 2;
// Word w of query qi's row: bit c = key 32 w + c is kept; 0 beyond the tensor.
template <int kMask>
__device__ __forceinline__ uint32_t mask_word(const CoreArgs& a, int b, int qi, int w) {
    if (qi >= a.Sq || w >= a.mask_nw) return 0u;
    const int64_t row = (int64_t)b * a.Sq + qi;
    if constexpr (kMask == kWords) return a.mask_bits[row * a.mask_nw + w];
    const float* m = a.keep_mask + row * a.Sk + 32 * w;
    const int n = min(32, a.Sk - 32 * w);
    uint32_t bits = 0;
#pragma unroll 1
    for (int c = 0; c < n; ++c) bits |= (__ldg(m + c) != 0.f ? 1u : 0u) << c;
    return bits;
}

__device__ __forceinline__ bool key_visible(const CoreArgs& a, int b, int qi, int kj, int kvlen) {
    if (kj >= kvlen) return false;
    if (a.causal && kj > qi + a.causal_off) return false;
    if (a.keep_mask && qi < a.Sq && a.keep_mask[((int64_t)b * a.Sq + qi) * a.Sk + kj] == 0.f)
        return false;
    return true;
}

// ----------------------------------------------------------------------------------------------
// Score tiles of 64 (16 for calls with few rows) query rows x 64 keys for head_dim up to 128.
//
// A thread multiplies a block of 8 rows x 4 columns of a score tile, P (and dS) go through shared memory into the
// accumulating products, whose threads hold 4 neighbouring columns of several rows.  Both read their operands as 16-byte
// vectors along the contraction: a quarter of the shared-memory instructions of one word per operand, which is what
// bounded these kernels before (1 read per 2 multiply-adds; now 12 per 128 and 8 per 64).  The sums run in the
// same order as with one word per read, so tiles of both heights and every launch width give the same bits.
// Measured at B16 H8 S250 D32 with a dense mask: forward 93 -> 48 us, backward 305 -> 174 us; at D64 without a mask, both
// 640 -> 336 us; the smallest calls (tiles of 16 rows) 10.7 -> 4 us.  What bounds them now is the issue rate: half of the
// instructions are multiply-adds, the rest masks, exponentials and reads, at 12 to 16 warps per SM (registers).
// One (query or key) row per lane group with the other side's rows broadcast from shared memory was built as well:
// fewer instructions, but a broadcast 16-byte read takes two wavefronts and the row state leaves two or three warps per
// scheduler; the same times within 5 % (without the mask forward 41 against 44 us, backward 167 against 162).
// ----------------------------------------------------------------------------------------------
constexpr int kOnePassThreads64 = 256;     // threads of the one-pass backward's CTA at DP = 64
constexpr int kPad = 4;      // floats added to a shared row: neighbouring rows' 16-byte pieces lie in different banks

// Rows [r0, r0 + ROWS) into shared [ROWS][DP + kPad]; see load_tile.
template <int DP, int ROWS, int NT, typename T>
__device__ __forceinline__ void load_padded(float* dst, const T* base, int64_t row_stride, int r0, int rows_total, int D, bool vec) {
    constexpr int C4 = DP / 4, LD = DP + kPad;
#pragma unroll
    for (int e0 = 0; e0 < ROWS * C4; e0 += NT) {
        const int e = e0 + threadIdx.x;
        if (ROWS * C4 % NT != 0 && e >= ROWS * C4) break;
        const int r = e / C4, c = (e % C4) * 4;
        const bool in = r0 + r < rows_total && c < D;
        const T* src = base + (int64_t)(r0 + r) * row_stride;
        if constexpr (sizeof(T) == 4) {
            if (vec) {
                cp_async16(dst + r * LD + c, in ? src + c : base, in ? 16 : 0);
                continue;
            }
        }
        *reinterpret_cast<float4*>(dst + r * LD + c) = in ? row4(src, c, D, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

// Lanes.  A 16-byte shared read takes two wavefronts where every lane shares its address with lane ^ 1 or lane ^ 2, and four
// where the lanes that share one lie further apart (measured: 2.1 and 4.0 cycles an SM, however few addresses there are).  So
// the two sides of every product below alternate at the lowest lane bits: bit 0 picks the row, bit 1 the column.
// With the row at bit 4 and with it at bit 0, us: tiles of 16 rows, B4 H4 S512 D32 forward 40 and 30, backward 136 and 103; tiles
// of 64 rows, B16 H8 S250 backward D16 92 and 83, D32 135 and 130.
//
// Thread layout of the score products: NT threads as (NT / 16) x 16.  Thread (ty, tx) owns columns tx + 16 j and rows
// row_of(ty) + (NT / 16) i; the two rows that a warp holds per i lie four apart, which puts their words in different banks.
__device__ __forceinline__ int score_tx() { return (threadIdx.x >> 1) & 15; }
__device__ __forceinline__ int score_ty() { return 2 * (threadIdx.x >> 5) + (threadIdx.x & 1); }
__device__ __forceinline__ int row_of(int ty) { return ((ty >> 1) & 3) + 4 * (ty & 1) + 8 * (ty >> 3); }

// s[i][j] = A[row i] . B[col j] over DP features
template <int DP, int NT, int RM, int CN, int kUnroll = 2>
__device__ __forceinline__ void tile_dot(float (&s)[RM][CN], const float* A, const float* B, int row0, int tx) {
    constexpr int LD = DP + kPad, RS = NT / 16;
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < CN; ++j) s[i][j] = 0.f;
#pragma unroll kUnroll
    for (int d = 0; d < DP; d += 4) {
        float4 b[CN];
#pragma unroll
        for (int j = 0; j < CN; ++j) b[j] = *reinterpret_cast<const float4*>(B + (tx + 16 * j) * LD + d);
#pragma unroll
        for (int i = 0; i < RM; ++i) {
            const float4 x = *reinterpret_cast<const float4*>(A + (row0 + RS * i) * LD + d);
#pragma unroll
            for (int j = 0; j < CN; ++j) {
                s[i][j] = fmaf(x.x, b[j].x, s[i][j]);
                s[i][j] = fmaf(x.y, b[j].y, s[i][j]);
                s[i][j] = fmaf(x.z, b[j].z, s[i][j]);
                s[i][j] = fmaf(x.w, b[j].w, s[i][j]);
            }
        }
    }
}

// Thread layout of the accumulating products: a [ROWS, DP] result, 4 columns (8 at DP = 128: two groups 64 apart) and
// NR rows per thread.
template <int DP, int ROWS, int NT>
struct AccLayout {
    static constexpr int TX = DP < 64 ? DP / 4 : 16;            // threads across the columns
    static constexpr int CG = DP / (4 * TX);                    // column groups of 4 per thread
    static constexpr int TY = NT / TX < ROWS ? NT / TX : ROWS;  // threads down the rows (the others idle)
    static constexpr int NR = ROWS / TY;
    int tx, ty;
    bool active;
    __device__ __forceinline__ AccLayout() {
        tx = (threadIdx.x & 31) / 2 % TX;
        ty = 32 / TX * (threadIdx.x / 32) + 2 * ((threadIdx.x & 31) / 2 / TX) + threadIdx.x % 2;
        active = ty < TY;
    }
};
// acc[row][cols] += sum over j < n of A[row][j] * V[j][cols], j ascending; A has row pitch LA, n is a multiple of 4 (zeros
// beyond).
template <int DP, int ROWS, int NT>
__device__ __forceinline__ void accumulate(f32x2 (&acc)[AccLayout<DP, ROWS, NT>::NR][2 * AccLayout<DP, ROWS, NT>::CG],
                                           const AccLayout<DP, ROWS, NT>& L, const float* A, int LA, const float* V, int n) {
    using Lt = AccLayout<DP, ROWS, NT>;
    constexpr int LD = DP + kPad;
#pragma unroll 2
    for (int j = 0; j < n; j += 4) {
        float4 x[Lt::NR];
#pragma unroll
        for (int i = 0; i < Lt::NR; ++i) x[i] = *reinterpret_cast<const float4*>(A + (L.ty + Lt::TY * i) * LA + j);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int c = 0; c < Lt::CG; ++c) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(V + (j + e) * LD + 4 * L.tx + 64 * c);
#pragma unroll
                for (int i = 0; i < Lt::NR; ++i) {
                    const float w = e == 0 ? x[i].x : e == 1 ? x[i].y : e == 2 ? x[i].z : x[i].w;
                    const f32x2 ww = pair(w, w);
                    acc[i][2 * c] = fma2(ww, v.x, acc[i][2 * c]);
                    acc[i][2 * c + 1] = fma2(ww, v.y, acc[i][2 * c + 1]);
                }
            }
    }
}
template <int NR>
__device__ __forceinline__ void ld_row(float (&x)[NR], const float* p) {       // NR consecutive floats of a shared row
    if constexpr (NR % 4 == 0) {
#pragma unroll
        for (int i = 0; i < NR; i += 4) {
            const float4 v = *reinterpret_cast<const float4*>(p + i);
            x[i] = v.x; x[i + 1] = v.y; x[i + 2] = v.z; x[i + 3] = v.w;
        }
    } else if constexpr (NR == 2) {
        const float2 v = *reinterpret_cast<const float2*>(p);
        x[0] = v.x; x[1] = v.y;
    } else {
        x[0] = *p;
    }
}

// Visibility of the CN columns k + 16 j of a row whose last visible key (without the mask) is `last`: bit j.
template <int CN>
__device__ __forceinline__ uint32_t row_limit(int k, int last) {
    uint32_t bits = 0;
#pragma unroll
    for (int j = 0; j < CN; ++j) bits |= (k + 16 * j <= last ? 1u : 0u) << j;
    return bits;
}
// The same columns of a row of mask bits (`words`: 32 keys each, from the tile's first key on).
template <int CN>
__device__ __forceinline__ uint32_t row_mask(const uint32_t* words, int tx) {
    uint32_t bits = 0;
#pragma unroll
    for (int j = 0; j < CN; ++j) bits |= (words[j / 2] >> (tx + 16 * (j % 2)) & 1u) << j;
    return bits;
}
// over a row's 16 threads (score_tx)
__device__ __forceinline__ float row_max(float v) {
#pragma unroll
    for (int o = 16; o > 1; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float row_sum(float v) {
#pragma unroll
    for (int o = 16; o > 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ----------------------------------------------------------------------------------------------
// forward: one CTA per TM query rows of a (batch, head) pair, 64 keys per step
//
// K arrives for the next step under the value product, V under the next scores; several CTAs per SM cover the rest.
// ----------------------------------------------------------------------------------------------
template <typename T, int DP, int TM, int NT, bool kMask>
__global__ void __launch_bounds__(NT, TM < 64 ? 4 : DP <= 32 ? 4 : DP <= 64 ? 3 : 1) attn_fwd_fp32_kernel(const CoreArgs a) {
    grid_dependency_wait();
    constexpr int KN = 64, LD = DP + kPad, LP = KN + kPad, RS = NT / 16, RM = TM / RS, CN = KN / 16;
    using Lt = AccLayout<DP, TM, NT>;
    extern __shared__ __align__(16) float sm[];
    float* Qs = sm;
    float* Ks = Qs + TM * LD;
    float* Vs = Ks + KN * LD;
    float* Ps = Vs + KN * LD;
    float* row_scale = Ps + TM * LP;     // [TM]: what the accumulator is multiplied with (step), 1 / sum (end)
    const bool vec = a.vec != 0;

    const int tx = score_tx(), row0 = row_of(score_ty());
    const int q0 = blockIdx.x * TM;
    const int h = blockIdx.y, b = blockIdx.z;
    int kvlen = a.Sk;
    if (a.kv_len) kvlen = min(max(a.kv_len[b], 0), a.Sk);
    int k_end = kvlen;
    if (a.causal) k_end = min(k_end, min(q0 + TM - 1, a.Sq - 1) + a.causal_off + 1);

    const T* qb = reinterpret_cast<const T*>(a.q) + b * a.qs.batch + h * a.qs.head;
    const T* kb = reinterpret_cast<const T*>(a.k) + b * a.ks.batch + h * a.ks.head;
    const T* vb = reinterpret_cast<const T*>(a.v) + b * a.vs.batch + h * a.vs.head;
    load_padded<DP, TM, NT>(Qs, qb, a.qs.seq, q0, a.Sq, a.D, vec);
    load_padded<DP, KN, NT>(Ks, kb, a.ks.seq, 0, a.Sk, a.D, vec);
    cp_async_commit();
    load_padded<DP, KN, NT>(Vs, vb, a.vs.seq, 0, a.Sk, a.D, vec);
    cp_async_commit();

    // Dense mask: every warp votes its share of the next step's words (32 keys of a row each) in two halves.  64-row tiles of heads up to
    // 32 (kEarly) read one under the score product and the other under the value product, into one of two sets of words; others the
    // first under the value product and the second behind it, under the wait for the next keys.  (us, late and early: B64 H8 S128 D32
    // 44.9 and 43.2, B16 H8 S250 D32 47.1 and 45.7, D16 33.8 and 33.3, D64 83.7 and 83.3, B24 H8 S200 D64 105.9 and 106.7, B2 H4 S200 D64
    // in 16-row tiles 13.0 and 13.3.  Both halves under the value product: spills at D32, 4 % slower.)
    constexpr bool kEarly = TM == 64 && DP <= 32;
    constexpr int kWords2 = TM / (NT / 32);                               // words of half a warp's rows
    uint32_t* mask_sm = reinterpret_cast<uint32_t*>(row_scale + TM);      // [TM][2], kEarly: of two steps
    const int lane = threadIdx.x & 31, mask_row = (threadIdx.x >> 5) * kWords2;
    float mv[kWords2];
    static_assert(kWords2 % 2 == 0, "whole rows");
    auto mask_read = [&](float (&mv)[kWords2], int half, int k) {
        const int r0 = q0 + mask_row + half * (kWords2 / 2);
        const float* p = a.keep_mask + ((int64_t)b * a.Sq + r0) * a.Sk + k + lane;
#pragma unroll
        for (int w = 0; w < kWords2; w += 2, p += a.Sk) {
            const bool row = r0 + w / 2 < a.Sq;
            mv[w] = row && k + lane < k_end ? __ldg(p) : 0.f;
            mv[w + 1] = row && k + 32 + lane < k_end ? __ldg(p + 32) : 0.f;
        }
    };
    auto mask_vote = [&](const float (&mv)[kWords2], uint32_t* words, int half) {
#pragma unroll
        for (int w = 0; w < kWords2; w += 2) {
            const uint32_t x = __ballot_sync(0xffffffffu, mv[w] != 0.f), y = __ballot_sync(0xffffffffu, mv[w + 1] != 0.f);
            if (lane == 0) *reinterpret_cast<uint2*>(words + 2 * mask_row + half * kWords2 + w) = make_uint2(x, y);
        }
    };
    if (kMask) {
        float first[kWords2];                                             // the first step's halves in flight together
        mask_read(first, 0, 0);
        mask_read(mv, 1, 0);
        mask_vote(first, mask_sm, 0);
        if (kEarly) mask_vote(mv, mask_sm, 1);
    }

    const Lt L;
    float m_run[RM], l_run[RM];
    f32x2 acc[Lt::NR][2 * Lt::CG];
#pragma unroll
    for (int i = 0; i < RM; ++i) { m_run[i] = kNegInf; l_run[i] = 0.f; }
#pragma unroll
    for (int i = 0; i < Lt::NR; ++i)
#pragma unroll
        for (int c = 0; c < 2 * Lt::CG; ++c) acc[i][c] = 0ull;

    for (int k0 = 0; k0 < k_end; k0 += KN) {
        const bool more = k0 + KN < k_end;
        uint32_t* mask_now = mask_sm + (kEarly ? (k0 / KN & 1) * (2 * TM) : 0);
        uint32_t* mask_next = mask_sm + (kEarly ? ((k0 / KN + 1) & 1) * (2 * TM) : 0);
        if (kMask && kEarly && more) mask_read(mv, 0, k0 + KN);
        cp_async_wait<1>();
        if (kMask && !kEarly) mask_vote(mv, mask_now, 1);
        __syncthreads();
        float s[RM][CN];
        tile_dot<DP, NT, RM, CN, TM == 64 && (kMask || DP >= 32) ? 1 : 2>(s, Qs, Ks, row0, tx);      // (two at a time spill there)
        if (kMask && kEarly && more) mask_vote(mv, mask_next, 0);
        const bool all_visible = k0 + KN <= kvlen && !kMask && (!a.causal || k0 + KN - 1 <= q0 + a.causal_off);
#pragma unroll
        for (int i = 0; i < RM; ++i) {
            const int r = row0 + RS * i;
            uint32_t visible = ~0u;
            if (!all_visible) {
                const int last = a.causal ? min(kvlen - 1, q0 + r + a.causal_off) : kvlen - 1;
                visible = row_limit<CN>(k0 + tx, last);
                if (kMask) visible &= row_mask<CN>(mask_now + 2 * r, tx);
            }
            float mt = kNegInf;
#pragma unroll
            for (int j = 0; j < CN; ++j) {
                float v = s[i][j] * a.scale;
                if (a.use_clamp) v = fminf(v, a.clamp);
                if (!(visible >> j & 1u)) v = kNegInf;
                s[i][j] = v;
                mt = fmaxf(mt, v);
            }
            mt = row_max(mt);
            const float m_new = fmaxf(m_run[i], mt);
            const float m_safe = (m_new == kNegInf) ? 0.f : m_new;
            const float corr = (m_run[i] == kNegInf) ? 0.f : expf(m_run[i] - m_safe);
            float rs = 0.f;
#pragma unroll
            for (int j = 0; j < CN; ++j) {
                const float p = expf(s[i][j] - m_safe);      // exp(-inf) = 0 for hidden keys
                Ps[r * LP + tx + 16 * j] = p;
                rs += p;
            }
            rs = row_sum(rs);
            l_run[i] = l_run[i] * corr + rs;
            m_run[i] = m_new;
            if (tx == 0) row_scale[r] = corr;
        }
        if (kMask && kEarly && more) mask_read(mv, 1, k0 + KN);
        cp_async_wait<0>();
        __syncthreads();
        if (kMask && !kEarly && more) mask_read(mv, 0, k0 + KN);
        if (more) load_padded<DP, KN, NT>(Ks, kb, a.ks.seq, k0 + KN, a.Sk, a.D, vec);
        cp_async_commit();
        if (L.active) {
#pragma unroll
            for (int i = 0; i < Lt::NR; ++i) {
                const float corr = row_scale[L.ty + Lt::TY * i];
                const f32x2 cc = pair(corr, corr);
#pragma unroll
                for (int c = 0; c < 2 * Lt::CG; ++c) acc[i][c] = mul2(acc[i][c], cc);
            }
            accumulate<DP, TM, NT>(acc, L, Ps, LP, Vs, min(KN, (k_end - k0 + 3) & ~3));
        }
        if (kMask && kEarly && more) mask_vote(mv, mask_next, 1);
        if (kMask && !kEarly && more) {
            mask_vote(mv, mask_next, 0);
            mask_read(mv, 1, k0 + KN);
        }
        __syncthreads();
        if (more) load_padded<DP, KN, NT>(Vs, vb, a.vs.seq, k0 + KN, a.Sk, a.D, vec);
        cp_async_commit();
    }
    cp_async_wait<0>();

#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int r = row0 + RS * i, qi = q0 + r;
        if (tx == 0) {
            row_scale[r] = l_run[i] > 0.f ? 1.f / l_run[i] : 0.f;
            if (a.lse && qi < a.Sq)
                a.lse[((int64_t)b * a.H + h) * a.Sq + qi] = l_run[i] > 0.f ? m_run[i] + logf(l_run[i]) : kNegInf;
        }
    }
    __syncthreads();
    if (!L.active) return;
    T* ob = reinterpret_cast<T*>(a.o) + b * a.os.batch + h * a.os.head;
#pragma unroll
    for (int i = 0; i < Lt::NR; ++i) {
        const int r = L.ty + Lt::TY * i;
        if (q0 + r >= a.Sq) continue;
        const float inv = row_scale[r];
#pragma unroll
        for (int c = 0; c < Lt::CG; ++c) {
            const float2 x = halves(acc[i][2 * c]), y = halves(acc[i][2 * c + 1]);
            store4(ob + (int64_t)(q0 + r) * a.os.seq, 4 * L.tx + 64 * c, a.D, make_float4(x.x * inv, x.y * inv, y.x * inv, y.y * inv),
                   vec);
        }
    }
}

// ----------------------------------------------------------------------------------------------
// backward helper of the wide-head kernels: delta[b,h,i] = sum_d dO[i,d] * O[i,d]   (one warp per query row)
// ----------------------------------------------------------------------------------------------
template <typename T>
__global__ void attn_bwd_delta_kernel(const CoreArgs a) {
    const int warps_per_block = blockDim.x >> 5;
    const int64_t row = (int64_t)blockIdx.x * warps_per_block + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    const int64_t total = (int64_t)a.B * a.H * a.Sq;
    if (row >= total) return;
    const int qi = (int)(row % a.Sq);
    const int64_t bh = row / a.Sq;
    const int h = (int)(bh % a.H), b = (int)(bh / a.H);
    const T* o = reinterpret_cast<const T*>(a.o_in) + b * a.os.batch + h * a.os.head + (int64_t)qi * a.os.seq;
    const T* g = reinterpret_cast<const T*>(a.dout) + b * a.dos.batch + h * a.dos.head + (int64_t)qi * a.dos.seq;
    float acc = 0.f;
    for (int d = lane; d < a.D; d += 32) acc = fmaf(ld_elem(o + d), ld_elem(g + d), acc);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) a.delta[row] = acc;
}

// ----------------------------------------------------------------------------------------------
// backward
// ----------------------------------------------------------------------------------------------
// dst[r][c] = dO[r0 + r][c] = sum over e of dy[r0 + r][e] Wo[h D + c][e], e ascending as in the product that this replaces, also
// written to dO's rows.  A thread keeps a row of Wo's head for its column c and goes down the tile's rows, whose dy its warp
// reads at one address.  kRows: dO's rows are written as well.
template <int DP, int ROWS, int NT, bool kRows>
__device__ __forceinline__ void form_dout(float* dst, const CoreArgs& a, int b, int h, int r0) {
    constexpr int LD = DP + kPad, RT = NT / DP, NR = ROWS / RT;
    const int c = threadIdx.x % DP, rt = threadIdx.x / DP;
    const float* w = a.wo + ((int64_t)h * a.D + min(c, a.D - 1)) * a.E;
    const float* d = a.dy + b * a.dy_batch;
    float g[NR];
#pragma unroll
    for (int i = 0; i < NR; ++i) g[i] = 0.f;
    for (int e = 0; e < a.E; e += 8) {                         // (a multiple of 8)
        const float4 w0 = ld4(w + e), w1 = ld4(w + e + 4);
#pragma unroll
        for (int i = 0; i < NR; ++i) {
            const float* row = d + (int64_t)min(r0 + rt + RT * i, a.Sq - 1) * a.dy_seq + e;
            const float4 x0 = ld4(row), x1 = ld4(row + 4);
            g[i] = fmaf(x0.x, w0.x, g[i]); g[i] = fmaf(x0.y, w0.y, g[i]); g[i] = fmaf(x0.z, w0.z, g[i]); g[i] = fmaf(x0.w, w0.w, g[i]);
            g[i] = fmaf(x1.x, w1.x, g[i]); g[i] = fmaf(x1.y, w1.y, g[i]); g[i] = fmaf(x1.z, w1.z, g[i]); g[i] = fmaf(x1.w, w1.w, g[i]);
        }
    }
    float* out = const_cast<float*>(reinterpret_cast<const float*>(a.dout)) + b * a.dos.batch + h * a.dos.head + c;
#pragma unroll
    for (int i = 0; i < NR; ++i) {
        const int r = rt + RT * i;
        const bool in = r0 + r < a.Sq && c < a.D;
        dst[r * LD + c] = in ? g[i] : 0.f;
        if (kRows && in) out[(int64_t)(r0 + r) * a.dos.seq] = g[i];
    }
}

// pass 1: delta = rowsum(dO o O), left for pass 2, and dQ.  One CTA per TM query rows, KN keys per step.
// kForm: dO is formed here (a kernel of its own, since form_dout takes registers: without it twice as many CTAs fit on an SM).
template <typename T, int DP, int TM, int KN, int NT, int kMask, bool kForm>
__global__ void __launch_bounds__(NT, NT == 128 ? 3 : 1) attn_bwd_dq_fp32_kernel(const CoreArgs a) {
    grid_dependency_wait();
    constexpr int LD = DP + kPad, LP = KN + kPad, RS = NT / 16, RM = TM / RS, CN = KN / 16, NW = KN / 32;
    using Lt = AccLayout<DP, TM, NT>;
    extern __shared__ __align__(16) float sm[];
    float* Qs = sm;
    float* Gs = Qs + TM * LD;            // dO
    float* Ks = Gs + TM * LD;
    float* Vs = Ks + KN * LD;
    float* Ss = Vs + KN * LD;            // dS
    float* row_delta = Ss + TM * LP;
    const bool vec = a.vec != 0;

    const int tx = score_tx(), row0 = row_of(score_ty());
    const int q0 = blockIdx.x * TM;
    const int h = blockIdx.y, b = blockIdx.z;
    int kvlen = a.Sk;
    if (a.kv_len) kvlen = min(max(a.kv_len[b], 0), a.Sk);

    const T* qb = reinterpret_cast<const T*>(a.q) + b * a.qs.batch + h * a.qs.head;
    const T* kb = reinterpret_cast<const T*>(a.k) + b * a.ks.batch + h * a.ks.head;
    const T* vb = reinterpret_cast<const T*>(a.v) + b * a.vs.batch + h * a.vs.head;
    const T* gb = reinterpret_cast<const T*>(a.dout) + b * a.dos.batch + h * a.dos.head;
    const T* ob = reinterpret_cast<const T*>(a.o_in) + b * a.os.batch + h * a.os.head;
    load_padded<DP, TM, NT>(Qs, qb, a.qs.seq, q0, a.Sq, a.D, vec);
    if constexpr (!kForm) load_padded<DP, TM, NT>(Gs, gb, a.dos.seq, q0, a.Sq, a.D, vec);
    load_padded<DP, KN, NT>(Ks, kb, a.ks.seq, 0, a.Sk, a.D, vec);
    load_padded<DP, KN, NT>(Vs, vb, a.vs.seq, 0, a.Sk, a.D, vec);
    cp_async_commit();
    if constexpr (kForm) form_dout<DP, TM, NT, true>(Gs, a, b, h, q0);
    cp_async_wait<0>();
    __syncthreads();

    const int64_t stat0 = ((int64_t)b * a.H + h) * a.Sq;
    // one warp per row, as the wide-head kernels form it
    for (int r = threadIdx.x >> 5; r < TM; r += NT / 32) {
        float d = 0.f;
        if (q0 + r < a.Sq) {
            const T* orow = ob + (int64_t)(q0 + r) * a.os.seq;
            for (int c = threadIdx.x & 31; c < a.D; c += 32) d = fmaf(ld_elem(orow + c), Gs[r * LD + c], d);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if ((threadIdx.x & 31) == 0) {
            row_delta[r] = d;
            if (q0 + r < a.Sq) a.delta[stat0 + q0 + r] = d;
        }
    }
    __syncthreads();

    const Lt L;
    // A row without visible keys (lse = -inf) and rows beyond the tensor take lse = +inf: their probabilities are 0.
    float lse[RM], dlt[RM];
    f32x2 acc[Lt::NR][2 * Lt::CG];
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int r = row0 + RS * i;
        const float l = q0 + r < a.Sq ? a.lse_in[stat0 + q0 + r] : kNegInf;
        lse[i] = l == kNegInf ? INFINITY : l;
        dlt[i] = row_delta[r];
    }
#pragma unroll
    for (int i = 0; i < Lt::NR; ++i)
#pragma unroll
        for (int c = 0; c < 2 * Lt::CG; ++c) acc[i][c] = 0ull;

    int k_end = kvlen;
    if (a.causal) k_end = min(k_end, min(q0 + TM - 1, a.Sq - 1) + a.causal_off + 1);
    for (int k0 = 0; k0 < k_end; k0 += KN) {
        if (k0 > 0) {
            cp_async_wait<0>();
            __syncthreads();
        }
        uint32_t words[RM][NW];
        if (kMask) {
#pragma unroll
            for (int i = 0; i < RM; ++i)
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    const int qi = q0 + row0 + RS * i, kw = k0 / 32 + w;
                    words[i][w] = mask_word<kMask>(a, b, qi, kw);
                }
        }
        float s[RM][CN], dp[RM][CN];
        tile_dot<DP, NT, RM, CN>(s, Qs, Ks, row0, tx);
        tile_dot<DP, NT, RM, CN>(dp, Gs, Vs, row0, tx);
        const bool all_visible = k0 + KN <= kvlen && !kMask && (!a.causal || k0 + KN - 1 <= q0 + a.causal_off);
#pragma unroll
        for (int i = 0; i < RM; ++i) {
            const int r = row0 + RS * i;
            uint32_t visible = ~0u;
            if (!all_visible) {
                const int last = a.causal ? min(kvlen - 1, q0 + r + a.causal_off) : kvlen - 1;
                visible = row_limit<CN>(k0 + tx, last);
                if (kMask) visible &= row_mask<CN>(words[i], tx);
            }
#pragma unroll
            for (int j = 0; j < CN; ++j) {
                float v = s[i][j] * a.scale;
                bool zero = !(visible >> j & 1u);
                if (a.use_clamp && v >= a.clamp) { v = a.clamp; zero = true; }     // the gradient of a clamped score
                const float p = expf(v - lse[i]);
                Ss[r * LP + tx + 16 * j] = zero ? 0.f : p * (dp[i][j] - dlt[i]) * a.scale;
            }
        }
        __syncthreads();
        const bool more = k0 + KN < k_end;
        if (more) load_padded<DP, KN, NT>(Vs, vb, a.vs.seq, k0 + KN, a.Sk, a.D, vec);
        cp_async_commit();
        if (L.active) accumulate<DP, TM, NT>(acc, L, Ss, LP, Ks, min(KN, (k_end - k0 + 3) & ~3));   // columns beyond k_end are 0
        __syncthreads();
        if (more) load_padded<DP, KN, NT>(Ks, kb, a.ks.seq, k0 + KN, a.Sk, a.D, vec);
        cp_async_commit();
    }
    cp_async_wait<0>();
    if (!L.active) return;
    T* dqb = reinterpret_cast<T*>(a.dq) + b * a.dqs.batch + h * a.dqs.head;
#pragma unroll
    for (int i = 0; i < Lt::NR; ++i) {
        const int r = L.ty + Lt::TY * i;
        if (q0 + r >= a.Sq) continue;
#pragma unroll
        for (int c = 0; c < Lt::CG; ++c) {
            const float2 x = halves(acc[i][2 * c]), y = halves(acc[i][2 * c + 1]);
            store4(dqb + (int64_t)(q0 + r) * a.dqs.seq, 4 * L.tx + 64 * c, a.D, make_float4(x.x, x.y, y.x, y.y), vec);
        }
    }
}

// pass 2: dK and dV.  One CTA per TK keys, QN query rows per step; a thread accumulates NR neighbouring keys.
template <typename T, int DP, int TK, int QN, int NT, int kMask>
__global__ void __launch_bounds__(NT, TK < 64 || DP <= 32 ? 3 : DP <= 64 ? 2 : 1) attn_bwd_dkv_fp32_kernel(const CoreArgs a) {
    grid_dependency_wait();
    constexpr int LD = DP + kPad, LP = TK + kPad, RS = NT / 16, RM = QN / RS, CN = TK / 16, NW = (TK + 31) / 32;
    using Lt = AccLayout<DP, TK, NT>;
    extern __shared__ __align__(16) float sm[];
    float* Ks = sm;
    float* Vs = Ks + TK * LD;
    float* Qs = Vs + TK * LD;
    float* Gs = Qs + QN * LD;
    float* Ps = Gs + QN * LD;            // P  [QN][LP]
    float* Ss = Ps + QN * LP;            // dS [QN][LP]
    float* row_lse = Ss + QN * LP;
    float* row_delta = row_lse + QN;
    const bool vec = a.vec != 0;

    const int tx = score_tx(), row0 = row_of(score_ty());
    const int k0 = blockIdx.x * TK;
    const int h = blockIdx.y, b = blockIdx.z;
    int kvlen = a.Sk;
    if (a.kv_len) kvlen = min(max(a.kv_len[b], 0), a.Sk);

    const T* qb = reinterpret_cast<const T*>(a.q) + b * a.qs.batch + h * a.qs.head;
    const T* kb = reinterpret_cast<const T*>(a.k) + b * a.ks.batch + h * a.ks.head;
    const T* vb = reinterpret_cast<const T*>(a.v) + b * a.vs.batch + h * a.vs.head;
    const T* gb = reinterpret_cast<const T*>(a.dout) + b * a.dos.batch + h * a.dos.head;
    load_padded<DP, TK, NT>(Ks, kb, a.ks.seq, k0, a.Sk, a.D, vec);
    load_padded<DP, TK, NT>(Vs, vb, a.vs.seq, k0, a.Sk, a.D, vec);

    const Lt L;
    f32x2 acck[Lt::NR][2 * Lt::CG], accv[Lt::NR][2 * Lt::CG];
#pragma unroll
    for (int i = 0; i < Lt::NR; ++i)
#pragma unroll
        for (int c = 0; c < 2 * Lt::CG; ++c) { acck[i][c] = 0ull; accv[i][c] = 0ull; }

    const int64_t stat0 = ((int64_t)b * a.H + h) * a.Sq;
    // first query row that can see key k0 (causal): qi >= k0 - causal_off
    int q_begin = 0;
    if (a.causal) q_begin = max(0, k0 - a.causal_off) / QN * QN;
    const bool tile_live = k0 < kvlen;
    for (int q0 = q_begin; q0 < a.Sq && tile_live; q0 += QN) {
        load_padded<DP, QN, NT>(Qs, qb, a.qs.seq, q0, a.Sq, a.D, vec);
        load_padded<DP, QN, NT>(Gs, gb, a.dos.seq, q0, a.Sq, a.D, vec);
        cp_async_commit();
        if (threadIdx.x < QN) {
            // rows without visible keys and rows beyond the tensor: lse = +inf, probabilities 0
            const int qi = q0 + threadIdx.x;
            const float l = qi < a.Sq ? a.lse_in[stat0 + qi] : kNegInf;
            row_lse[threadIdx.x] = l == kNegInf ? INFINITY : l;
            row_delta[threadIdx.x] = qi < a.Sq ? a.delta[stat0 + qi] : 0.f;
        }
        uint32_t words[RM][NW];
        if (kMask) {
#pragma unroll
            for (int i = 0; i < RM; ++i)
#pragma unroll
                for (int w = 0; w < NW; ++w) {
                    const int qi = q0 + row0 + RS * i, kw = k0 / 32 + w;
                    const uint32_t x = mask_word<kMask>(a, b, qi, kw);
                    words[i][w] = TK < 32 ? x >> (k0 % 32) : x;
                }
        }
        cp_async_wait<0>();
        __syncthreads();
        float s[RM][CN], dp[RM][CN];
        tile_dot<DP, NT, RM, CN>(s, Qs, Ks, row0, tx);
        tile_dot<DP, NT, RM, CN>(dp, Gs, Vs, row0, tx);
        const bool all_visible = k0 + TK <= kvlen && !kMask && (!a.causal || k0 + TK - 1 <= q0 + a.causal_off);
#pragma unroll
        for (int i = 0; i < RM; ++i) {
            const int r = row0 + RS * i;
            const float lse = row_lse[r], dlt = row_delta[r];
            uint32_t visible = ~0u;
            if (!all_visible) {
                const int last = a.causal ? min(kvlen - 1, q0 + r + a.causal_off) : kvlen - 1;
                visible = row_limit<CN>(k0 + tx, last);
                if (kMask) visible &= row_mask<CN>(words[i], tx);
            }
#pragma unroll
            for (int j = 0; j < CN; ++j) {
                float v = s[i][j] * a.scale;
                bool clamped = false;
                if (a.use_clamp && v >= a.clamp) { v = a.clamp; clamped = true; }
                float p = expf(v - lse);
                if (!(visible >> j & 1u)) p = 0.f;
                Ps[r * LP + tx + 16 * j] = p;
                Ss[r * LP + tx + 16 * j] = clamped ? 0.f : p * (dp[i][j] - dlt) * a.scale;
            }
        }
        __syncthreads();
        if (L.active) {
            const int n = min(QN, a.Sq - q0);
#pragma unroll 4
            for (int r = 0; r < n; ++r) {
                float pp[Lt::NR], dd[Lt::NR];
                ld_row<Lt::NR>(pp, Ps + r * LP + Lt::NR * L.ty);
                ld_row<Lt::NR>(dd, Ss + r * LP + Lt::NR * L.ty);
#pragma unroll
                for (int c = 0; c < Lt::CG; ++c) {
                    const ulonglong2 g = *reinterpret_cast<const ulonglong2*>(Gs + r * LD + 4 * L.tx + 64 * c);
                    const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(Qs + r * LD + 4 * L.tx + 64 * c);
#pragma unroll
                    for (int i = 0; i < Lt::NR; ++i) {
                        const f32x2 pw = pair(pp[i], pp[i]), dw = pair(dd[i], dd[i]);
                        accv[i][2 * c] = fma2(pw, g.x, accv[i][2 * c]);
                        accv[i][2 * c + 1] = fma2(pw, g.y, accv[i][2 * c + 1]);
                        acck[i][2 * c] = fma2(dw, q.x, acck[i][2 * c]);
                        acck[i][2 * c + 1] = fma2(dw, q.y, acck[i][2 * c + 1]);
                    }
                }
            }
        }
        __syncthreads();
    }
    cp_async_wait<0>();
    if (!L.active) return;
    T* dkb = reinterpret_cast<T*>(a.dk) + b * a.dks.batch + h * a.dks.head;
    T* dvb = reinterpret_cast<T*>(a.dv) + b * a.dvs.batch + h * a.dvs.head;
#pragma unroll
    for (int i = 0; i < Lt::NR; ++i) {
        const int kj = k0 + Lt::NR * L.ty + i;
        if (kj >= a.Sk) continue;
#pragma unroll
        for (int c = 0; c < Lt::CG; ++c) {
            const float2 x = halves(acck[i][2 * c]), y = halves(acck[i][2 * c + 1]);
            const float2 u = halves(accv[i][2 * c]), w = halves(accv[i][2 * c + 1]);
            store4(dkb + (int64_t)kj * a.dks.seq, 4 * L.tx + 64 * c, a.D, make_float4(x.x, x.y, y.x, y.y), vec);
            store4(dvb + (int64_t)kj * a.dvs.seq, 4 * L.tx + 64 * c, a.D, make_float4(u.x, u.y, w.x, w.y), vec);
        }
    }
}

// ----------------------------------------------------------------------------------------------
// one pass: dK, dV and dQ from one evaluation of the scores and of dP.  One CTA per 64 keys, 64 query rows per step.
//
// Five products a tile instead of the seven of the two kernels above.  dQ of a step is this CTA's 64 keys' share of it, written
// out and added up by attn_bwd_dq_sum_kernel in the order of the keys; a call of 64 keys or fewer writes it where it belongs.
// P and then dS go through the same shared memory: what a tile holds beside it (K, V, Q, dO) leaves room for four CTAs an SM
// at head widths up to 32.  A thread reads its own probabilities back for dS, so they take no registers under dP's product.
// Against the two kernels, us: B16 H8 S250 D32 130 -> 89, causal 109 -> 66, with a dense mask 156 -> 96; B32 H8 S256 D16 143 -> 94;
// B8 H8 S512 D64 459 -> 323, causal 349 -> 175; one block of keys, B64 H8 S60 D32 43 -> 24.  256 threads at D = 64: 293 us for B32
// H8 S256, with 128 (a larger block of scores each, half the warps) 318.  What bounds it: issue slots (about 6300 cycles a tile and
// SM at D = 32) and shared-memory wavefronts (5000), at 16 warps an SM.
// ----------------------------------------------------------------------------------------------
template <typename T, int DP, int N, int NT, int kMask, bool kForm>
__global__ void __launch_bounds__(NT, kForm ? 256 / NT : DP <= 32 ? 4 : 2) attn_bwd_fp32_kernel(const CoreArgs a) {
    grid_dependency_wait();
    constexpr int LD = DP + kPad, LP = N + kPad, RS = NT / 16, RM = N / RS, CN = N / 16, NW = N / 32;
    constexpr int kPer = NT / N, kOq = DP / (4 * kPer);       // delta: threads of a row, 16-byte pieces of each
    using Lt = AccLayout<DP, N, NT>;
    extern __shared__ __align__(16) float sm[];
    float* Ks = sm;
    float* Vs = Ks + N * LD;
    float* Qs = Vs + N * LD;
    float* Gs = Qs + N * LD;             // dO
    float* Ps = Gs + N * LD;             // P, then dS
    float* row_lse = Ps + N * LP;
    float* row_delta = row_lse + N;
    uint32_t* mask_sm = reinterpret_cast<uint32_t*>(row_delta + N);      // [N][NW]
    const bool vec = a.vec != 0;

    const int tx = score_tx(), row0 = row_of(score_ty());
    const int bh = a.pair0 + blockIdx.x, b = bh / a.H, h = bh % a.H;
    const int k0 = blockIdx.y * N;
    int kvlen = a.Sk;
    if (a.kv_len) kvlen = min(max(a.kv_len[b], 0), a.Sk);

    const T* qb = reinterpret_cast<const T*>(a.q) + b * a.qs.batch + h * a.qs.head;
    const T* kb = reinterpret_cast<const T*>(a.k) + b * a.ks.batch + h * a.ks.head;
    const T* vb = reinterpret_cast<const T*>(a.v) + b * a.vs.batch + h * a.vs.head;
    const T* gb = reinterpret_cast<const T*>(a.dout) + b * a.dos.batch + h * a.dos.head;
    const T* ob = reinterpret_cast<const T*>(a.o_in) + b * a.os.batch + h * a.os.head;
    load_padded<DP, N, NT>(Ks, kb, a.ks.seq, k0, a.Sk, a.D, vec);
    load_padded<DP, N, NT>(Vs, vb, a.vs.seq, k0, a.Sk, a.D, vec);

    const Lt L;
    f32x2 acck[Lt::NR][2 * Lt::CG], accv[Lt::NR][2 * Lt::CG];
#pragma unroll
    for (int i = 0; i < Lt::NR; ++i)
#pragma unroll
        for (int c = 0; c < 2 * Lt::CG; ++c) { acck[i][c] = 0ull; accv[i][c] = 0ull; }

    const int64_t stat0 = (int64_t)bh * a.Sq;
    // first query row that can see key k0 (causal): qi >= k0 - causal_off
    const int q_begin = a.causal ? max(0, k0 - a.causal_off) / N * N : 0;
    const int q_end = k0 < kvlen ? a.Sq : 0;
    for (int q0 = q_begin; q0 < q_end; q0 += N) {
        load_padded<DP, N, NT>(Qs, qb, a.qs.seq, q0, a.Sq, a.D, vec);
        if constexpr (!kForm) load_padded<DP, N, NT>(Gs, gb, a.dos.seq, q0, a.Sq, a.D, vec);
        cp_async_commit();
        const int dr = threadIdx.x / kPer, dc = 4 * (threadIdx.x % kPer);
        float4 orow[kOq];
#pragma unroll
        for (int i = 0; i < kOq; ++i) {
            const int c = dc + 4 * kPer * i;
            orow[i] = q0 + dr < a.Sq ? row4(ob + (int64_t)(q0 + dr) * a.os.seq, c, a.D, vec) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (threadIdx.x < N) {
            // rows without visible keys and rows beyond the tensor: lse = +inf, probabilities 0
            const int qi = q0 + threadIdx.x;
            const float l = qi < a.Sq ? a.lse_in[stat0 + qi] : kNegInf;
            row_lse[threadIdx.x] = l == kNegInf ? INFINITY : l;
        }
        // dense mask: as words where there are any, else every warp votes the words (32 keys of a row each) of its share of the
        // rows.  The words cost a launch, the votes 2 to 7 % of a step: up to two steps a CTA go without (backward, us, words and
        // votes: B8 H8 S32 D32 8.9 and 5.7, B16 H4 S100 D32 26.5 and 25.3, B16 H8 S250 D32 95.2 and 94.4, B12 H8 S400 D32 203 and 217).
        constexpr int kRows = N / (NT / 32);
        float mv[kRows * NW];
        const int lane = threadIdx.x & 31, mask_row = (threadIdx.x >> 5) * kRows;
        if constexpr (kMask == kDense) {
            const float* p = a.keep_mask + ((int64_t)b * a.Sq + q0 + mask_row) * a.Sk + k0 + lane;
#pragma unroll
            for (int r = 0; r < kRows; ++r, p += a.Sk)
#pragma unroll
                for (int w = 0; w < NW; ++w)
                    mv[r * NW + w] = q0 + mask_row + r < a.Sq && k0 + 32 * w + lane < a.Sk ? __ldg(p + 32 * w) : 0.f;
        } else if constexpr (kMask == kWords) {
            if (threadIdx.x < NW * N) mask_sm[threadIdx.x] = mask_word<kWords>(a, b, q0 + threadIdx.x / NW, k0 / 32 + threadIdx.x % NW);
        }
        if constexpr (kForm) form_dout<DP, N, NT, false>(Gs, a, b, h, q0);
        cp_async_wait<0>();
        if constexpr (kMask == kDense) {
#pragma unroll
            for (int w = 0; w < kRows * NW; ++w) {
                const uint32_t bits = __ballot_sync(0xffffffffu, mv[w] != 0.f);
                if (lane == 0) mask_sm[mask_row * NW + w] = bits;
            }
        }
        __syncthreads();
        {   // delta = rowsum(dO o O)
            float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < kOq; ++i) {
                const float4 g = *reinterpret_cast<const float4*>(Gs + dr * LD + dc + 4 * kPer * i);
                e.x = fmaf(orow[i].x, g.x, e.x); e.y = fmaf(orow[i].y, g.y, e.y);
                e.z = fmaf(orow[i].z, g.z, e.z); e.w = fmaf(orow[i].w, g.w, e.w);
            }
            float d = (e.x + e.y) + (e.z + e.w);
#pragma unroll
            for (int o = kPer / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
            if (threadIdx.x % kPer == 0) row_delta[dr] = d;
        }
        const bool all_visible = k0 + N <= kvlen && !kMask && (!a.causal || k0 + N - 1 <= q0 + a.causal_off);
        uint32_t dead = 0;               // scores whose gradient is 0: hidden or clamped ones, bit CN i + j
        {
            float s[RM][CN];
            tile_dot<DP, NT, RM, CN>(s, Qs, Ks, row0, tx);
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                const int r = row0 + RS * i;
                const float lse = row_lse[r];
                uint32_t visible = ~0u;
                if (!all_visible) {
                    const int last = a.causal ? min(kvlen - 1, q0 + r + a.causal_off) : kvlen - 1;
                    visible = row_limit<CN>(k0 + tx, last);
                    if (kMask) visible &= row_mask<CN>(mask_sm + NW * r, tx);
                }
#pragma unroll
                for (int j = 0; j < CN; ++j) {
                    float v = s[i][j] * a.scale;
                    bool hidden = !(visible >> j & 1u), zero = hidden;
                    if (a.use_clamp && v >= a.clamp) { v = a.clamp; zero = true; }     // the gradient of a clamped score
                    const float p = expf(v - lse);
                    Ps[r * LP + tx + 16 * j] = hidden ? 0.f : p;
                    dead |= (zero ? 1u : 0u) << (CN * i + j);
                }
            }
        }
        __syncthreads();
        const int n = min(N, a.Sq - q0);
        if (L.active) {
#pragma unroll 4
            for (int r = 0; r < n; ++r) {
                float pp[Lt::NR];
                ld_row<Lt::NR>(pp, Ps + r * LP + Lt::NR * L.ty);
#pragma unroll
                for (int c = 0; c < Lt::CG; ++c) {
                    const ulonglong2 g = *reinterpret_cast<const ulonglong2*>(Gs + r * LD + 4 * L.tx + 64 * c);
#pragma unroll
                    for (int i = 0; i < Lt::NR; ++i) {
                        const f32x2 pw = pair(pp[i], pp[i]);
                        accv[i][2 * c] = fma2(pw, g.x, accv[i][2 * c]);
                        accv[i][2 * c + 1] = fma2(pw, g.y, accv[i][2 * c + 1]);
                    }
                }
            }
        }
        {
            float dp[RM][CN];
            tile_dot<DP, NT, RM, CN>(dp, Gs, Vs, row0, tx);
            __syncthreads();
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                const int r = row0 + RS * i;
                const float dlt = row_delta[r];
#pragma unroll
                for (int j = 0; j < CN; ++j) {
                    float* x = Ps + r * LP + tx + 16 * j;
                    *x = dead >> (CN * i + j) & 1u ? 0.f : *x * (dp[i][j] - dlt) * a.scale;
                }
            }
        }
        __syncthreads();
        if (L.active) {
#pragma unroll 4
            for (int r = 0; r < n; ++r) {
                float dd[Lt::NR];
                ld_row<Lt::NR>(dd, Ps + r * LP + Lt::NR * L.ty);
#pragma unroll
                for (int c = 0; c < Lt::CG; ++c) {
                    const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(Qs + r * LD + 4 * L.tx + 64 * c);
#pragma unroll
                    for (int i = 0; i < Lt::NR; ++i) {
                        const f32x2 dw = pair(dd[i], dd[i]);
                        acck[i][2 * c] = fma2(dw, q.x, acck[i][2 * c]);
                        acck[i][2 * c + 1] = fma2(dw, q.y, acck[i][2 * c + 1]);
                    }
                }
            }
            f32x2 acc[Lt::NR][2 * Lt::CG];
#pragma unroll
            for (int i = 0; i < Lt::NR; ++i)
#pragma unroll
                for (int c = 0; c < 2 * Lt::CG; ++c) acc[i][c] = 0ull;
            int k_end = kvlen;                                // no row of the tile sees a key beyond it
            if (a.causal) k_end = min(k_end, min(q0 + N - 1, a.Sq - 1) + a.causal_off + 1);
            accumulate<DP, N, NT>(acc, L, Ps, LP, Ks, min(N, (k_end - k0 + 3) & ~3));
#pragma unroll
            for (int i = 0; i < Lt::NR; ++i) {
                const int qi = q0 + L.ty + Lt::TY * i;
                if (qi >= a.Sq) continue;
#pragma unroll
                for (int c = 0; c < Lt::CG; ++c) {
                    const int col = 4 * L.tx + 64 * c;
                    const float2 x = halves(acc[i][2 * c]), y = halves(acc[i][2 * c + 1]);
                    const float4 v = make_float4(x.x, x.y, y.x, y.y);
                    if (a.dq_part) {
                        if (col < a.part_ld)
                            *reinterpret_cast<float4*>(a.dq_part + (((int64_t)blockIdx.y * a.pairs + blockIdx.x) * a.Sq + qi) * a.part_ld + col) = v;
                    } else {
                        T* dqb = reinterpret_cast<T*>(a.dq) + b * a.dqs.batch + h * a.dqs.head;
                        store4(dqb + (int64_t)qi * a.dqs.seq, col, a.D, v, vec);
                    }
                }
            }
        }
        __syncthreads();
    }
    cp_async_wait<0>();
    if (!a.dq_part) {                    // rows that see none of the keys
        T* dqb = reinterpret_cast<T*>(a.dq) + b * a.dqs.batch + h * a.dqs.head;
        const int rows = q_end > 0 ? min(q_begin, a.Sq) : a.Sq;
        for (int e = threadIdx.x; e < rows * (DP / 4); e += NT)
            store4(dqb + (int64_t)(e / (DP / 4)) * a.dqs.seq, 4 * (e % (DP / 4)), a.D, make_float4(0.f, 0.f, 0.f, 0.f), vec);
    }
    if (!L.active) return;
    T* dkb = reinterpret_cast<T*>(a.dk) + b * a.dks.batch + h * a.dks.head;
    T* dvb = reinterpret_cast<T*>(a.dv) + b * a.dvs.batch + h * a.dvs.head;
#pragma unroll
    for (int i = 0; i < Lt::NR; ++i) {
        const int kj = k0 + Lt::NR * L.ty + i;
        if (kj >= a.Sk) continue;
#pragma unroll
        for (int c = 0; c < Lt::CG; ++c) {
            const float2 x = halves(acck[i][2 * c]), y = halves(acck[i][2 * c + 1]);
            const float2 u = halves(accv[i][2 * c]), w = halves(accv[i][2 * c + 1]);
            store4(dkb + (int64_t)kj * a.dks.seq, 4 * L.tx + 64 * c, a.D, make_float4(x.x, x.y, y.x, y.y), vec);
            store4(dvb + (int64_t)kj * a.dvs.seq, 4 * L.tx + 64 * c, a.D, make_float4(u.x, u.y, w.x, w.y), vec);
        }
    }
}

// dQ = the sum of the key blocks' shares, in the order of the keys; a block that no row of a 64-row tile sees left none.
template <typename T>
__global__ void __launch_bounds__(256) attn_bwd_dq_sum_kernel(const CoreArgs a) {
    grid_dependency_wait();
    const int quads = a.part_ld / 4;
    const int64_t total = (int64_t)a.pairs * a.Sq * quads, step = total * 4;
    for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < total; e += (int64_t)gridDim.x * 256) {
        const int64_t row = e / quads;
        const int c = 4 * (int)(e - row * quads), qi = (int)(row % a.Sq), bh = a.pair0 + (int)(row / a.Sq);
        const int b = bh / a.H, h = bh % a.H;
        int keys = a.Sk;
        if (a.kv_len) keys = min(max(a.kv_len[b], 0), a.Sk);
        if (a.causal) keys = min(keys, qi / 64 * 64 + 64 + a.causal_off);
        const float* src = a.dq_part + 4 * e;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int k = 0; k < keys; k += 64, src += step) {
            const float4 x = *reinterpret_cast<const float4*>(src);
            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
        }
        store4(reinterpret_cast<T*>(a.dq) + b * a.dqs.batch + h * a.dqs.head + (int64_t)qi * a.dqs.seq, c, a.D, v, a.vec != 0);
    }
}

CoreArgs make_args(const ltca_attn_params* p) {
    CoreArgs a;
    memset(&a, 0, sizeof(a));
    a.B = p->B; a.H = p->H; a.Sq = p->Sq; a.Sk = p->Sk; a.D = p->D;
    a.causal = p->causal ? 1 : 0;
    a.causal_off = p->Sk - p->Sq;
    a.scale = p->scale;
    a.use_clamp = p->score_clamp > 0.f ? 1 : 0;
    a.clamp = p->score_clamp;
    a.q = p->q; a.k = p->k; a.v = p->v; a.o = p->o; a.o_in = p->o; a.dout = p->dout;
    a.dq = p->dq; a.dk = p->dk; a.dv = p->dv;
    a.qs = p->q_strides; a.ks = p->k_strides; a.vs = p->v_strides; a.os = p->o_strides;
    a.dos = p->do_strides; a.dqs = p->dq_strides; a.dks = p->dk_strides; a.dvs = p->dv_strides;
    a.lse = p->lse; a.lse_in = p->lse;
    a.keep_mask = p->keep_mask;
    a.kv_len = p->kv_len;
    const int es = elem_size(p->dtype);
    bool vec = p->D % 4 == 0;
    auto rows = [&](const void* ptr, const ltca_strides& st) {
        if (!ptr) return;
        if ((reinterpret_cast<uintptr_t>(ptr) % (4 * es)) || (st.seq % 4) || (st.head % 4) || (st.batch % 4)) vec = false;
    };
    rows(a.q, a.qs); rows(a.k, a.ks); rows(a.v, a.vs); rows(a.o, a.os);
    rows(a.dout, a.dos); rows(a.dq, a.dqs); rows(a.dk, a.dks); rows(a.dv, a.dvs);
    a.vec = vec ? 1 : 0;
    return a;
}

template <typename K>
int set_smem(ltca_ctx* ctx, K kern, size_t bytes, SmemOptIn& once) {
    if (bytes > 48 * 1024) LTCA_CUDA_OK(ctx, opt_in_dynamic_smem(once, ctx->device, kern, (int)bytes));
    return LTCA_OK;
}

template <typename T, int DP, int TM, int NT, bool kMask>
int run_fwd(ltca_ctx* ctx, const CoreArgs& a) {
    static SmemOptIn once;
    constexpr size_t smem = ((size_t)(TM + 128) * (DP + kPad) + TM * (64 + kPad) + TM + (kMask ? (TM == 64 && DP <= 32 ? 4 : 2) * TM : 0)) * sizeof(float);
    int rc = set_smem(ctx, attn_fwd_fp32_kernel<T, DP, TM, NT, kMask>, smem, once);
    if (rc) return rc;
    dim3 grid((a.Sq + TM - 1) / TM, a.H, a.B);
    LTCA_CUDA_OK(ctx, launch_dependent(attn_fwd_fp32_kernel<T, DP, TM, NT, kMask>, grid, dim3(NT), smem, ctx->stream, a));
    return LTCA_OK;
}

template <typename T, int DP, int TM, int KN, int NT, int kMask, bool kForm = false>
int run_dq(ltca_ctx* ctx, const CoreArgs& a) {
    static SmemOptIn once;
    constexpr size_t smem = ((size_t)(2 * TM + 2 * KN) * (DP + kPad) + TM * (KN + kPad) + TM) * sizeof(float);
    int rc = set_smem(ctx, attn_bwd_dq_fp32_kernel<T, DP, TM, KN, NT, kMask, kForm>, smem, once);
    if (rc) return rc;
    dim3 grid((a.Sq + TM - 1) / TM, a.H, a.B);
    LTCA_CUDA_OK(ctx, launch_dependent(attn_bwd_dq_fp32_kernel<T, DP, TM, KN, NT, kMask, kForm>, grid, dim3(NT), smem, ctx->stream, a));
    return LTCA_OK;
}
template <typename T, int DP, int TK, int QN, int NT, int kMask>
int run_dkv(ltca_ctx* ctx, const CoreArgs& a) {
    static SmemOptIn once;
    constexpr size_t smem = ((size_t)(2 * TK + 2 * QN) * (DP + kPad) + 2 * QN * (TK + kPad) + 2 * QN) * sizeof(float);
    int rc = set_smem(ctx, attn_bwd_dkv_fp32_kernel<T, DP, TK, QN, NT, kMask>, smem, once);
    if (rc) return rc;
    dim3 grid((a.Sk + TK - 1) / TK, a.H, a.B);
    LTCA_CUDA_OK(ctx, launch_dependent(attn_bwd_dkv_fp32_kernel<T, DP, TK, QN, NT, kMask>, grid, dim3(NT), smem, ctx->stream, a));
    return LTCA_OK;
}

// (None of these kernels lets the next one's CTAs be placed before it ends: released at the start, or when the tile loop is
// done, they take whatever slots are left and sit unevenly on the SMs, 82 or 62 us instead of 57 for B16 H8 S100 D32.)
// Tiles of 64 rows reuse what they load most; where they would leave SMs idle, tiles of 16 rows give four times the CTAs
// and a quarter of the serial work.  The two-kernel backward is left for heads above 64 and where one_pass says so: few CTAs of 64
// keys (16-row tiles, of dQ 64-row ones where many queries meet few keys) and calls without room for dQ's shares (64-row tiles).
template <typename T, int DP, int kMask>
int run_small_dq(ltca_ctx* ctx, const CoreArgs& a) {
    if constexpr (sizeof(T) == 4 && DP <= 64) {
        if (a.dy) return run_dq<T, DP, 16, 32, 128, kMask, true>(ctx, a);
    }
    return run_dq<T, DP, 16, 32, 128, kMask>(ctx, a);
}
bool fills_sms(const ltca_ctx* ctx, int B, int H, int S) { return (int64_t)B * H * ((S + 63) / 64) >= ctx->sm_device; }
// The one-pass backward, in as many launches as the room for dQ's shares allows.
template <typename T, int DP, int N, int NT, int kMask, bool kForm = false>
int launch_one_pass(ltca_ctx* ctx, CoreArgs a) {
    static SmemOptIn once;
    constexpr size_t smem = ((size_t)4 * N * (DP + kPad) + N * (N + kPad) + 2 * N + (kMask ? N * N / 32 : 0)) * sizeof(float);
    int rc = set_smem(ctx, attn_bwd_fp32_kernel<T, DP, N, NT, kMask, kForm>, smem, once);
    if (rc) return rc;
    const int all = a.B * a.H, most = a.pairs;
    for (a.pair0 = 0; a.pair0 < all; a.pair0 += most) {
        a.pairs = all - a.pair0 < most ? all - a.pair0 : most;
        const dim3 grid(a.pairs, (a.Sk + N - 1) / N);
        LTCA_CUDA_OK(ctx, launch_dependent(attn_bwd_fp32_kernel<T, DP, N, NT, kMask, kForm>, grid, dim3(NT), smem, ctx->stream, a));
        if (!a.dq_part) continue;
        const int64_t blocks = ((int64_t)a.pairs * a.Sq * (a.part_ld / 4) + 255) / 256, limit = 16ll * ctx->sm_device;
        const dim3 rg((unsigned)(blocks < limit ? blocks : limit));
        LTCA_CUDA_OK(ctx, launch_dependent(attn_bwd_dq_sum_kernel<T>, rg, dim3(256), 0, ctx->stream, a));
    }
    return LTCA_OK;
}
// Key blocks of 64, or of 32 where that holds all keys: a quarter of a tile's scores (B16 H8 S16: D16 6.7 -> 3.8 us, D32 9.1 -> 4.6).
template <typename T, int DP, bool kMask>
int run_one_pass(ltca_ctx* ctx, const CoreArgs& a) {
    constexpr int NT = DP <= 32 ? 128 : kOnePassThreads64, kM = kMask ? kDense : kNoMask;
    if constexpr (sizeof(T) == 4) {
        if (a.dy) return launch_one_pass<T, DP, 32, 128, kM, true>(ctx, a);
    }
    if (a.Sk <= 32) return launch_one_pass<T, DP, 32, 128, kM>(ctx, a);
    if (kMask && a.mask_bits) return launch_one_pass<T, DP, 64, NT, kWords>(ctx, a);
    return launch_one_pass<T, DP, 64, NT, kM>(ctx, a);
}
template <typename T, int DP, bool kMask>
int run_rows(ltca_ctx* ctx, const CoreArgs& a, bool bwd) {
    auto fills = [&](int S) { return fills_sms(ctx, a.B, a.H, S); };
    constexpr int NT = DP > 64 ? 256 : 128;         // at DP = 128 eight columns per thread need the wider CTA
    if constexpr (DP <= 64) {
        if (bwd && a.pairs) return run_one_pass<T, DP, kMask>(ctx, a);
    }
    if (!bwd) return fills(a.Sq) ? run_fwd<T, DP, 64, NT, kMask>(ctx, a) : run_fwd<T, DP, 16, 128, kMask>(ctx, a);
    int rc;
    if constexpr (kMask) {
        // without room for the mask's words: the small tiles alone, whose results have the same bits
        if (!a.mask_bits) return (rc = run_small_dq<T, DP, kDense>(ctx, a)) ? rc : run_dkv<T, DP, 16, 32, 128, kDense>(ctx, a);
    }
    constexpr int kM = kMask ? kWords : kNoMask;
    if ((rc = fills(a.Sq) ? run_dq<T, DP, 64, 64, NT, kM>(ctx, a) : run_small_dq<T, DP, kM>(ctx, a))) return rc;
    return fills(a.Sk) ? run_dkv<T, DP, 64, 64, NT, kM>(ctx, a) : run_dkv<T, DP, 16, 32, 128, kM>(ctx, a);
}
template <typename T, int DP>
int run_rows(ltca_ctx* ctx, const CoreArgs& a, bool bwd) {
    if (!a.keep_mask) return run_rows<T, DP, false>(ctx, a, bwd);
    return run_rows<T, DP, true>(ctx, a, bwd);
}

// ----------------------------------------------------------------------------------------------
// Wide heads (128 < head_dim <= 512): the reference-compatible TimeSelfAttention gives every head
// the full model width (include/cuDNN_ops.h:166-169 of the reference), so a 512-wide model has
// 512-wide heads.  A tile of such rows no longer fits in shared memory next to its keys, so these
// kernels give one warp to one query row (or one key row in the dK/dV pass): the lanes split the
// feature dimension, a score is a warp reduction, and the row's accumulator lives in registers.
// Same arithmetic and the same masks as the tiled kernels above; no atomics.
// ----------------------------------------------------------------------------------------------
constexpr int kWideMaxD = 512;
constexpr int kWC = kWideMaxD / 32;        // feature columns per lane
constexpr int kWideWarps = 4;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <typename T>
__device__ __forceinline__ void load_row(float (&r)[kWC], const T* p, int D, int lane, float mul) {
#pragma unroll
    for (int c = 0; c < kWC; ++c) {
        const int d = lane + 32 * c;
        r[c] = d < D ? ld_elem(p + d) * mul : 0.f;
    }
}
__device__ __forceinline__ float dot_row(const float (&x)[kWC], const float (&y)[kWC]) {
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < kWC; ++c) s = fmaf(x[c], y[c], s);
    return warp_sum(s);
}

template <typename T>
__global__ void __launch_bounds__(kWideWarps * 32) attn_fwd_wide_kernel(const CoreArgs a) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * kWideWarps + (threadIdx.x >> 5);
    if (row >= (int64_t)a.B * a.H * a.Sq) return;
    const int qi = (int)(row % a.Sq);
    const int64_t bh = row / a.Sq;
    const int h = (int)(bh % a.H), b = (int)(bh / a.H);
    int kvlen = a.Sk;
    if (a.kv_len) kvlen = min(max(a.kv_len[b], 0), a.Sk);
    const T* kb = reinterpret_cast<const T*>(a.k) + b * a.ks.batch + h * a.ks.head;
    const T* vb = reinterpret_cast<const T*>(a.v) + b * a.vs.batch + h * a.vs.head;
    float q[kWC], acc[kWC];
    load_row(q, reinterpret_cast<const T*>(a.q) + b * a.qs.batch + h * a.qs.head + (int64_t)qi * a.qs.seq, a.D,
             lane, a.scale);
#pragma unroll
    for (int c = 0; c < kWC; ++c) acc[c] = 0.f;
    float m = -INFINITY, l = 0.f;
    int k_end = kvlen;
    if (a.causal) k_end = min(k_end, qi + a.causal_off + 1);
    for (int j = 0; j < k_end; ++j) {
        if (!key_visible(a, b, qi, j, kvlen)) continue;          // the same answer in every lane
        float kr[kWC];
        load_row(kr, kb + (int64_t)j * a.ks.seq, a.D, lane, 1.f);
        float v = dot_row(q, kr);
        if (a.use_clamp) v = fminf(v, a.clamp);
        const float m_new = fmaxf(m, v);
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
        const float p = expf(v - m_new);
        l = l * corr + p;
        m = m_new;
        load_row(kr, vb + (int64_t)j * a.vs.seq, a.D, lane, 1.f);
#pragma unroll
        for (int c = 0; c < kWC; ++c) acc[c] = fmaf(p, kr[c], acc[c] * corr);
    }
    T* op = reinterpret_cast<T*>(a.o) + b * a.os.batch + h * a.os.head + (int64_t)qi * a.os.seq;
    const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
    for (int c = 0; c < kWC; ++c) {
        const int d = lane + 32 * c;
        if (d < a.D) st_elem(op + d, acc[c] * inv);
    }
    if (a.lse && lane == 0) a.lse[row] = l > 0.f ? m + logf(l) : -INFINITY;
}

// dQ: one warp per query row.
template <typename T>
__global__ void __launch_bounds__(kWideWarps * 32) attn_bwd_dq_wide_kernel(const CoreArgs a) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * kWideWarps + (threadIdx.x >> 5);
    if (row >= (int64_t)a.B * a.H * a.Sq) return;
    const int qi = (int)(row % a.Sq);
    const int64_t bh = row / a.Sq;
    const int h = (int)(bh % a.H), b = (int)(bh / a.H);
    int kvlen = a.Sk;
    if (a.kv_len) kvlen = min(max(a.kv_len[b], 0), a.Sk);
    const T* kb = reinterpret_cast<const T*>(a.k) + b * a.ks.batch + h * a.ks.head;
    const T* vb = reinterpret_cast<const T*>(a.v) + b * a.vs.batch + h * a.vs.head;
    float q[kWC], g[kWC], acc[kWC];
    load_row(q, reinterpret_cast<const T*>(a.q) + b * a.qs.batch + h * a.qs.head + (int64_t)qi * a.qs.seq, a.D,
             lane, a.scale);
    load_row(g, reinterpret_cast<const T*>(a.dout) + b * a.dos.batch + h * a.dos.head + (int64_t)qi * a.dos.seq,
             a.D, lane, 1.f);
#pragma unroll
    for (int c = 0; c < kWC; ++c) acc[c] = 0.f;
    const float lse = a.lse_in[row], dlt = a.delta[row];
    int k_end = kvlen;
    if (a.causal) k_end = min(k_end, qi + a.causal_off + 1);
    if (lse == -INFINITY) k_end = 0;
    for (int j = 0; j < k_end; ++j) {
        if (!key_visible(a, b, qi, j, kvlen)) continue;
        float kr[kWC], vr[kWC];
        load_row(kr, kb + (int64_t)j * a.ks.seq, a.D, lane, 1.f);
        load_row(vr, vb + (int64_t)j * a.vs.seq, a.D, lane, 1.f);
        float v = dot_row(q, kr);
        const float dp = dot_row(g, vr);
        bool clamped = false;
        if (a.use_clamp && v >= a.clamp) { v = a.clamp; clamped = true; }
        const float ds = clamped ? 0.f : expf(v - lse) * (dp - dlt) * a.scale;
#pragma unroll
        for (int c = 0; c < kWC; ++c) acc[c] = fmaf(ds, kr[c], acc[c]);
    }
    T* dqp = reinterpret_cast<T*>(a.dq) + b * a.dqs.batch + h * a.dqs.head + (int64_t)qi * a.dqs.seq;
#pragma unroll
    for (int c = 0; c < kWC; ++c) {
        const int d = lane + 32 * c;
        if (d < a.D) st_elem(dqp + d, acc[c]);
    }
}

// dK and dV: one warp per key row, looping over the queries that see the key.
template <typename T>
__global__ void __launch_bounds__(kWideWarps * 32) attn_bwd_dkv_wide_kernel(const CoreArgs a) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * kWideWarps + (threadIdx.x >> 5);
    if (row >= (int64_t)a.B * a.H * a.Sk) return;
    const int kj = (int)(row % a.Sk);
    const int64_t bh = row / a.Sk;
    const int h = (int)(bh % a.H), b = (int)(bh / a.H);
    int kvlen = a.Sk;
    if (a.kv_len) kvlen = min(max(a.kv_len[b], 0), a.Sk);
    const T* qb = reinterpret_cast<const T*>(a.q) + b * a.qs.batch + h * a.qs.head;
    const T* gb = reinterpret_cast<const T*>(a.dout) + b * a.dos.batch + h * a.dos.head;
    float kr[kWC], vr[kWC], dk[kWC], dv[kWC];
    load_row(kr, reinterpret_cast<const T*>(a.k) + b * a.ks.batch + h * a.ks.head + (int64_t)kj * a.ks.seq, a.D,
             lane, a.scale);
    load_row(vr, reinterpret_cast<const T*>(a.v) + b * a.vs.batch + h * a.vs.head + (int64_t)kj * a.vs.seq, a.D,
             lane, 1.f);
#pragma unroll
    for (int c = 0; c < kWC; ++c) { dk[c] = 0.f; dv[c] = 0.f; }
    int q_begin = 0;
    if (a.causal) q_begin = max(0, kj - a.causal_off);
    const int q_end = kj < kvlen ? a.Sq : 0;
    const int64_t stat0 = bh * a.Sq;
    for (int qi = q_begin; qi < q_end; ++qi) {
        if (!key_visible(a, b, qi, kj, kvlen)) continue;
        const float lse = a.lse_in[stat0 + qi];
        if (lse == -INFINITY) continue;
        float qr[kWC], gr[kWC];
        load_row(qr, qb + (int64_t)qi * a.qs.seq, a.D, lane, 1.f);
        load_row(gr, gb + (int64_t)qi * a.dos.seq, a.D, lane, 1.f);
        float v = dot_row(qr, kr);                     // kr carries the scale
        const float dp = dot_row(gr, vr);
        bool clamped = false;
        if (a.use_clamp && v >= a.clamp) { v = a.clamp; clamped = true; }
        const float p = expf(v - lse);
        const float ds = clamped ? 0.f : p * (dp - a.delta[stat0 + qi]) * a.scale;
#pragma unroll
        for (int c = 0; c < kWC; ++c) {
            dv[c] = fmaf(p, gr[c], dv[c]);
            dk[c] = fmaf(ds, qr[c], dk[c]);
        }
    }
    T* dkp = reinterpret_cast<T*>(a.dk) + b * a.dks.batch + h * a.dks.head + (int64_t)kj * a.dks.seq;
    T* dvp = reinterpret_cast<T*>(a.dv) + b * a.dvs.batch + h * a.dvs.head + (int64_t)kj * a.dvs.seq;
#pragma unroll
    for (int c = 0; c < kWC; ++c) {
        const int d = lane + 32 * c;
        if (d < a.D) { st_elem(dkp + d, dk[c]); st_elem(dvp + d, dv[c]); }
    }
}

template <typename T>
int run_wide(ltca_ctx* ctx, const CoreArgs& a, bool bwd) {
    const int64_t qrows = (int64_t)a.B * a.H * a.Sq, krows = (int64_t)a.B * a.H * a.Sk;
    const unsigned qblocks = (unsigned)((qrows + kWideWarps - 1) / kWideWarps);
    if (!bwd) {
        attn_fwd_wide_kernel<T><<<qblocks, kWideWarps * 32, 0, ctx->stream>>>(a);
        LTCA_LAUNCH_OK(ctx, "attn_fwd_wide_kernel");
        return LTCA_OK;
    }
    attn_bwd_delta_kernel<T><<<(unsigned)((qrows + 7) / 8), 256, 0, ctx->stream>>>(a);
    LTCA_LAUNCH_OK(ctx, "attn_bwd_delta_kernel");
    attn_bwd_dq_wide_kernel<T><<<qblocks, kWideWarps * 32, 0, ctx->stream>>>(a);
    LTCA_LAUNCH_OK(ctx, "attn_bwd_dq_wide_kernel");
    attn_bwd_dkv_wide_kernel<T><<<(unsigned)((krows + kWideWarps - 1) / kWideWarps), kWideWarps * 32, 0,
                                  ctx->stream>>>(a);
    LTCA_LAUNCH_OK(ctx, "attn_bwd_dkv_wide_kernel");
    return LTCA_OK;
}

template <typename T>
int dispatch(ltca_ctx* ctx, const CoreArgs& a, bool bwd) {
    if (a.D > 128) return run_wide<T>(ctx, a, bwd);
    if (a.D <= 16) return run_rows<T, 16>(ctx, a, bwd);
    if (a.D <= 32) return run_rows<T, 32>(ctx, a, bwd);
    if (a.D <= 64) return run_rows<T, 64>(ctx, a, bwd);
    return run_rows<T, 128>(ctx, a, bwd);
}

}  // namespace

// delta, and the dense mask as bits (the kernels for head_dim up to 128)
static size_t delta_bytes(const ltca_attn_params* p) { return align_up((size_t)p->B * p->H * p->Sq * sizeof(float), 256); }
// The one-pass backward: how many (batch, head) pairs a launch takes, and the room for their shares of dQ, one per 64 keys (none where
// there is one block of keys).  kPartBytes and the room there is bound it: beyond them several launches.
constexpr size_t kPartBytes = 512u << 20;
struct OnePass {
    int pairs = 0, ld = 0;        // 0: the two kernels
    size_t bytes = 0;
};
// Where one pass over the scores is the faster one.  A CTA walks all queries of its 64 keys, which the two kernels deal out; with few
// CTAs that chain is the longer one.  (Of a CTA per SM; the time in units of the two kernels', or us of either.)
//   - One key block writes dQ where it belongs, which saves a launch (and the mask's words another).  Up to 64 queries, one or two steps,
//     always (B2 H4 S64 D32 11.4 and 10.9 us; at worst 32 queries, 64 keys, D32 1.07); to 128 where blocks of 32 keys gain as much or most
//     queries see no key.  Up to 512 queries from 0.35 (50 keys, 512 queries: 56 pairs D16 0.90, D64 0.89; 44 pairs D16 1.15), to 256 from
//     0.25 where the two kernels' dQ goes to 64-row tiles (20 keys, 256 queries, D16: 36 pairs 1.14, 40 pairs 0.81), beyond from 0.42, in
//     blocks of 64 keys up to head width 32 from 0.54 (1024 queries: 80 pairs D16 0.94, 64 pairs D64 0.87).  A tenth more for blocks of 64
//     keys at head widths 17 to 32 (0.05 to 0.1 slower than at others throughout), 0.15 for causal calls with dQ in 16-row tiles, which skip
//     more (B26 H2, 93 queries, 46 keys, D8 1.15).
//   - Several blocks: a CTA for each SM, or two thirds, above head width 32, where a tile has twice the warps, one third (128 CTAs, B4 H4
//     S512: D16 67 and 56 us, D32 103 and 77; 64 CTAs, B2 H4 S512 D64 105 and 93; 28 CTAs, B1 H4 S400 D64 70 and 80); there with more
//     than 512 queries and more than there are keys 0.54 (256 keys, 3000 queries: 16 pairs 1.07, 24 pairs 0.85).  Three quarters of that
//     in keys, since a last block may hold few.  Causal calls with dQ in 16-row tiles: in keys 0.75, above head width 32 0.37 (S256 D16
//     100 CTAs 1.00, 128 0.93; D64 40 CTAs 1.02, 64 0.91; S65, two blocks, D32 128 CTAs 1.25), unless a mask's words even that out.
//   - Several launches drain one by one, and a causal one lasts as long as the chain of the first keys, twice the mean.  Where a launch
//     has on average 0.6 of the CTAs that are resident at once; causal 0.6 in two launches, a tenth more for each further one, 0.9 in
//     the end.  Full, D64 S8192 13 pairs 0.80 of them 20270 and 16750, S10000 0.53 29170 and 39880; D32 S6000 8 pairs 0.64 3920 and
//     3140, S10000 0.53 9730 and 10320.  Causal, two launches: D32 S6000 0.64 2510 and 2170, S8192 5 pairs 0.54 2740 and 2750; four:
//     S8192 8 pairs in two of 0.86 4300 and 3340, 13 in four of 0.70 6040 and 6180; seven: D64 S8192 0.80 11200 and 12210; one pair a
//     launch, D32 S12000 0.32 8240 and 14320.
static OnePass one_pass(const ltca_attn_params* p, int sms, size_t room) {
    OnePass o;
    const int64_t all = (int64_t)p->B * p->H, blocks = ((int64_t)p->Sk + 63) / 64;
    if (p->D > 64 || p->B > 65535 || p->H > 65535 || all > 0x7fffffff || blocks > 65535) return o;     // (B, H: as the two kernels' grids)
    o.ld = (p->D + 3) / 4 * 4;
    const bool narrow = p->D <= 32, small = p->Sk <= 32;                   // small: blocks of 32 keys
    const int unseeing = p->causal && p->Sq > p->Sk ? (p->Sq - p->Sk) / (small ? 32 : 64) * (small ? 32 : 64) : 0;
    const int rows = p->Sq - unseeing;                                     // less whole tiles of queries that see no key
    const bool dq64 = all * (((int64_t)p->Sq + 63) / 64) >= sms;           // the two kernels' dQ in 64-row tiles
    if (blocks == 1) {
        int need = rows > 512 ? (narrow && !small ? 54 : 42) : rows <= 256 && dq64 ? 25 : 35;
        if (narrow && p->D > 16 && !small) need += 10;
        if (p->causal && !dq64) need += 15;
        if (rows <= 64 || (rows <= 128 && ((small && (p->D <= 16 || p->keep_mask)) || (unseeing && dq64)))) need = 0;
        if (100 * all >= need * (int64_t)sms) o.pairs = (int)all;
        return o;
    }
    const size_t one = (size_t)blocks * p->Sq * o.ld * sizeof(float);
    const int64_t fit = (int64_t)((room < kPartBytes ? room : kPartBytes) / one);
    if (fit == 0) return o;
    const int64_t launches = (all + fit - 1) / fit, slots = (narrow ? 4 : 2) * (int64_t)sms;      // slots: CTAs resident at once
    // As many pairs a launch as there is room for, or as many in each where that takes less time: waves of CTAs, causal the chain (D32
    // 8 pairs S6000 7 + 1 3395 us, 4 + 4 3140; D16 S10000 5 + 3 5000, 4 + 4 5480).
    auto time = [&](int64_t n) { return p->causal ? (n * blocks > 2 * slots ? n * blocks : 2 * slots) : (n * blocks + slots - 1) / slots; };
    auto total = [&](int64_t n) { return (launches - 1) * time(n) + time(all - (launches - 1) * n); };
    int64_t pairs = (all + launches - 1) / launches;
    if (launches > 1 && total(pairs) >= total(fit)) pairs = fit;
    if (pairs * blocks < sms) {
        const bool skips = p->causal && rows > 64 && !dq64 && !p->keep_mask;
        const int need = skips ? (narrow ? 100 : 49) : narrow ? 66 : rows <= 512 || rows <= p->Sk ? 33 : 54;      // in keys three quarters
        if ((!skips && 100 * pairs * blocks < need * (int64_t)sms) || 400 * pairs * p->Sk < 3 * need * 64 * (int64_t)sms) return o;
    }
    const int64_t tenths = p->causal && launches > 2 ? (launches < 5 ? 4 + launches : 9) : 6;
    if (launches > 1 && 10 * all * blocks < tenths * launches * slots) return o;
    o.pairs = (int)pairs;
    o.bytes = pairs * one;
    return o;
}
size_t attn_bwd_fp32_workspace(const ltca_attn_params* p, bool shares) {
    return delta_bytes(p) + (p->D <= 128 ? mask_words_bytes(p) + (shares ? one_pass(p, kPlanSms, kPartBytes).bytes : 0) : 0);
}

int launch_attn_fwd_fp32(ltca_ctx* ctx, const ltca_attn_params* p) {
    if (p->D < 1 || p->D > kWideMaxD)
        return fail(ctx, LTCA_ERR_UNSUPPORTED, "fp32 attention supports head_dim 1..%d, got %d", kWideMaxD, p->D);
    CoreArgs a = make_args(p);
    return p->dtype == LTCA_BF16 ? dispatch<__nv_bfloat16>(ctx, a, false) : dispatch<float>(ctx, a, false);
}

bool attn_bwd_fp32_forms_dout(const ltca_ctx* ctx, const ltca_attn_params* p, const FromOutput& f) {
    const auto al = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    return p->dtype == LTCA_F32 && p->D <= 64 && (p->Sk <= 32 || p->Sk > 64) && !fills_sms(ctx, p->B, p->H, p->Sq) && f.E <= kFormDoutMaxE && (f.E % 8) == 0 &&
           (int64_t)p->B * p->Sq <= kFormDoutRows && al(f.dy) && al(f.wo);
}

int launch_attn_bwd_fp32(ltca_ctx* ctx, const ltca_attn_params* p, const FromOutput* from) {
    if (p->D < 1 || p->D > kWideMaxD)
        return fail(ctx, LTCA_ERR_UNSUPPORTED, "fp32 attention supports head_dim 1..%d, got %d", kWideMaxD, p->D);
    if (p->workspace_bytes < delta_bytes(p) || !p->workspace)
        return fail(ctx, LTCA_ERR_WORKSPACE, "backward needs %zu bytes of workspace", delta_bytes(p));
    CoreArgs a = make_args(p);
    a.delta = reinterpret_cast<float*>(p->workspace);
    if (from) {
        a.dy = from->dy; a.wo = from->wo; a.E = from->E;
        a.dy_batch = from->batch; a.dy_seq = from->seq;
    }
    if (p->D <= 128) {
        // delta, dQ's shares, the mask's words (not in a workspace sized without the mask); without room for the shares the two
        // kernels run
        const OnePass one = !from || p->Sk <= 32 ? one_pass(p, ctx->sm_device, p->workspace_bytes - delta_bytes(p)) : OnePass();
        const bool once = one.pairs > 0;
        if (once) {
            a.pairs = one.pairs;
            a.part_ld = one.ld;
            a.dq_part = one.bytes ? reinterpret_cast<float*>(reinterpret_cast<char*>(p->workspace) + delta_bytes(p)) : nullptr;
        }
        const void* words = nullptr;
        if (!once || p->Sk > 128) {
            if (int rc = mask_words_of(ctx, p, delta_bytes(p) + (once ? one.bytes : 0), &words)) return rc;
        }
        const MaskArgs m = mask_args(p, words);
        a.mask_bits = m.by_query;
        a.mask_nw = m.nk;
    }
    return p->dtype == LTCA_BF16 ? dispatch<__nv_bfloat16>(ctx, a, true) : dispatch<float>(ctx, a, true);
}

}  // namespace ltca
