// Single-query attention over a key/value cache with per-sequence lengths.  The work is pure
// streaming of K and V (about 0.5 FLOP per byte), so the kernel is built around wide coalesced
// loads and keeps all arithmetic in fp32 registers:
//   - a group of lanes owns one key at a time (each lane 16 bytes of the row), the score is a shuffle
//     reduction inside the group, the value row is accumulated by the same lanes without further
//     communication; the next keys are loaded while these are multiplied;
//   - every group runs its own online softmax over the keys it visits; a warp's groups are merged by
//     shuffles, a CTA's warps through shared memory;
//   - a pair's keys are split over several CTAs where batch x heads cannot fill the GPU, and over two
//     or four where it does but the sequences differ in length (less of a tail in which only the
//     longest are still streaming).  Up to 16 CTAs of a pair are one thread-block cluster whose
//     first CTA receives the others' partial (max, sum, output) triples in its shared memory; more
//     go through a caller-provided scratch buffer and a second small kernel.
// The reference has no counterpart: its cuDNN call always passes currIdx = -1
// (reference src/ml/cuDNN_ops.cu:206).
#include <cooperative_groups.h>
#include <math.h>

#include "host_common.h"
#include "sm100_ptx.cuh"

namespace ltca {

namespace {

constexpr int kMaxCluster = 16;             // CTAs of one (batch, head) pair that merge through shared memory
constexpr int kUnroll = 4;                  // keys per group and iteration
constexpr int kStages = 2;                  // iterations of keys in shared memory, all but one of them in flight
// Whether the keys go through a ring in shared memory or straight to registers (see attn_decode_kernel).
template <typename T, int W, int kSplit>
constexpr bool kRing = !(sizeof(T) == 4 && W == 4 && kSplit == 0);
template <typename T, int W, int kSplit>
constexpr int kRingBytes = kRing<T, W, kSplit> ? kStages * kUnroll * 2 * 32 * W * 16 : 0;

struct DecodeArgs {
    int B, H, Sk, D;
    float scale, clamp;
    int use_clamp;
    const void *q, *k, *v;
    void* o;
    ltca_strides qs, ks, vs, os;
    float* lse;
    const float* keep_mask;     // [B, 1, Sk]
    const int32_t* kv_len;
    int nsplit;
    int vec16;                  // every K and V row starts on a 16-byte boundary
    float* partial;             // [B*H][nsplit][D + 2]; null when the splits are one cluster
};

// A lane's 16 bytes of a row: 4 fp32 or 8 bf16 values.
template <typename T>
constexpr int kLaneElems = 16 / (int)sizeof(T);
__device__ __forceinline__ uint4 ld_lane(const float* p) { return __ldg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ uint4 ld_lane(const __nv_bfloat16* p) {
    const uint2 a = __ldg(reinterpret_cast<const uint2*>(p)), b = __ldg(reinterpret_cast<const uint2*>(p) + 1);
    return make_uint4(a.x, a.y, b.x, b.y);
}
// The same 16 bytes into this lane's own slot of the shared ring.
template <typename T>
__device__ __forceinline__ void fetch_lane(uint32_t dst, const T* p, bool vec16) {
    if (sizeof(T) == 4 || vec16) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(p) : "memory");
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(p) : "memory");
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + 8), "l"(p + 4) : "memory");
    }
}
__device__ __forceinline__ void unpack(const uint4& u, float (&v)[4]) {
    v[0] = __uint_as_float(u.x); v[1] = __uint_as_float(u.y); v[2] = __uint_as_float(u.z); v[3] = __uint_as_float(u.w);
}
__device__ __forceinline__ void unpack(const uint4& u, float (&v)[8]) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = __uint_as_float(w[i] << 16);
        v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
}
__device__ __forceinline__ void st1(float* p, float v) { *p = v; }
__device__ __forceinline__ void st1(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

// Result of a (batch, head) pair from n partials (max, sum, D unnormalised outputs), by the first D threads.
template <typename T>
__device__ __forceinline__ void merge_partials(const DecodeArgs& a, const float* part, int n, int b, int h) {
    const int d = threadIdx.x, stride = a.D + 2;
    float M = -INFINITY;
    for (int s = 0; s < n; ++s) M = fmaxf(M, part[s * stride]);
    const float Ms = (M == -INFINITY) ? 0.f : M;
    float L = 0.f, acc = 0.f;
    for (int s = 0; s < n; ++s) {
        const float* ps = part + s * stride;
        const float w = (ps[0] == -INFINITY) ? 0.f : expf(ps[0] - Ms);
        L = fmaf(ps[1], w, L);
        acc = fmaf(ps[2 + d], w, acc);
    }
    T* op = reinterpret_cast<T*>(a.o) + b * a.os.batch + h * a.os.head;
    st1(op + d, L > 0.f ? acc / L : 0.f);
    if (d == 0 && a.lse) a.lse[(int64_t)b * a.H + h] = L > 0.f ? M + logf(L) : -INFINITY;
}

// LPK lanes own one key at a time.  kSplit 0: one CTA per pair; 1: the nsplit CTAs of a pair form a cluster (1, nsplit, 1)
// whose first CTA receives the others' partials in its shared memory; 2: partials go to scratch for a second kernel.
template <typename T, int LPK, int W, int kSplit>
__global__ void __launch_bounds__(32 * W) attn_decode_kernel(const DecodeArgs a) {
    constexpr int EL = kLaneElems<T>;
    constexpr int D = EL * LPK;
    constexpr int G = 32 / LPK;                         // key groups per warp
    constexpr int NG = W * G;                           // key groups per CTA
    // The ring: every lane has slots of its own and reads back only what it fetched itself, so the pipeline needs no
    // barrier and holds no registers for keys in flight.  Where fp32 caches of one length fill the GPU with pairs, plain
    // loads of one iteration at a time are the better stream (B=32 H=16 D=128, 2000 keys each: 170 us against 190; 8 CTAs
    // per SM); with lengths that differ, with bf16 rows (twice the arithmetic per byte) and with few CTAs it is the
    // ring: B=64 H=16 D=64 bf16 up to 4000 keys 85 us against 114.
    extern __shared__ __align__(16) unsigned char ring[];
    __shared__ __align__(16) float sm_o[W][D];
    __shared__ float sm_m[W], sm_l[W];
    __shared__ float sm_part[kSplit == 1 ? kMaxCluster * (D + 2) : 1];
    namespace cg = cooperative_groups;
    grid_dependency_wait();
    // the other CTAs of the cluster may be written to once they have started: waited for behind the key loop
    if (kSplit == 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");

    const int bh = blockIdx.x;
    const int b = bh / a.H, h = bh % a.H;
    const int split = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = warp * G + lane / LPK;
    const int sub = lane % LPK;

    // the CTA's splits interleave at the granularity of one iteration (NG * kUnroll keys), so only
    // the sequence's last iteration is ragged, whatever the split count
    int ke = a.Sk;
    if (a.kv_len) ke = min(max(a.kv_len[b], 0), a.Sk);
    const T* qp = reinterpret_cast<const T*>(a.q) + b * a.qs.batch + h * a.qs.head + EL * sub;
    const T* kp = reinterpret_cast<const T*>(a.k) + b * a.ks.batch + h * a.ks.head + EL * sub;
    const T* vp = reinterpret_cast<const T*>(a.v) + b * a.vs.batch + h * a.vs.head + EL * sub;
    const float* mrow = a.keep_mask ? a.keep_mask + (int64_t)b * a.Sk : nullptr;
    const bool vec16 = a.vec16 != 0;
    float q[EL];
    unpack(ld_lane(qp), q);
#pragma unroll
    for (int i = 0; i < EL; ++i) q[i] *= a.scale;

    float m = -INFINITY, l = 0.f, o[EL];
#pragma unroll
    for (int i = 0; i < EL; ++i) o[i] = 0.f;
    const int iters = (ke + NG * kUnroll - 1) / (NG * kUnroll);

    const uint32_t slot0 = smem_u32(ring) + threadIdx.x * 16;
    constexpr uint32_t kSlot = 32 * W * 16, kStage = 2 * kUnroll * kSlot;
    auto key_of = [&](int it, int u) { return (it * kUnroll + u) * NG + g; };
    auto fetch = [&](int it, int stage) {
        if (it < iters) {
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const int j = min(key_of(it, u), ke - 1);            // in range: ke > 0 here
                fetch_lane(slot0 + stage * kStage + 2 * u * kSlot, kp + (int64_t)j * a.ks.seq, vec16);
                fetch_lane(slot0 + stage * kStage + (2 * u + 1) * kSlot, vp + (int64_t)j * a.vs.seq, vec16);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // key(u), value(u): this lane's 16 bytes of key u's rows; live[u]: the key is visible
    auto consume = [&](auto key, auto value, const bool (&live)[kUnroll]) {
        float s[kUnroll];
        float mt = m;
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            float kk[EL];
            unpack(key(u), kk);
            float d = q[0] * kk[0];
#pragma unroll
            for (int i = 1; i < EL; ++i) d = fmaf(q[i], kk[i], d);
#pragma unroll
            for (int off = LPK / 2; off > 0; off >>= 1) d += __shfl_xor_sync(0xffffffffu, d, off);
            if (a.use_clamp) d = fminf(d, a.clamp);
            s[u] = live[u] ? d : -INFINITY;
            mt = fmaxf(mt, s[u]);
        }
        const float m_safe = (mt == -INFINITY) ? 0.f : mt;
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_safe);
        l *= corr;
#pragma unroll
        for (int i = 0; i < EL; ++i) o[i] *= corr;
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const float p = expf(s[u] - m_safe);
            l += p;
            float vv[EL];
            unpack(value(u), vv);
#pragma unroll
            for (int i = 0; i < EL; ++i) o[i] = fmaf(p, vv[i], o[i]);
        }
        m = mt;
    };
    if constexpr (!kRing<T, W, kSplit>) {
        for (int it = split; it < iters; it += a.nsplit) {
            uint4 kk[kUnroll], vv[kUnroll];
            bool live[kUnroll];
            // (the mask test between the loads keeps the compiler from moving the values' loads behind the scores)
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const int j = key_of(it, u);
                live[u] = j < ke;
                const int jj = live[u] ? j : (ke - 1);
                kk[u] = ld_lane(kp + (int64_t)jj * a.ks.seq);
                vv[u] = ld_lane(vp + (int64_t)jj * a.vs.seq);
                if (live[u] && mrow && mrow[j] == 0.f) live[u] = false;
            }
            consume([&](int u) { return kk[u]; }, [&](int u) { return vv[u]; }, live);
        }
    } else {
        int stage = 0;
#pragma unroll
        for (int i = 0; i < kStages - 1; ++i) fetch(split + i * a.nsplit, i);
        for (int it = split; it < iters; it += a.nsplit) {
            fetch(it + (kStages - 1) * a.nsplit, (stage + kStages - 1) % kStages);
            bool live[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) {
                const int j = key_of(it, u);
                live[u] = j < ke && !(mrow && mrow[j] == 0.f);
            }
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 1) : "memory");
            const unsigned char* mine = ring + threadIdx.x * 16 + stage * kStage;
            consume([&](int u) { return *reinterpret_cast<const uint4*>(mine + 2 * u * kSlot); },
                    [&](int u) { return *reinterpret_cast<const uint4*>(mine + (2 * u + 1) * kSlot); }, live);
            stage = (stage + 1) % kStages;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    // Only now may the next kernel's CTAs be placed: released at the start they take whatever slots the SMs have left, and
    // the next decode step's pairs then sit unevenly on the SMs (B=32 H=16 D=128, 2000 keys: 214 us against 170).
    grid_launch_dependents();
    // the groups of a warp, then the warps of the CTA
#pragma unroll
    for (int off = LPK; off < 32; off <<= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, off), l2 = __shfl_xor_sync(0xffffffffu, l, off);
        const float mm = fmaxf(m, m2), ms = (mm == -INFINITY) ? 0.f : mm;
        const float w1 = (m == -INFINITY) ? 0.f : expf(m - ms), w2 = (m2 == -INFINITY) ? 0.f : expf(m2 - ms);
        l = l * w1 + l2 * w2;
#pragma unroll
        for (int i = 0; i < EL; ++i) o[i] = o[i] * w1 + __shfl_xor_sync(0xffffffffu, o[i], off) * w2;
        m = mm;
    }
    if (lane < LPK) {
#pragma unroll
        for (int i = 0; i < EL; i += 4)
            *reinterpret_cast<float4*>(&sm_o[warp][EL * sub + i]) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
    }
    if (lane == 0) { sm_m[warp] = m; sm_l[warp] = l; }
    __syncthreads();
    if (kSplit == 1) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (threadIdx.x < D) {
        const int d = threadIdx.x;
        float M = -INFINITY;
#pragma unroll
        for (int i = 0; i < W; ++i) M = fmaxf(M, sm_m[i]);
        const float Ms = (M == -INFINITY) ? 0.f : M;
        float L = 0.f, acc = 0.f;
#pragma unroll
        for (int i = 0; i < W; ++i) {
            const float w = (sm_m[i] == -INFINITY) ? 0.f : expf(sm_m[i] - Ms);
            L = fmaf(sm_l[i], w, L);
            acc = fmaf(sm_o[i][d], w, acc);
        }
        if (kSplit == 0) {
            T* op = reinterpret_cast<T*>(a.o) + b * a.os.batch + h * a.os.head;
            st1(op + d, L > 0.f ? acc / L : 0.f);
            if (d == 0 && a.lse) a.lse[bh] = L > 0.f ? M + logf(L) : -INFINITY;
        } else {
            float* part = kSplit == 1 ? cg::this_cluster().map_shared_rank(sm_part, 0) + split * (D + 2)
                                      : a.partial + ((int64_t)bh * a.nsplit + split) * (D + 2);
            part[2 + d] = acc;
            if (d == 0) { part[0] = M; part[1] = L; }
        }
    }
    if (kSplit == 1) {
        cg::this_cluster().sync();                       // every partial is in the first CTA's shared memory
        if (split == 0 && threadIdx.x < D) merge_partials<T>(a, sm_part, a.nsplit, b, h);
    }
}

template <typename T>
__global__ void __launch_bounds__(128) attn_decode_merge_kernel(const DecodeArgs a) {
    grid_dependency_wait();
    const int bh = blockIdx.x;
    if ((int)threadIdx.x < a.D) merge_partials<T>(a, a.partial + (int64_t)bh * a.nsplit * (a.D + 2), a.nsplit, bh / a.H, bh % a.H);
}

// How a (batch, head) pair's keys are dealt out.  cluster: the splits merge through distributed shared memory; few: the
// pairs alone do not fill the GPU.
struct SplitPlan { int n; bool cluster; bool few; };
SplitPlan plan_splits(const ltca_attn_params* p) {
    SplitPlan s{1, false, false};
    if (p->B < 1 || p->H < 1 || p->Sk < 1 || p->D < 1) return s;      // (nothing to split, no division by zero below)
    constexpr int sms = kPlanSms;
    const int64_t bh = (int64_t)p->B * p->H;
    if (bh >= 2 * sms) {
        // With lengths that differ, two or four CTAs take alternate blocks of a pair's keys, so that the longest
        // sequences do not stream alone at the end; measured at B=256 H=8 lengths U{1..1024}: 2 CTAs 6112 GB/s,
        // 4: 6011, 8: 4869 (1: 4820).
        if (p->kv_len && p->Sk >= 512) { s.n = p->Sk < 2048 ? 2 : 4; s.cluster = true; }
        return s;
    }
    // About three CTAs of eight warps per SM, each with at least two iterations of keys.  Up to 16 splits are one
    // cluster and one launch; where a pair has the keys and the GPU the room for more, scratch and a merge kernel.
    s.few = true;
    const int es = p->dtype == LTCA_BF16 ? 2 : 4;
    const int64_t iter = 8 * kUnroll * 32 * 16 / ((int64_t)p->D * es);        // keys per iteration of an 8-warp CTA
    const int64_t want = (3 * (int64_t)sms + bh - 1) / bh, cap = (p->Sk + 2 * iter - 1) / (2 * (iter > 0 ? iter : 1));
    int64_t n = want < cap ? want : cap;
    if (n > 64) n = 64;
    if (n > kMaxCluster) {
        s.n = (int)n;
        return s;
    }
    while (s.n < n) s.n *= 2;
    s.cluster = s.n > 1;
    return s;
}

template <typename T, int LPK, int W, int kSplit>
int launch_decode(ltca_ctx* ctx, const DecodeArgs& a) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(a.B * a.H, a.nsplit);
    cfg.blockDim = dim3(32 * W);
    cfg.dynamicSmemBytes = kRingBytes<T, W, kSplit>;
    cfg.stream = ctx->stream;
    static SmemOptIn once;
    if (kRingBytes<T, W, kSplit> > 40 * 1024)
        LTCA_CUDA_OK(ctx, opt_in_dynamic_smem(once, ctx->device, attn_decode_kernel<T, LPK, W, kSplit>, kRingBytes<T, W, kSplit>));
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = 1;
    attr[1].val.clusterDim.y = (unsigned)a.nsplit;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = kSplit == 1 ? 2 : 1;
    if (kSplit == 1 && a.nsplit > 8) {
        static SmemOptIn wide;      // clusters of more than eight CTAs are an opt-in of a kernel on one device
        const uint64_t bit = (ctx->device >= 0 && ctx->device < 64) ? (1ull << ctx->device) : 0ull;
        if (!bit || !(wide.done.load(std::memory_order_acquire) & bit)) {
            LTCA_CUDA_OK(ctx, cudaFuncSetAttribute(attn_decode_kernel<T, LPK, W, kSplit>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
            wide.done.fetch_or(bit, std::memory_order_release);
        }
    }
    LTCA_CUDA_OK(ctx, cudaLaunchKernelEx(&cfg, attn_decode_kernel<T, LPK, W, kSplit>, a));
    return LTCA_OK;
}

template <typename T, int LPK>
int run_decode(ltca_ctx* ctx, const DecodeArgs& a, const SplitPlan& plan) {
    if (plan.cluster) return plan.few ? launch_decode<T, LPK, 8, 1>(ctx, a) : launch_decode<T, LPK, 4, 1>(ctx, a);
    if (plan.n == 1) return plan.few ? launch_decode<T, LPK, 8, 0>(ctx, a) : launch_decode<T, LPK, 4, 0>(ctx, a);
    if (int rc = launch_decode<T, LPK, 8, 2>(ctx, a)) return rc;
    LTCA_CUDA_OK(ctx, launch_dependent(attn_decode_merge_kernel<T>, dim3(a.B * a.H), dim3(128), 0, ctx->stream, a));
    return LTCA_OK;
}

template <typename T>
int dispatch_decode(ltca_ctx* ctx, const DecodeArgs& a, const SplitPlan& plan) {
    constexpr int EL = kLaneElems<T>;
    switch (a.D) {
        case 16: return run_decode<T, 16 / EL>(ctx, a, plan);
        case 32: return run_decode<T, 32 / EL>(ctx, a, plan);
        case 64: return run_decode<T, 64 / EL>(ctx, a, plan);
        case 128: return run_decode<T, 128 / EL>(ctx, a, plan);
    }
    return fail(ctx, LTCA_ERR_UNSUPPORTED, "decode supports head_dim 16, 32, 64, 128 (got %d)", a.D);
}

// Bytes of the partial results of n splits per pair.
size_t partial_bytes(const ltca_attn_params* p, int64_t n) {
    return n > 1 ? align_up((size_t)p->B * p->H * n * (p->D + 2) * sizeof(float), 256) : 0;
}

}  // namespace

// The split count must not depend on the context, so that the size query (which has no
// context) and the launch agree.  Non-positive shapes need no scratch (the launch refuses them).
// The answer is never below what the partials would take at one CTA per 256 keys and four per SM, although splits that
// merge inside a cluster use no scratch: by that size ltca_attn_decode_static tells the shapes it takes from those it
// refuses, and which it takes does not move with the split.
size_t attn_decode_workspace(const ltca_attn_params* p) {
    if (p->B < 1 || p->H < 1 || p->Sk < 1 || p->D < 1) return 0;
    const SplitPlan s = plan_splits(p);
    if (!s.few) return 0;
    const int64_t bh = (int64_t)p->B * p->H, want = (4 * (int64_t)kPlanSms + bh - 1) / bh, cap = (p->Sk + 255) / 256;
    int64_t n = want < cap ? want : cap;
    if (n > 64) n = 64;
    if (!s.cluster && s.n > n) n = s.n;
    return partial_bytes(p, n);
}

int launch_attn_decode(ltca_ctx* ctx, const ltca_attn_params* p) {
    if (p->Sq != 1) return fail(ctx, LTCA_ERR_INVALID, "decode needs Sq == 1 (got %d)", p->Sq);
    const int es = elem_size(p->dtype);
    const int vec = 4 * es;     // bytes per lane load
    auto misaligned = [&](const void* ptr, const ltca_strides& s) {
        return (reinterpret_cast<uintptr_t>(ptr) % vec) || ((s.seq * es) % vec) ||
               ((s.head * es) % vec) || ((s.batch * es) % vec);
    };
    if (misaligned(p->q, p->q_strides) || misaligned(p->k, p->k_strides) ||
        misaligned(p->v, p->v_strides))
        return fail(ctx, LTCA_ERR_INVALID, "decode needs %d-byte aligned q/k/v rows", vec);
    DecodeArgs a;
    memset(&a, 0, sizeof(a));
    a.B = p->B; a.H = p->H; a.Sk = p->Sk; a.D = p->D;
    a.scale = p->scale;
    a.use_clamp = p->score_clamp > 0.f ? 1 : 0;
    a.clamp = p->score_clamp;
    a.q = p->q; a.k = p->k; a.v = p->v; a.o = p->o;
    a.qs = p->q_strides; a.ks = p->k_strides; a.vs = p->v_strides; a.os = p->o_strides;
    a.lse = p->lse;
    a.keep_mask = p->keep_mask;
    a.kv_len = p->kv_len;
    a.vec16 = 1;
    for (const ltca_strides* st : {&p->k_strides, &p->v_strides})
        if ((st->seq * es) % 16 || (st->head * es) % 16 || (st->batch * es) % 16) a.vec16 = 0;
    if ((reinterpret_cast<uintptr_t>(p->k) | reinterpret_cast<uintptr_t>(p->v)) % 16) a.vec16 = 0;
    const SplitPlan plan = plan_splits(p);
    a.nsplit = plan.n;
    if (plan.n > 1 && !plan.cluster) {
        const size_t need = partial_bytes(p, plan.n);
        if (!p->workspace || p->workspace_bytes < need)
            return fail(ctx, LTCA_ERR_WORKSPACE, "decode needs %zu bytes of workspace", need);
        a.partial = reinterpret_cast<float*>(p->workspace);
    }
    return p->dtype == LTCA_BF16 ? dispatch_decode<__nv_bfloat16>(ctx, a, plan)
                                 : dispatch_decode<float>(ctx, a, plan);
}

}  // namespace ltca

// ---------------------------------------------------------------------------------------------
// Allocation-free variant of the decode step.
//
// The regular entry point needs a context (whose creation makes one small device allocation)
// and, when the key range is split, a scratch buffer that the caller has to allocate.  Code
// that runs where device allocation is off limits -- a plug-in called from inside another
// framework's memory pool or arena, a real-time loop that forbids driver allocations after
// start-up, a host that hands out all device memory up front -- cannot provide either.  For
// those callers the split's partial results live in a fixed array that is part of the loaded
// library image, so the call touches no allocator at all.
// ---------------------------------------------------------------------------------------------
namespace {

constexpr size_t kStaticScratchBytes = 256u << 10;   // 256 KiB, resident on every GPU that loads the library
static __device__ __align__(256) unsigned char g_decode_static_scratch[kStaticScratchBytes];

// Device address of the array on each GPU, looked up on the first call there.  Host threads that make that
// first call at the same time all store the same value, hence relaxed atomics are enough.
constexpr int kMaxDevices = 64;
std::atomic<void*> g_static_scratch_ptr[kMaxDevices];

void set_err(char* buf, size_t len, const char* msg) {
    if (buf && len) snprintf(buf, len, "%s", msg);
}

}  // namespace

extern "C" int ltca_attn_decode_static(void* stream, const ltca_attn_params* p, char* err,
                                       size_t err_len) {
    if (!p) { set_err(err, err_len, "null parameter block"); return LTCA_ERR_INVALID; }
    // Arguments first: nothing below may divide by, or size a buffer from, a shape that is not positive.
    if (p->B < 1 || p->H < 1 || p->Sk < 1 || p->D < 1 || !p->q || !p->k || !p->v || !p->o ||
        !(p->scale > 0.f) || (p->dtype != LTCA_F32 && p->dtype != LTCA_BF16)) {
        set_err(err, err_len, "bad decode arguments (shape, null pointer, scale or dtype)");
        return LTCA_ERR_INVALID;
    }
    if (p->Sq != 1) {
        set_err(err, err_len, "decode needs Sq == 1");
        return LTCA_ERR_INVALID;
    }
    const size_t need = ltca::attn_decode_workspace(p);
    if (need > kStaticScratchBytes) {
        char msg[200];
        snprintf(msg, sizeof(msg),
                 "ltca_attn_decode_workspace_bytes answers %zu for this shape, this entry point takes up to %zu; "
                 "use ltca_attn_decode with a caller-provided workspace", need, kStaticScratchBytes);
        set_err(err, err_len, msg);
        return LTCA_ERR_WORKSPACE;
    }
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
        set_err(err, err_len, "no current CUDA device (or device index above 63)");
        return LTCA_ERR_NO_DEVICE;
    }
    // One-time set-up per device, with that device current: in host code the array's name is
    // only a stand-in, the kernel needs the address the symbol has on THIS device.
    void* scratch = g_static_scratch_ptr[dev].load(std::memory_order_relaxed);
    if (!scratch) {
        cudaError_t e = cudaGetSymbolAddress(&scratch, g_decode_static_scratch);
        if (e != cudaSuccess || !scratch) {
            set_err(err, err_len, cudaGetErrorString(e));
            return LTCA_ERR_CUDA;
        }
        g_static_scratch_ptr[dev].store(scratch, std::memory_order_relaxed);
    }
    ltca_ctx tmp;                       // host-only bookkeeping: stream and error text
    tmp.device = dev;
    tmp.stream = reinterpret_cast<cudaStream_t>(stream);
    tmp.sm_count = tmp.sm_device = ltca::kPlanSms;    // only the split plan uses it, and that is fixed (see kPlanSms)
    ltca_attn_params q = *p;
    q.workspace = scratch;
    q.workspace_bytes = kStaticScratchBytes;
    const int rc = ltca::launch_attn_decode(&tmp, &q);
    if (rc) set_err(err, err_len, tmp.err);
    return rc;
}
