// Device side of the learned path planner, shared by the planner kernels
// (abf_planner.cu) and the plan kernel (abf_kernels.cu), which runs the same
// feature + MLP code inline for ABF_PATH_AUTO queries when parameters are
// installed, so a batch pays no separate planner launch.
//
// The MLP is 16 -> 64 -> 64 -> 3 with ReLU; the three outputs predict
// log(microseconds) of the PROBE, UNION and HYBRID paths of one query.
// Parameter layout (ABF_PLANNER_PARAMS floats, include/adabool.h):
//   mu[16] sd[16] | W1[64][16] b1[64] | W2[64][64] b2[64] | W3[3][64] b3[3]
#pragma once

#include "abf_kernels.cuh"

namespace abf {
namespace plan_dev {
namespace {

constexpr int F = ABF_PLANNER_FEATURES;
constexpr int H = ABF_PLANNER_HIDDEN;
constexpr int O = ABF_PLANNER_OUTPUTS;
constexpr int kMu = 0, kSd = 16, kW1 = 32, kB1 = kW1 + H * F, kW2 = kB1 + H, kB2 = kW2 + H * H, kW3 = kB2 + H,
              kB3 = kW3 + O * H, kNParams = kB3 + O;
static_assert(kNParams == ABF_PLANNER_PARAMS, "parameter layout");
constexpr int kFeatThreads = 256;
constexpr int kFeatUnroll = 4;  // terms per thread per pass, their loads in flight together

__device__ __forceinline__ uint32_t lane() { return threadIdx.x & 31u; }

template <class T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ uint32_t warp_max(uint32_t v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = max(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

struct FeatCtx {
    uint32_t hybrid_min;
    uint64_t n_postings;
    uint32_t n_q;
};

__device__ __forceinline__ TermFeat load_feat(const TermFeat* p) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
    return TermFeat{__hiloint2double(int(v.y), int(v.x)), v.z, v.w};
}

// The 16 features of query q (and its plain lists' blocks), whose terms are
// terms[qb .. qe), computed by the whole CTA (kFeatThreads threads) into f[] in
// shared memory. The caller gives the range: inside a batch, offsets past the
// workspace's terms are an empty query and must not be followed here. Term ids >= n_terms are skipped;
// repeated terms count once per occurrence. The logarithm that each term adds
// is in a table (taken here, four per thread and step of 64-bit arithmetic, it
// was ~1 us a step: 20,000 terms are 20 steps). Each thread takes kFeatUnroll
// terms per pass and issues all their table loads before using any, so a
// query of thousands of terms costs a few memory latencies, not one per term.
__device__ void query_features(const IndexView& ix, const uint32_t* terms, uint64_t qb, uint64_t qe, uint32_t q,
                               const FeatCtx& c, float* f, unsigned long long* blocks = nullptr) {
    __shared__ unsigned long long s_b[2][kFeatThreads / 32];
    __shared__ double s_d[6][kFeatThreads / 32];
    __shared__ uint32_t s_u[4][kFeatThreads / 32];
    uint32_t n = 0, mx = 0, nd = 0, nl = 0;
    unsigned long long pb = 0, pm = 0;  // blocks of the plain lists, and of those HYBRID merges
    double S = 0, Q = 0, Cb = 0, Lg = 0, Sd = 0, Bnd = 0;
    const double inv_ads = 1.0 / double(ix.n_ads);
    for (uint64_t i0 = qb + threadIdx.x; i0 < qe; i0 += uint64_t(kFeatThreads) * kFeatUnroll) {
        uint32_t t[kFeatUnroll];
        uint4 e[kFeatUnroll];  // {first block, postings, dense bitmap, plain list}
        TermFeat w[kFeatUnroll];
#pragma unroll
        for (int u = 0; u < kFeatUnroll; ++u) {
            const uint64_t i = i0 + uint64_t(u) * kFeatThreads;
            t[u] = i < qe ? terms[i] : kNone;
        }
#pragma unroll
        for (int u = 0; u < kFeatUnroll; ++u) {
            const bool ok = t[u] < ix.n_terms;
            e[u] = ok ? __ldg(ix.term_info + t[u]) : make_uint4(0u, 0u, kNone, kNone);
            w[u] = ok ? load_feat(ix.term_feat + t[u]) : TermFeat{0.0, 0u, 0u};
        }
#pragma unroll
        for (int u = 0; u < kFeatUnroll; ++u) {
            if (t[u] >= ix.n_terms) continue;
            const uint32_t len = e[u].y;
            ++n;
            mx = max(mx, len);
            S += len;
            Q += double(len) * len;
            Cb += w[u].cbytes;
            Lg += w[u].log_miss;
            if (e[u].z != kNone) {
                ++nd;
                Sd += len;
            } else {
                const uint32_t nb = (len + ABF_BLOCK_POSTINGS - 1u) / ABF_BLOCK_POSTINGS;
                Bnd += nb;
                if (len < c.hybrid_min) ++nl;
                if (e[u].w != kNone) {
                    pb += nb;
                    if (len >= c.hybrid_min) pm += nb;
                }
            }
        }
    }
    const uint32_t w = threadIdx.x >> 5;
    n = warp_sum(n);
    nd = warp_sum(nd);
    nl = warp_sum(nl);
    mx = warp_max(mx);
    S = warp_sum(S);
    Q = warp_sum(Q);
    Cb = warp_sum(Cb);
    Lg = warp_sum(Lg);
    Sd = warp_sum(Sd);
    Bnd = warp_sum(Bnd);
    if (blocks) {
        pb = warp_sum(pb);
        pm = warp_sum(pm);
    }
    if (lane() == 0) {
        s_b[0][w] = pb; s_b[1][w] = pm;
        s_u[0][w] = n; s_u[1][w] = nd; s_u[2][w] = nl; s_u[3][w] = mx;
        s_d[0][w] = S; s_d[1][w] = Q; s_d[2][w] = Cb; s_d[3][w] = Lg; s_d[4][w] = Sd; s_d[5][w] = Bnd;
    }
    __syncthreads();
    if (blocks && threadIdx.x >= 32 && threadIdx.x < 34) {
        unsigned long long t = 0;
        for (int k = 0; k < kFeatThreads / 32; ++k) t += s_b[threadIdx.x - 32][k];
        blocks[threadIdx.x - 32] = t;
    }
    // each of the first 16 threads sums the warps' partials and computes one
    // feature (the transcendentals run side by side, not one after another)
    if (threadIdx.x < F) {
        n = nd = nl = mx = 0;
        S = Q = Cb = Lg = Sd = Bnd = 0;
        for (int k = 0; k < kFeatThreads / 32; ++k) {
            n += s_u[0][k]; nd += s_u[1][k]; nl += s_u[2][k]; mx = max(mx, s_u[3][k]);
            S += s_d[0][k]; Q += s_d[1][k]; Cb += s_d[2][k]; Lg += s_d[3][k]; Sd += s_d[4][k]; Bnd += s_d[5][k];
        }
        // Each thread picks its argument, then all take the logarithm at
        // once: inside the cases the ten calls would run one after another
        // (the plan kernel of one query 18 us, here 13).
        const double nn = n > 0 ? double(n) : 1.0;
        double r = 0.0;
        bool log = true;
        switch (threadIdx.x) {
            case 0: r = double(n); break;
            case 1: r = S; break;
            case 2: r = double(mx); break;
            case 3: r = S / nn; break;
            case 4: {
                const double mean = S / nn;
                r = sqrt(fmax(Q / nn - mean * mean, 0.0));
                break;
            }
            case 5: r = Cb; break;
            case 6: r = 1.0 - exp(Lg); log = false; break;
            case 7: r = double(nd); break;
            case 8: r = Sd / fmax(S, 1.0); log = false; break;
            case 9: r = Bnd; break;
            case 10: r = S / double(c.n_postings ? c.n_postings : 1); log = false; break;
            case 11: r = double(nl); break;
            case 12: r = double(q) / double(c.n_q ? c.n_q : 1); log = false; break;
            case 13: r = double(c.n_q); break;
            case 14: r = double(mx) * inv_ads; log = false; break;
            default: r = 1.0; log = false; break;
        }
        if (log) r = log1p(r);
        f[threadIdx.x] = float(r);
    }
    __syncthreads();
}

// MLP forward on standardised x (shared, F floats) by threads 0..63:
// h1, h2 (shared, H each, post-ReLU) and y (shared, O).
__device__ __forceinline__ void mlp_forward_cta(const float* __restrict__ p, const float* xs, float* h1, float* h2,
                                                float* y) {
    const int j = threadIdx.x;
    if (j < H) {
        float a = __ldg(p + kB1 + j);
#pragma unroll
        for (int k = 0; k < F; ++k) a = fmaf(__ldg(p + kW1 + j * F + k), xs[k], a);
        h1[j] = fmaxf(a, 0.0f);
    }
    __syncthreads();
    if (j < H) {
        float a = __ldg(p + kB2 + j);
#pragma unroll 8
        for (int k = 0; k < H; ++k) a = fmaf(__ldg(p + kW2 + j * H + k), h1[k], a);
        h2[j] = fmaxf(a, 0.0f);
    }
    __syncthreads();
    if (j < O) {
        float a = __ldg(p + kB3 + j);
#pragma unroll 8
        for (int k = 0; k < H; ++k) a = fmaf(__ldg(p + kW3 + j * H + k), h2[k], a);
        y[j] = a;
    }
    __syncthreads();
}

// The state the planner keeps in shared memory: the parameters, copied in once
// per CTA, and one query's values.
constexpr int kParamVecs = (kNParams + 3) / 4;
struct PlannerSmem {
    float4 p4[kParamVecs];
    float f[F], xs[F], h1[H], h2[H], y[O];
    unsigned long long blocks[2];  // of the query's plain lists, and of those HYBRID merges
    __device__ const float* p() const { return reinterpret_cast<const float*>(p4); }
};

// Starts the copy of the parameters (16-byte aligned); planner_path waits for it.
__device__ __forceinline__ void load_params(const float* __restrict__ p, PlannerSmem& sm) {
    for (int i = threadIdx.x; i < kNParams / 4; i += kFeatThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(sm.p4 + i))),
                     "l"(reinterpret_cast<const float4*>(p) + i)
                     : "memory");
    for (int i = kNParams / 4 * 4 + threadIdx.x; i < kNParams; i += kFeatThreads)
        reinterpret_cast<float*>(sm.p4)[i] = __ldg(p + i);
    asm volatile("cp.async.commit_group;" ::: "memory");
}

// MLP forward on standardised x by the whole CTA: four threads per hidden unit
// (a quarter of its inputs each, in 16-byte steps whose order turns with the
// unit, so that a warp's eight units read all banks), a warp per output.
__device__ __forceinline__ void mlp_forward_smem(PlannerSmem& sm) {
    const int j = threadIdx.x >> 2, r = threadIdx.x & 3, w = threadIdx.x >> 5, l = threadIdx.x & 31;
    static_assert(kFeatThreads == 4 * H && F == 16 && H == 64, "four threads per unit");
    const float* p = sm.p();
    {
        const float4 v = *reinterpret_cast<const float4*>(p + kW1 + j * F + 4 * r);
        float a = fmaf(v.w, sm.xs[4 * r + 3], fmaf(v.z, sm.xs[4 * r + 2], fmaf(v.y, sm.xs[4 * r + 1], v.x * sm.xs[4 * r])));
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        if (r == 0) sm.h1[j] = fmaxf(a + p[kB1 + j], 0.0f);
    }
    __syncthreads();
    {
        float a = 0.0f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = 16 * r + 4 * ((i + j) & 3);
            const float4 v = *reinterpret_cast<const float4*>(p + kW2 + j * H + k);
            a = fmaf(v.w, sm.h1[k + 3], fmaf(v.z, sm.h1[k + 2], fmaf(v.y, sm.h1[k + 1], fmaf(v.x, sm.h1[k], a))));
        }
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        if (r == 0) sm.h2[j] = fmaxf(a + p[kB2 + j], 0.0f);
    }
    __syncthreads();
    if (w < O) {
        const float* q = p + kW3 + w * H;
        float a = fmaf(q[l + 32], sm.h2[l + 32], q[l] * sm.h2[l]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (l == 0) sm.y[w] = a + p[kB3 + w];
    }
    __syncthreads();
}

// features -> standardise -> MLP -> cheapest path (an abf_path) of query q (terms[qb .. qe)),
// by the whole CTA (kFeatThreads threads), after load_params; sm.f holds the
// features and sm.y the predictions afterwards.
__device__ __forceinline__ uint32_t planner_path(const IndexView& ix, const uint32_t* terms, uint64_t qb, uint64_t qe,
                                                 uint32_t q, const FeatCtx& c, PlannerSmem& sm) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    query_features(ix, terms, qb, qe, q, c, sm.f, sm.blocks);  // ends with a barrier: every thread's copies are there
    if (threadIdx.x < F) {
        const float sd = sm.p()[kSd + threadIdx.x];
        sm.xs[threadIdx.x] = (sm.f[threadIdx.x] - sm.p()[kMu + threadIdx.x]) / (sd > 0.0f ? sd : 1.0f);
    }
    __syncthreads();
    mlp_forward_smem(sm);
    int best = 0;
    for (int o = 1; o < O; ++o)
        if (sm.y[o] < sm.y[best]) best = o;
    return best == 0 ? ABF_PATH_PROBE : best == 1 ? ABF_PATH_UNION : ABF_PATH_HYBRID;
}

}  // namespace
}  // namespace plan_dev
}  // namespace abf
