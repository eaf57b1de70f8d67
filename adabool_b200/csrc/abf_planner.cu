// Learned path planner: per-query features, the fused feature + MLP
// inference kernel used inside abf_batch_run, and the MLP's training
// kernels (forward, mean-squared-error gradient, Adam), all FP32 SIMT.
//
// The MLP is 16 -> 64 -> 64 -> 3 with ReLU; the three outputs predict
// log(microseconds) of the PROBE, UNION and HYBRID paths of one query.
// Parameter layout (ABF_PLANNER_PARAMS floats, include/adabool.h):
//   mu[16] sd[16] | W1[64][16] b1[64] | W2[64][64] b2[64] | W3[3][64] b3[3]
// No reference counterpart: the reference runs both of its paths on every
// query (test/adsfilter_q_all.cu:414-452) and has no selection rule.
#include "abf_planner_dev.cuh"

#include <atomic>
#include <cmath>

namespace abf {

namespace {

using namespace plan_dev;

// Fused planner: features -> standardise -> MLP -> cheapest path.
__global__ void __launch_bounds__(kFeatThreads) planner_kernel(IndexView ix, const float* __restrict__ p,
                                                               const uint32_t* terms, const uint64_t* q_off,
                                                               FeatCtx c, float* feat_out, float* pred_out,
                                                               uint8_t* path_out) {
    __shared__ PlannerSmem sm;
    if (p) load_params(p, sm);
    for (uint32_t q = blockIdx.x; q < c.n_q; q += gridDim.x) {
        if (!p) {
            query_features(ix, terms, q_off[q], q_off[q + 1], q, c, sm.f);
            if (feat_out && threadIdx.x < F) feat_out[uint64_t(q) * F + threadIdx.x] = sm.f[threadIdx.x];
            continue;
        }
        const uint32_t path = planner_path(ix, terms, q_off[q], q_off[q + 1], q, c, sm);
        if (feat_out && threadIdx.x < F) feat_out[uint64_t(q) * F + threadIdx.x] = sm.f[threadIdx.x];
        if (threadIdx.x == 0) {
            if (pred_out)
                for (int o = 0; o < O; ++o) pred_out[uint64_t(q) * O + o] = sm.y[o];
            if (path_out) path_out[q] = uint8_t(path);
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(64) mlp_forward_kernel(const float* __restrict__ p, const float* x, uint32_t n,
                                                         float* y_out) {
    __shared__ float xs[F], h1[H], h2[H], y[O];
    for (uint32_t s = blockIdx.x; s < n; s += gridDim.x) {
        if (threadIdx.x < F) xs[threadIdx.x] = x[uint64_t(s) * F + threadIdx.x];
        __syncthreads();
        mlp_forward_cta(p, xs, h1, h2, y);
        if (threadIdx.x < O) y_out[uint64_t(s) * O + threadIdx.x] = y[threadIdx.x];
        __syncthreads();
    }
}

// d_grad and the loss zeroed, the masked entries counted: one CTA, for a
// batch of up to kInitSamples samples (its mask is at most 192 KB, a few
// loads in flight per thread), so that a training step has one launch here
// instead of two memsets and a counting kernel.
constexpr uint32_t kInitSamples = 16384;
__global__ void __launch_bounds__(1024) grad_init_kernel(const float* mask, uint32_t n, float* g, float* loss2) {
    __shared__ float s_part[32];
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (int i = threadIdx.x; i < kNParams; i += 1024) g[i] = 0.0f;
    float c = 0.0f;
#pragma unroll 8
    for (uint32_t i = threadIdx.x; i < n; i += 1024) c += mask[i] != 0.0f ? 1.0f : 0.0f;
    c = warp_sum(c);
    if (lane() == 0) s_part[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x < 32) {
        c = warp_sum(s_part[threadIdx.x]);
        if (threadIdx.x == 0) {
            loss2[0] = 0.0f;
            loss2[1] = c;
        }
    }
}

// the same count for larger batches, after memsets of g and the loss
__global__ void mask_sum_kernel(const float* mask, uint64_t n, float* out) {
    float s = 0;
    for (uint64_t i = blockIdx.x * uint64_t(blockDim.x) + threadIdx.x; i < n; i += uint64_t(gridDim.x) * blockDim.x)
        s += mask[i] != 0.0f ? 1.0f : 0.0f;
    s = warp_sum(s);
    if (lane() == 0) atomicAdd(out, s);
}

// Gradient of L = sum(mask * (y - t)^2) / sum(mask).
//
// FP32 FMA and shared-memory bound: 6 x 5,312 flops per sample against 88
// bytes read. A CTA takes tiles of 64 samples; thread (tx, ty) owns a 4 x 4
// block of every 64 x 64 product (forward, dH1, dW2), its operands read from
// shared memory as 16-byte vectors (three wavefronts per 16 FMAs), and keeps
// its share of the parameter gradient in registers over all its tiles. The
// three outputs of a sample are summed over the 16 threads of its row by a
// shuffle reduction that leaves one (sample, output) pair per thread.
// Gradients are accumulated without the 1 / sum(mask) factor, so everything
// up to the final adds runs before the wait on the kernel that zeroes g and
// counts the mask. (That kernel lets this one start only after its own wait,
// so the parameters and the batch are there.)
// One sample per 64-thread CTA at a time, with every weight read through L1
// and 5,443 atomics from each of 1,184 CTAs, took 247.8 us for 8,192 samples;
// here a whole step (this kernel with its 128 tiles on 148 SMs, the launch before
// it and Adam, each launched early) takes 18.3 us instead of 256.
constexpr int kTS = 64;        // samples per tile
constexpr int kLd = H + 4;     // row stride: the two rows a warp reads start 16 banks apart
constexpr int kLdX = F + 4;
constexpr int kGradThreads = 256;
struct GradSmem {
    float w1t[F][H];           // W1 transposed: [input][unit]
    float w2t[H][kLd];         // W2 transposed: [unit of layer 1][unit of layer 2]
    float w2[H][kLd];
    float w3[O][H];
    float b1[H], b2[H];
    float h1[kTS][kLd];        // per sample: layer 1 after ReLU
    float d2[kTS][kLd];        // dL/d(layer 2 before ReLU)
    float d1[kTS][kLd];        // dL/d(layer 1 before ReLU)
    float x[kTS][kLdX];
    float red[kGradThreads / 32][O * H + 2 * H + 8];
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

// acc[r][c] += sum over k of A[s0 + r][k] * B[k][c0 + c]
template <int K, int LA, int LB>
__device__ __forceinline__ void mac_tile(const float (*A)[LA], const float (*B)[LB], int s0, int c0,
                                         float (&acc)[4][4]) {
#pragma unroll 4
    for (int k = 0; k < K; k += 4) {
        float4 a[4], b[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) a[r] = ld4(&A[s0 + r][k]);
#pragma unroll
        for (int e = 0; e < 4; ++e) b[e] = ld4(&B[k + e][c0]);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const float av[4] = {a[r].x, a[r].y, a[r].z, a[r].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                acc[r][0] = fmaf(av[e], b[e].x, acc[r][0]);
                acc[r][1] = fmaf(av[e], b[e].y, acc[r][1]);
                acc[r][2] = fmaf(av[e], b[e].z, acc[r][2]);
                acc[r][3] = fmaf(av[e], b[e].w, acc[r][3]);
            }
        }
    }
}

__global__ void __launch_bounds__(kGradThreads, 1) mlp_grad_kernel(const float* __restrict__ p,
                                                                   const float* __restrict__ x,
                                                                   const float* __restrict__ t,
                                                                   const float* __restrict__ mask, uint32_t n,
                                                                   float* g, float* loss2) {
    extern __shared__ __align__(16) unsigned char g_smem[];
    GradSmem& sm = *reinterpret_cast<GradSmem*>(g_smem);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, wp = tid >> 5;
    const int c0 = tx * 4, s0 = ty * 4;  // this thread's units and samples
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    for (int i = tid; i < H * F; i += kGradThreads) sm.w1t[i % F][i / F] = p[kW1 + i];
    for (int i = tid; i < H * H; i += kGradThreads) {
        const float v = p[kW2 + i];
        sm.w2[i / H][i % H] = v;
        sm.w2t[i % H][i / H] = v;
    }
    for (int i = tid; i < O * H; i += kGradThreads) sm.w3[i / H][i % H] = p[kW3 + i];
    if (tid < H) {
        sm.b1[tid] = p[kB1 + tid];
        sm.b2[tid] = p[kB2 + tid];
    }
    const int ro = tx & 3, rs = tx >> 2;  // the (sample s0 + rs, output ro) this thread sums up; ro 3: none
    const float b3 = ro < O ? p[kB3 + ro] : 0.0f;
    float gw1[4] = {}, gw2[4][4] = {}, gw3[O][4] = {}, gb1[4] = {}, gb2[4] = {}, gb3 = 0.0f, lsum = 0.0f;
    const uint32_t tiles = (n + kTS - 1) / kTS;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint64_t base = uint64_t(tile) * kTS;
        const uint32_t rows = n - base < uint64_t(kTS) ? uint32_t(n - base) : uint32_t(kTS);
        for (int i = tid; i < kTS * F; i += kGradThreads)
            sm.x[i / F][i % F] = uint32_t(i / F) < rows ? x[base * F + i] : 0.0f;
        __syncthreads();
        float h2[4][4], a[4][4];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int r = 0; r < 4; ++r) a[r][c] = sm.b1[c0 + c];
        mac_tile<F>(sm.x, sm.w1t, s0, c0, a);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
#pragma unroll
            for (int c = 0; c < 4; ++c) a[r][c] = fmaxf(a[r][c], 0.0f);
            st4(&sm.h1[s0 + r][c0], a[r]);
        }
        // bit 4r + c: unit c0 + c of sample s0 + r is active in layer 1
        uint32_t on1 = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) on1 |= (a[r][c] > 0.0f ? 1u : 0u) << (4 * r + c);
        __syncthreads();
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int r = 0; r < 4; ++r) h2[r][c] = sm.b2[c0 + c];
        mac_tile<H>(sm.h1, sm.w2t, s0, c0, h2);
        // outputs: partial sums over this thread's four units, v[4 * sample + output]
        float v[16];
        float w3[O][4];
#pragma unroll
        for (int o = 0; o < O; ++o) {
            const float4 w = ld4(&sm.w3[o][c0]);
            w3[o][0] = w.x; w3[o][1] = w.y; w3[o][2] = w.z; w3[o][3] = w.w;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
#pragma unroll
            for (int c = 0; c < 4; ++c) h2[r][c] = fmaxf(h2[r][c], 0.0f);
#pragma unroll
            for (int o = 0; o < 4; ++o) {
                float q = 0.0f;
                if (o < O) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) q = fmaf(w3[o][c], h2[r][c], q);
                }
                v[4 * r + o] = q;
            }
        }
        // 16 values over 16 threads: each step halves the values a thread
        // keeps; thread tx ends with the total of v[tx]
#pragma unroll
        for (int h = 8; h > 0; h >>= 1) {
            const bool up = tx & h;
#pragma unroll
            for (int i = 0; i < h; ++i) {
                const float mine = up ? v[i + h] : v[i], other = up ? v[i] : v[i + h];
                v[i] = mine + __shfl_xor_sync(0xffffffffu, other, h);
            }
        }
        float dy = 0.0f;
        if (ro < O && uint32_t(s0 + rs) < rows) {
            const uint64_t i = (base + s0 + rs) * O + ro;
            const float r = (mask[i] != 0.0f ? 1.0f : 0.0f) * (v[0] + b3 - t[i]);
            dy = 2.0f * r;
            lsum = fmaf(r, r, lsum);
            gb3 += dy;
        }
        // layer 3: dW3[o][c] = sum_s dy[s][o] h2[s][c]; d2 = relu'(h2) sum_o dy[s][o] W3[o][c]
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float d[4] = {};
#pragma unroll
            for (int o = 0; o < O; ++o) {
                const float e = __shfl_sync(0xffffffffu, dy, (tid & 16) + 4 * r + o);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    gw3[o][c] = fmaf(e, h2[r][c], gw3[o][c]);
                    d[c] = fmaf(e, w3[o][c], d[c]);
                }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                d[c] = h2[r][c] > 0.0f ? d[c] : 0.0f;
                gb2[c] += d[c];
            }
            st4(&sm.d2[s0 + r][c0], d);
        }
        __syncthreads();
        // layer 2: dW2[i][j] = sum_s d2[s][i] h1[s][j] (i = s0.., j = c0..);
        // d1 = relu'(h1) sum_i d2[s][i] W2[i][j]
#pragma unroll 8
        for (int s = 0; s < kTS; ++s) {
            const float4 e = ld4(&sm.d2[s][s0]), f = ld4(&sm.h1[s][c0]);
            const float ev[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                gw2[r][0] = fmaf(ev[r], f.x, gw2[r][0]);
                gw2[r][1] = fmaf(ev[r], f.y, gw2[r][1]);
                gw2[r][2] = fmaf(ev[r], f.z, gw2[r][2]);
                gw2[r][3] = fmaf(ev[r], f.w, gw2[r][3]);
            }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c) a[r][c] = 0.0f;
        mac_tile<H>(sm.d2, sm.w2, s0, c0, a);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                a[r][c] = on1 >> (4 * r + c) & 1u ? a[r][c] : 0.0f;
                gb1[c] += a[r][c];
            }
            st4(&sm.d1[s0 + r][c0], a[r]);
        }
        __syncthreads();
        // layer 1: dW1[j][k] = sum_s d1[s][j] x[s][k]; thread: unit tid / 4, inputs 4 (tid % 4) ..
#pragma unroll 8
        for (int s = 0; s < kTS; ++s) {
            const float d = sm.d1[s][tid >> 2];
            const float4 xv = ld4(&sm.x[s][4 * (tid & 3)]);
            gw1[0] = fmaf(d, xv.x, gw1[0]);
            gw1[1] = fmaf(d, xv.y, gw1[1]);
            gw1[2] = fmaf(d, xv.z, gw1[2]);
            gw1[3] = fmaf(d, xv.w, gw1[3]);
        }
        __syncthreads();
    }
    // sums over the CTA of what several threads hold: the two sample rows of
    // a warp by a shuffle, the warps through shared memory
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int o = 0; o < O; ++o) gw3[o][c] += __shfl_xor_sync(0xffffffffu, gw3[o][c], 16);
        gb1[c] += __shfl_xor_sync(0xffffffffu, gb1[c], 16);
        gb2[c] += __shfl_xor_sync(0xffffffffu, gb2[c], 16);
    }
    lsum = warp_sum(lsum);
#pragma unroll
    for (int h = 4; h <= 16; h <<= 1) gb3 += __shfl_xor_sync(0xffffffffu, gb3, h);  // over the lanes of output ro
    float* red = sm.red[wp];
    if ((tid & 16) == 0) {
#pragma unroll
        for (int o = 0; o < O; ++o) st4(red + o * H + c0, gw3[o]);
        st4(red + O * H + c0, gb1);
        st4(red + O * H + H + c0, gb2);
    }
    if ((tid & 31) < 4) red[O * H + 2 * H + (tid & 3)] = gb3;  // entry 3 is not used
    if ((tid & 31) == 0) red[O * H + 2 * H + 4] = lsum;
    __syncthreads();
    // g is zeroed and the mask counted by the launches before this one
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float inv = 1.0f / fmaxf(*reinterpret_cast<volatile float*>(loss2 + 1), 1.0f);
    const bool v4 = (reinterpret_cast<uintptr_t>(g) & 15u) == 0;
    auto add4 = [&](float* dst, const float (&e)[4]) {
        if (v4) {
            atomicAdd(reinterpret_cast<float4*>(dst), make_float4(e[0] * inv, e[1] * inv, e[2] * inv, e[3] * inv));
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) atomicAdd(dst + c, e[c] * inv);
        }
    };
#pragma unroll
    for (int r = 0; r < 4; ++r) add4(g + kW2 + (s0 + r) * H + c0, gw2[r]);
    add4(g + kW1 + 4 * tid, gw1);
    for (int i = tid; i < O * H + 2 * H + 5; i += kGradThreads) {
        float e = 0.0f;
#pragma unroll
        for (int k = 0; k < kGradThreads / 32; ++k) e += sm.red[k][i];
        float* dst = i < O * H             ? g + kW3 + i
                     : i < O * H + H       ? g + kB1 + (i - O * H)
                     : i < O * H + 2 * H   ? g + kB2 + (i - O * H - H)
                     : i < O * H + 2 * H + O ? g + kB3 + (i - O * H - 2 * H)
                     : i == O * H + 2 * H + 4 ? loss2
                                              : nullptr;
        if (dst) atomicAdd(dst, e * inv);
    }
}

__global__ void adam_kernel(float* p, const float* g, float* m, float* v, float lr, float b1, float b2, float eps,
                            float c1, float c2) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int i = kW1 + blockIdx.x * blockDim.x + threadIdx.x; i < kNParams; i += gridDim.x * blockDim.x) {
        const float gi = g[i];
        const float mi = b1 * m[i] + (1.0f - b1) * gi;
        const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
        m[i] = mi;
        v[i] = vi;
        p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    }
}

int grid_of(uint32_t n, uint32_t cap) { return int(n < cap ? (n ? n : 1) : cap); }

}  // namespace

cudaError_t launch_planner(const IndexView& v, const float* params, const uint32_t* terms, const uint64_t* q_off,
                           uint32_t n_q, uint32_t hybrid_min, uint64_t n_postings, float* feat, float* pred,
                           uint8_t* paths, cudaStream_t s) {
    if (n_q == 0) return cudaSuccess;
    FeatCtx c{hybrid_min, n_postings, n_q};
    planner_kernel<<<grid_of(n_q, 65535u * 4u), kFeatThreads, 0, s>>>(v, params, terms, q_off, c, feat, pred, paths);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mlp_forward(const float* p, const float* x, uint32_t n, float* y, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    mlp_forward_kernel<<<grid_of(n, 148u * 16u), 64, 0, s>>>(p, x, n, y);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_mlp_grad(const float* p, const float* x, const float* t, const float* mask, uint32_t n, float* g,
                            float* loss2, cudaStream_t s) {
    static std::atomic<uint64_t> done{0};  // devices whose attribute is set
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && !(done.load() >> (dev & 63) & 1ull)) {
        e = cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(sizeof(GradSmem)));
        if (e == cudaSuccess) done.fetch_or(1ull << (dev & 63));
    }
    if (e != cudaSuccess) return e;
    if (n == 0 || n > kInitSamples) {
        e = cudaMemsetAsync(g, 0, sizeof(float) * kNParams, s);
        if (e == cudaSuccess) e = cudaMemsetAsync(loss2, 0, 2 * sizeof(float), s);
        if (e != cudaSuccess || n == 0) return e;
        mask_sum_kernel<<<grid_of(uint32_t((uint64_t(n) * O + 255) / 256), 256u), 256, 0, s>>>(mask, uint64_t(n) * O,
                                                                                                loss2 + 1);
    } else {
        e = launch_after(grad_init_kernel, 1, 1024, 0, s, mask, n * O, g, loss2);
        if (e != cudaSuccess) return e;
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    count_launch(2);
    return launch_after(mlp_grad_kernel, uint32_t(grid_of((n + kTS - 1) / kTS, 148u)), kGradThreads, sizeof(GradSmem), s,
                        p, x, t, mask, n, g, loss2);
}

cudaError_t launch_adam(float* p, const float* g, float* m, float* v, uint32_t step, float lr, float b1, float b2,
                        float eps, cudaStream_t s) {
    const float c1 = 1.0f - std::pow(b1, float(step ? step : 1));
    const float c2 = 1.0f - std::pow(b2, float(step ? step : 1));
    count_launch();
    return launch_after(adam_kernel, (kNParams + 255) / 256, 256, 0, s, p, g, m, v, lr, b1, b2, eps, c1, c2);
}

}  // namespace abf
