// Kernels of libadabool for sm_100a. See abf_kernels.cuh for the overview
// and abf_internal.h for the list format they decode.
//
// Reference counterparts (yxr620/AdaBool):
//   scatter_kernel / tile_union_kernel  <- ListUnionKernel{1,,Bitset} and
//       SparseBatchListUnionKernel{1,,Bitset}
//       (src/AdaBool/load_balance_transformer.cu.h:16-91,138-220) with the
//       container decoders (src/AdaBool/inverted_list.cu.h:61-130)
//   probe_kernel  <- KeyBPTransformKernel{1,,Bitset} and
//       KeyBatchBPTransformKernel_Expanded{1,,Bitset}
//       (src/AdaBool/key_transformer.cu.h:11-331,
//        src/AdaBool/key_batch_transformer.cu.h:11-524)
//   count/scan/write  <- the host loop CollectIdsFromBitmap
//       (test/adsfilter_batch.cu:82-97)
#include "abf_kernels.cuh"
#include "abf_planner_dev.cuh"

#include <cuda.h>
#include <cstring>

#include <algorithm>
#include <atomic>

namespace abf {

namespace {

constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kProbeSmemWords = 8192;  // staged term-bitmap words per CTA
// look-back status word: flag in the top two bits, count below
constexpr uint64_t kFlagAgg = 1ull << 62;   // the item's own id count is known
constexpr uint64_t kFlagIncl = 2ull << 62;  // the ids of the item and all before it
constexpr uint64_t kValMask = (1ull << 62) - 1;

// Programmatic launch order: the kernels of a batch are launched so that each
// may come up while the one before it finishes. Every kernel begins with this
// wait, before it reads or writes any global memory, and on every CTA (a
// kernel is complete only when the ones before it are). What the kernel before
// it, or the caller, writes is read by plain loads: __ldg promises data that
// nobody writes while this kernel runs, which it does from before the wait, and
// the compiler may move it across the wait. It is for the index's arrays, and
// for what a kernel further back wrote (complete when this one comes up).
__device__ __forceinline__ void wait_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }
__device__ __forceinline__ uint32_t warp_id() { return threadIdx.x >> 5; }

// ---------------------------------------------------------------------------
// block decode: one warp, one block of up to 128 ids
// ---------------------------------------------------------------------------
// Lane j returns the ids of positions 4j..4j+3 of the block (ascending across
// the warp); position i is valid when i < cnt. The payload is staged in the
// warp's 512-byte shared buffer with one 16-byte load per lane; each lane
// extracts its four gaps with a funnel shift, sums them, and a shuffle scan
// over the lanes turns the gaps into ids.
// A block's descriptor and this lane's 16 bytes of its payload, loaded
// ahead of the decode so the loads of the next block overlap the work on
// the current one.
struct Fetched {
    uint4 pay;
    uint32_t first, meta;
};

__device__ __forceinline__ Fetched fetch_block(const IndexView& ix, uint32_t b) {
    Fetched r;
    const uint2 d = __ldg(ix.blk_desc + b);
    r.first = __ldg(ix.blk_first + b);
    r.meta = d.y;
    const uint32_t bits = d.y & 63u, cnt = (d.y >> 8) + 1u;
    const uint32_t units = ((cnt - 1u) * bits + 127u) >> 7;
    r.pay = lane_id() < units ? __ldg(ix.payload + d.x + lane_id()) : make_uint4(0u, 0u, 0u, 0u);
    return r;
}

__device__ __forceinline__ void decode_fetched(const Fetched& fb, uint4* stage, uint32_t (&id)[4], uint32_t& cnt) {
    const uint32_t lane = lane_id();
    const uint32_t first = fb.first;
    const uint32_t bits = fb.meta & 63u;
    cnt = (fb.meta >> 8) + 1u;
    __syncwarp();
    stage[lane] = fb.pay;
    __syncwarp();
    const uint32_t* w = reinterpret_cast<const uint32_t*>(stage);
    const uint32_t mask = bits >= 32u ? kFull : ((1u << bits) - 1u);
    uint32_t p[4];
    uint32_t run = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t i = lane * 4u + k;
        uint32_t g = 0;
        if (i >= 1u && i < cnt) {
            uint32_t v = 0;
            if (bits) {
                const uint32_t pos = (i - 1u) * bits;
                const uint32_t wi = pos >> 5;
                v = __funnelshift_r(w[wi], w[wi + 1], pos & 31u) & mask;
            }
            g = v + 1u;
        }
        run += g;
        p[k] = run;
    }
    uint32_t incl = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane >= uint32_t(o)) incl += y;
    }
    const uint32_t base = first + (incl - run);
#pragma unroll
    for (int k = 0; k < 4; ++k) id[k] = base + p[k];
}

// OR the decoded ids that fall in [lo, lo + span) into a shared-memory tile.
// A lane's ids are ascending, so runs in one word are combined before the
// atomic.
__device__ __forceinline__ void or_tile(uint32_t* tile, uint32_t lo, uint32_t span, const uint32_t (&id)[4],
                                        uint32_t cnt) {
    const uint32_t lane = lane_id();
    uint32_t cur = kFull, m = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t i = lane * 4u + k;
        const uint32_t rel = id[k] - lo;
        if (i < cnt && rel < span) {
            const uint32_t wd = rel >> 5, bit = 1u << (rel & 31u);
            if (wd != cur) {
                if (cur != kFull) atomicOr(tile + cur, m);
                cur = wd;
                m = bit;
            } else {
                m |= bit;
            }
        }
    }
    if (cur != kFull) atomicOr(tile + cur, m);
}

// OR of this lane's four ids (those below n_ads) into the bitmap, one atomic
// per distinct word
__device__ __forceinline__ void or_global(uint32_t* bm, uint32_t n_ads, const uint32_t (&id)[4], uint32_t cnt) {
    const uint32_t lane = lane_id();
    uint32_t cur = kFull, m = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t i = lane * 4u + k;
        if (i < cnt && id[k] < n_ads) {
            const uint32_t wd = id[k] >> 5, bit = 1u << (id[k] & 31u);
            if (wd != cur) {
                if (cur != kFull) atomicOr(bm + cur, m);
                cur = wd;
                m = bit;
            } else {
                m |= bit;
            }
        }
    }
    if (cur != kFull) atomicOr(bm + cur, m);
}

template <int NT>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* s_warp, uint32_t* total) {
    constexpr int NWARP = NT / 32;
    const uint32_t lane = lane_id(), warp = warp_id();
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= uint32_t(o)) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < uint32_t(NWARP) ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, w, o);
            if (lane >= uint32_t(o)) w += y;
        }
        if (lane < uint32_t(NWARP)) s_warp[lane] = w;
    }
    __syncthreads();
    const uint32_t wex = warp ? s_warp[warp - 1] : 0u;
    *total = s_warp[NWARP - 1];
    __syncthreads();
    return wex + x - v;
}

// exclusive scan of 64-bit values over the CTA (s: NT / 32 entries)
template <int NT>
__device__ __forceinline__ uint64_t block_excl_scan64(uint64_t v, unsigned long long* s, uint64_t* total) {
    const uint32_t lane = lane_id(), warp = warp_id();
    uint64_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= uint32_t(o)) x += y;
    }
    if (lane == 31) s[warp] = x;
    __syncthreads();
    uint64_t before = 0, all = 0;
#pragma unroll
    for (uint32_t i = 0; i < uint32_t(NT / 32); ++i) {
        const uint64_t y = s[i];
        if (i < warp) before += y;
        all += y;
    }
    __syncthreads();
    *total = all;
    return before + x - v;
}

template <int NT>
__device__ __forceinline__ uint64_t block_sum_u64(uint64_t v, unsigned long long* s) {
    const uint32_t lane = lane_id(), warp = warp_id();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(kFull, v, o);
    if (lane == 0) s[warp] = v;
    __syncthreads();
    uint64_t t = 0;
    for (int i = 0; i < NT / 32; ++i) t += s[i];
    __syncthreads();
    return t;
}

// first index in [a, b) with arr[index] >= key (arr ascending)
__device__ __forceinline__ uint32_t lower_bound_g(const uint32_t* arr, uint32_t a, uint32_t b, uint32_t key) {
    while (a < b) {
        const uint32_t m = (a + b) >> 1;
        if (__ldg(arr + m) < key) a = m + 1; else b = m;
    }
    return a;
}

// ---------------------------------------------------------------------------
// mbarrier + bulk async copy (TMA engine, 1-D form)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_addr(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_addr(dst)),
        "l"(src), "r"(bytes), "r"(smem_addr(bar))
        : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Waits for the phase of `bar` with the given parity; false after `limit`
// polls without it completing.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, uint32_t limit) {
    for (uint32_t spins = 0; !mbar_try_wait(bar, parity);)
        if (++spins > limit) return false;
    return true;
}

// async 4- and 16-byte copies global -> shared (LDGSTS: no register round trip)
__device__ __forceinline__ void cp_async4(void* sdst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(sdst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(sdst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// ---------------------------------------------------------------------------
// planning
// ---------------------------------------------------------------------------
// Exclusive scan of the queries' scattered block counts and, where the bin
// kernel runs, its work split; by one CTA. The counts may come from other CTAs
// of the same kernel: they are read past L1.
template <int NT>
__device__ __forceinline__ void queue_scan_body(const QueueArgs& a, uint32_t n_q, unsigned long long* s64,
                                                uint32_t* s32) {
    const uint32_t tid = threadIdx.x;
    uint64_t carry = 0, sum = 0;
    for (uint32_t c0 = 0; c0 < n_q; c0 += NT) {
        const uint32_t i = c0 + tid;
        const uint64_t v = i < n_q ? __ldcg(a.q_light_cnt + i) : 0ull;
        if (a.q_bblk && i < n_q) sum += __ldcg(a.q_bblk + i);
        uint64_t tot;
        const uint64_t ex = block_excl_scan64<NT>(v, s64, &tot);
        if (i < n_q) a.q_light_pref[i] = carry + ex;
        carry += tot;
    }
    if (tid == 0) a.q_light_pref[n_q] = carry;
    if (!a.q_bblk) return;
    // The bin kernel's items: every tile x every part of every query. A query
    // is cut into parts by its lists so that no item has much more than half
    // an even share of the work (or 64 blocks).
    sum = block_sum_u64<NT>(sum, s64);
    const uint64_t lim64 = max(64ull, static_cast<unsigned long long>(sum) / (2ull * a.slots)) * a.n_tiles;
    const uint32_t lim = lim64 < 0xffffffffull ? uint32_t(lim64) : kFull;
    uint32_t pc = 0;
    for (uint32_t c0 = 0; c0 < n_q; c0 += NT) {
        const uint32_t i = c0 + tid;
        uint32_t parts = 0;
        if (i < n_q) {
            const uint32_t nb = __ldcg(a.q_bblk + i);
            if (nb) parts = min((nb - 1u) / lim + 1u, __ldcg(a.q_nbin + i));
        }
        uint32_t tot;
        const uint32_t ex = block_excl_scan<NT>(parts, s32, &tot);
        if (i < n_q) a.parts_pref[i] = pc + ex;
        pc += tot;
    }
    if (tid == 0) {
        a.parts_pref[n_q] = pc;
        *a.ticket = 0;
    }
}

// No work for any query of a batch whose term slots overlap; after the scan.
__device__ __forceinline__ void drop_batch(const QueueArgs& a, uint32_t n_q) {
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n_q; i += blockDim.x) a.q_ndense[i] = 0u;
    if (threadIdx.x == 0) {
        a.q_light_pref[n_q] = 0ull;
        if (a.q_bblk) a.parts_pref[n_q] = 0u;
        *a.n_tile_list = 0u;
    }
}

// A CTA per query at a time, four terms per thread and step (one 16-byte load
// of a term's table entry each): a step's latency, not its work, is what the
// longest queries' CTAs wait for, and they end last (one term per step from
// four tables: 62 us for 512 queries of c1, 245 for 2,048 of c2; here 26 and
// 119 with the scan). The CTA that finishes
// last runs the scan over the queries (batches of up to kScanInPlan), which
// saves that launch.
constexpr uint32_t kPlanTerms = 4;
// added to the count of finished CTAs by a query whose followers overlap
// earlier ones (no load of a word of its own: it cost the scan 1.5 us)
constexpr uint32_t kOverlap = 1u << 16;
static_assert(kScanInPlan < kOverlap, "the count stays below it");
template <uint32_t kInline>
__global__ void __launch_bounds__(256, 4) plan_kernel(IndexView ix, PlanArgs a,
                                                      const __grid_constant__ InlineTerms<kInline> given) {
    __shared__ uint32_t s_warp[32];
    __shared__ unsigned long long s_red[8];
    __shared__ uint32_t s_path, s_max, s_slot, s_nbin;
    __shared__ uint32_t s_mask[2048];  // the query's dense bitmaps (n_dense <= 65535)
    __shared__ plan_dev::PlannerSmem s_pl;
    static_assert(plan_dev::kFeatThreads == 256, "the planner code runs with the plan kernel's 256 threads");
    const uint32_t tid = threadIdx.x;
    constexpr uint32_t kStep = 256u * kPlanTerms;
    if (a.planner) plan_dev::load_params(a.planner, s_pl);  // not written by any kernel of a batch
    wait_previous();
    if constexpr (kInline > 0) {
        uint32_t* terms = const_cast<uint32_t*>(a.terms);
        for (uint32_t i = tid; i < given.n; i += 256) terms[i] = given.t[i];
        if (tid < 2) const_cast<uint64_t*>(a.q_off)[tid] = tid ? given.n : 0u;
        for (uint32_t i = tid; i < a.ctl_words; i += 256) a.ctl[i] = 0u;
        __syncthreads();
    }
    const uint32_t n_q = a.d_n_q ? min(*a.d_n_q, a.n_q) : a.n_q;
    for (uint32_t q = blockIdx.x; q < n_q; q += gridDim.x) {
        uint64_t qb = a.q_off[q], qe = a.q_off[q + 1];
        if (qe < qb || qe > a.max_terms) {
            // offsets outside the scratch arrays: the query gets no work
            if (tid == 0 && a.err) atomicOr(a.err, kErrTermRange);
            if constexpr (kInline == 0) {
                if (tid == 0 && qe < qb && q + 1u < n_q) {
                    if (a.done) atomicAdd(a.done, kOverlap);
                    else if (a.overlap) *a.overlap = 1u;
                }
            }
            qe = qb = 0;
        }
        // what the later kernels find zeroed: the query's saturation marks,
        // its chunks' look-back words and its id count
        if (a.sat)
            for (uint32_t i = tid; i < a.sat_stride; i += 256) a.sat[uint64_t(q) * a.sat_stride + i] = 0u;
        if (a.status)
            for (uint32_t i = tid; i < a.n_chunks; i += 256) a.status[uint64_t(q) * a.n_chunks + i] = 0ull;
        if (a.id_counts && tid == 0) a.id_counts[q] = 0ull;
        // table entries of this thread's terms of the step at c0: {first
        // block, postings, dense bitmap, plain list}; no postings: skip it
        auto load_step = [&](uint64_t c0, uint4 (&e)[kPlanTerms]) {
            uint32_t t[kPlanTerms];
#pragma unroll
            for (uint32_t k = 0; k < kPlanTerms; ++k) {
                const uint64_t i = c0 + tid * kPlanTerms + k;
                t[k] = i < qe ? a.terms[i] : kNone;
            }
#pragma unroll
            for (uint32_t k = 0; k < kPlanTerms; ++k)
                e[k] = t[k] < ix.n_terms ? __ldg(ix.term_info + t[k]) : make_uint4(0u, 0u, kNone, kNone);
        };
        auto blocks_of = [](uint32_t len) { return (len + ABF_BLOCK_POSTINGS - 1u) / ABF_BLOCK_POSTINGS; };
        uint32_t path = a.paths ? a.paths[q] : a.path_uniform;
        const bool planned = path == ABF_PATH_AUTO && a.planner;
        if (planned) {
            // learned planner: features + MLP of this query, inline
            path = plan_dev::planner_path(ix, a.terms, qb, qe, q, plan_dev::FeatCtx{a.hybrid_min, a.n_postings, a.n_q},
                                          s_pl);
        } else if (path == ABF_PATH_AUTO) {
            // fixed rule: probe when the query's lists cover more than
            // probe_min_frac of all blocks; else HYBRID when one of its lists
            // has at least fixed_hybrid_min postings; else list-union
            uint64_t nb = 0;
            uint32_t mx = 0;
            for (uint64_t c0 = qb; c0 < qe; c0 += kStep) {
                uint4 e[kPlanTerms];
                load_step(c0, e);
#pragma unroll
                for (uint32_t k = 0; k < kPlanTerms; ++k) {
                    nb += blocks_of(e[k].y);
                    mx = max(mx, e[k].y);
                }
            }
            if (tid == 0) s_max = 0;
            nb = block_sum_u64<256>(nb, s_red);  // its barriers also order the s_max reset
            mx = __reduce_max_sync(kFull, mx);
            if (lane_id() == 0 && mx) atomicMax(&s_max, mx);
            __syncthreads();
            mx = s_max;
            path = (double(nb) > double(a.probe_min_frac) * double(ix.n_blocks)) ? ABF_PATH_PROBE
                   : (a.fixed_hybrid_min && mx >= a.fixed_hybrid_min) ? ABF_PATH_HYBRID
                                                                      : ABF_PATH_UNION;
        }
        if (tid == 0) {
            s_slot = kNone;
            if (path == ABF_PATH_PROBE) {
                const uint32_t slot = atomicAdd(a.n_probe, 1u);
                if (slot < a.probe_cap) {
                    a.probe_list[slot] = q;
                    s_slot = slot;
                } else {
                    path = ABF_PATH_UNION;  // no probe slot left: same result by list-union
                }
            }
            s_path = path;
            s_nbin = 0;
        }
        const bool merge_d = a.dense_in_tile && !(a.no_dense_from && q >= a.no_dense_from);
        const bool want_d = a.q_dense16 != nullptr && merge_d;
        const uint32_t mw = (ix.n_dense + 31u) / 32u;
        if (want_d)
            for (uint32_t i = tid; i < mw; i += 256) s_mask[i] = 0u;
        __syncthreads();
        path = s_path;
        const bool probe = path == ABF_PATH_PROBE;
        if (probe && a.probe_bm) {
            // the probe slot's term bitmap: zeroed, then this query's terms
            uint32_t* bm = a.probe_bm + uint64_t(s_slot) * a.probe_stride;
            for (uint64_t w = tid; w < a.probe_stride; w += 256) bm[w] = 0u;
            __syncthreads();
            for (uint64_t i = qb + tid; i < qe; i += 256) {
                const uint32_t t = a.terms[i];
                if (t < ix.n_terms) atomicOr(bm + (t >> 5), 1u << (t & 31u));
            }
        }
        // merge threshold: TILE merges every list, HYBRID the long ones,
        // UNION only those with a dense bitmap, PROBE none
        const uint32_t hm = path == ABF_PATH_TILE ? 0u
                            : path == ABF_PATH_HYBRID ? a.hybrid_min
                            : probe ? kNoHeavy : kDenseOnly;
        // shortest plain list that the bin kernel takes: any, where the query
        // holds enough of them; else those that the path merges
        uint32_t bin_from = kNone;
        if (a.bin_list) {
            uint64_t nb = 0, nh = 0;  // blocks of the plain lists, and of those the path merges
            if (planned) {  // added up with the features
                nb = s_pl.blocks[0];
                nh = path == ABF_PATH_HYBRID ? s_pl.blocks[1] : 0u;
            } else {
                for (uint64_t c0 = qb; c0 < qe; c0 += kStep) {
                    uint4 e[kPlanTerms];
                    load_step(c0, e);
#pragma unroll
                    for (uint32_t k = 0; k < kPlanTerms; ++k)
                        if (e[k].w != kNone) {
                            nb += blocks_of(e[k].y);
                            if (e[k].y >= hm) nh += blocks_of(e[k].y);
                        }
                }
                nb = block_sum_u64<256>(nb, s_red);
                nh = block_sum_u64<256>(nh, s_red);
            }
            if (probe || (a.mixed_from && q >= *a.mixed_from)) nb = nh = 0;
            if (nb < 0xffffffffull) {
                if (nb >= a.bin_min_blocks) bin_from = 0;
                else if (nh) bin_from = hm;
            }
            if (tid == 0) a.q_bblk[q] = bin_from == kNone ? 0u : uint32_t(bin_from ? nh : nb);
        }
        uint32_t carry = 0, nmerge = 0;
        for (uint64_t c0 = qb; c0 < qe; c0 += kStep) {
            uint4 e[kPlanTerms];
            load_step(c0, e);
            uint32_t cnt[kPlanTerms], sum = 0;
#pragma unroll
            for (uint32_t k = 0; k < kPlanTerms; ++k) {
                const uint64_t i = c0 + tid * kPlanTerms + k;
                const uint32_t d = merge_d ? e[k].z : kNone;
                uint32_t cls = kNone;
                cnt[k] = 0;
                if (i < qe && !probe && e[k].y) {
                    if (d != kNone) {
                        if (want_d) atomicOr(&s_mask[d >> 5], 1u << (d & 31u));
                    } else if (e[k].w != kNone && e[k].y >= bin_from) {
                        a.bin_list[qb + atomicAdd(&s_nbin, 1u)] = e[k].w;
                    } else if (e[k].y >= hm) {
                        cls = a.terms[i];
                        ++nmerge;
                    } else {
                        cnt[k] = blocks_of(e[k].y);
                    }
                }
                if (i < qe && a.tile_cls) a.tile_cls[i] = cls;
                sum += cnt[k];
            }
            uint32_t tot;
            uint32_t ex = carry + block_excl_scan<256>(sum, s_warp, &tot);
#pragma unroll
            for (uint32_t k = 0; k < kPlanTerms; ++k) {
                const uint64_t i = c0 + tid * kPlanTerms + k;
                if (i < qe) a.term_slot[i] = make_uint2(ex, e[k].x);
                ex += cnt[k];
            }
            carry += tot;
        }
        if (want_d) {
            // the query's distinct dense bitmaps in ascending order: each
            // thread expands a contiguous run of mask words at its prefix
            const uint32_t any_merge = __syncthreads_or(nmerge);
            const uint32_t per = (mw + 255u) / 256u;
            const uint32_t w0 = tid * per < mw ? tid * per : mw;
            const uint32_t w1 = w0 + per < mw ? w0 + per : mw;
            uint32_t c = 0;
            for (uint32_t w = w0; w < w1; ++w) c += __popc(s_mask[w]);
            uint32_t nd;
            uint32_t o = block_excl_scan<256>(c, s_warp, &nd);
            const uint32_t start = uint32_t((qb + 8ull * q + 7ull) & ~7ull);
            uint16_t* dst = a.q_dense16 + start;
            for (uint32_t w = w0; w < w1; ++w) {
                uint32_t m = s_mask[w];
                while (m) {
                    dst[o++] = uint16_t((w * 32u + uint32_t(__ffs(m)) - 1u) << a.dense_shift);
                    m &= m - 1u;
                }
            }
            for (uint32_t i = nd + tid; i < ((nd + 7u) & ~7u); i += 256) dst[i] = uint16_t(ix.n_dense << a.dense_shift);
            if (tid == 0) {
                a.q_dstart[q] = start;
                a.q_ndense[q] = nd;
                if (a.tile_list && any_merge) a.tile_list[atomicAdd(a.n_tile_list, 1u)] = q;
            }
        }
        if (tid == 0) {
            if (a.bin_list) a.q_nbin[q] = s_nbin;  // the scans' barriers order the last add
            a.q_light_cnt[q] = carry;
            if (a.path_out) a.path_out[q] = uint8_t(path);
        }
        __syncthreads();
    }
    if (!a.done) return;
    // A single query's CTA has nobody to wait for: without the fences and the
    // arrival a query of 40 short lists takes 22.6 us instead of 23.7.
    if (gridDim.x > 1) {
        __threadfence();  // this CTA's counts before its arrival
        __syncthreads();
        if (tid == 0) s_slot = atomicAdd(a.done, 1u);
        __syncthreads();
        if ((s_slot & (kOverlap - 1u)) != gridDim.x - 1u) return;
        __threadfence();
        if (tid == 0) *a.done = 0;  // for a next batch that does not zero it
    }
    queue_scan_body<256>(a.queue, n_q, s_red, s_warp);
    if constexpr (kInline == 0) {
        if (gridDim.x > 1 && s_slot >= kOverlap) drop_batch(a.queue, n_q);
    }
}

__global__ void __launch_bounds__(1024) queue_scan_kernel(QueueArgs a) {
    __shared__ unsigned long long s64[32];
    __shared__ uint32_t s32[32];
    wait_previous();
    const uint32_t n_q = a.d_n_q ? min(*a.d_n_q, a.n_q) : a.n_q;
    queue_scan_body<1024>(a, n_q, s64, s32);
    if (a.overlap && *a.overlap) drop_batch(a, n_q);
}

// Runs of consecutive keys with the same bitmap index, in one CTA: a flattened
// batch of queries has a run per query. (A bitmap index may come back in a
// later run: the kernels that follow OR with atomics.) Keys in no order would
// give a planning CTA a key each: 300,000 on 2^16 terms x 2^20 ads 2,669 us,
// as chunks 525.
// Merged run by run, the keys of 32 queries on 2^18 terms x 2^22 ads take 131 us; scattered key by
// key, one atomic per posting of every list, they took 1,234.
__global__ void __launch_bounds__(1024) key_runs_kernel(KeyRunsArgs a) {
    __shared__ uint32_t s_warp[32];
    const uint32_t tid = threadIdx.x;
    wait_previous();
    uint32_t carry = 0;
    for (uint64_t c0 = 0; c0 < a.n_keys; c0 += 4096) {
        uint32_t v[4], heads = 0;
        const uint64_t i0 = c0 + tid * 4u;
        uint32_t prev = i0 && i0 <= a.n_keys ? a.qidx[i0 - 1] : 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = i0 + k < a.n_keys ? a.qidx[i0 + k] : 0u;
            if (i0 + k < a.n_keys && (i0 + k == 0 || v[k] != prev)) heads |= 1u << k;
            prev = v[k];
        }
        uint32_t total;
        uint32_t r = carry + block_excl_scan<1024>(uint32_t(__popc(heads)), s_warp, &total);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (heads >> k & 1u) {
                a.off[r] = i0 + k;
                a.slot[r] = v[k];
                ++r;
            }
        }
        carry += total;
    }
    uint32_t n = carry, mixed = kNone;
    if (tid == 0) a.off[carry] = a.n_keys;
    if (carry > a.cap && carry > a.n_keys / 8u) {
        __syncthreads();  // the runs' first keys are written
        const uint64_t k0 = a.off[a.cap];
        const uint32_t chunks = uint32_t((a.n_keys - k0 + kKeyChunk - 1u) / kKeyChunk);
        __syncthreads();  // and read
        for (uint32_t c = tid; c <= chunks; c += 1024u)
            a.off[a.cap + c] = min(static_cast<unsigned long long>(k0 + uint64_t(c) * kKeyChunk), static_cast<unsigned long long>(a.n_keys));
        mixed = a.cap;
        n = a.cap + chunks;
    }
    if (tid == 0) {
        a.n_runs[0] = n;
        a.n_runs[1] = mixed;
    }
}

// ---------------------------------------------------------------------------
// term bitmaps -> term lists (bitmap-probe operators)
// ---------------------------------------------------------------------------
// A query bitmap costs n_terms / 8 bytes to read and names a few hundred or
// thousand lists; scanning the index's blocks for it reads 4 bytes of every
// block and finds the hit blocks bunched in a few warps' shares. So the
// bitmaps are turned into term lists (a CTA per query) and the list-union
// kernels, which split the named blocks evenly, do the rest: 32 queries on
// 2^18 terms x 2^22 ads 2,686 -> 142 us, on 2^20 x 2^24 6,290 -> 428 us; one
// query on 2^16 x 2^20 138 -> 47 us.
constexpr uint32_t kTermThreads = 512;
__device__ __forceinline__ uint32_t term_word(const uint32_t* bm, uint32_t w, uint32_t n_terms) {
    const uint32_t v = bm[w], left = n_terms - w * 32u;
    return left < 32u ? v & ((1u << left) - 1u) : v;
}
__device__ __forceinline__ uint32_t term_words(const TermListArgs& a) {
    const uint32_t nw = (a.n_terms + 31u) / 32u;
    return nw < a.qbm_words ? nw : a.qbm_words;
}

__global__ void __launch_bounds__(kTermThreads) term_count_kernel(TermListArgs a) {
    __shared__ unsigned long long s_red[kTermThreads / 32];
    wait_previous();
    if (blockIdx.x == 0 && threadIdx.x < a.n_zero) a.zero[threadIdx.x] = 0u;
    if (blockIdx.x == 0 && threadIdx.x == a.n_zero && a.err) *a.err = a.err_value;
    const uint32_t nw = term_words(a);
    for (uint32_t q = blockIdx.x; q < a.n_q; q += gridDim.x) {
        const uint32_t* bm = a.qbm + uint64_t(q) * a.qbm_stride;
        uint32_t c = 0;
#pragma unroll 8
        for (uint32_t w = threadIdx.x; w < nw; w += kTermThreads) c += __popc(term_word(bm, w, a.n_terms));
        const uint64_t t = block_sum_u64<int(kTermThreads)>(c, s_red);
        if (threadIdx.x == 0) a.cnt[q] = uint32_t(t);
    }
}

__global__ void __launch_bounds__(kTermThreads) term_list_kernel(TermListArgs a) {
    __shared__ unsigned long long s_red[kTermThreads / 32];
    __shared__ uint32_t s_wcnt[kTermThreads / 32];
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    constexpr uint32_t kNW = kTermThreads / 32u;
    wait_previous();
    const uint32_t nw = term_words(a);
    const uint32_t per = (nw + kNW * 32u - 1u) / (kNW * 32u) * 32u;  // words of a warp's share, whole warps' worth
    for (uint32_t q = blockIdx.x; q < a.n_q; q += gridDim.x) {
        uint64_t before = 0, all = 0;
        for (uint32_t i = tid; i < a.n_q; i += kTermThreads) {
            const uint32_t c = a.cnt[i];
            all += c;
            if (i < q) before += c;
        }
        all = block_sum_u64<int(kTermThreads)>(all, s_red);
        before = block_sum_u64<int(kTermThreads)>(before, s_red);
        const bool fits = all <= a.cap;
        if (tid == 0) {
            a.off[q] = fits ? before : 0u;
            if (q == a.n_q - 1u) a.off[a.n_q] = fits ? all : 0u;
            if (q == 0) *a.overflow = fits ? 0u : 1u;
        }
        if (!fits) continue;
        const uint32_t* bm = a.qbm + uint64_t(q) * a.qbm_stride;
        const uint32_t w0 = warp * per < nw ? warp * per : nw;
        const uint32_t w1 = w0 + per < nw ? w0 + per : nw;
        uint32_t c = 0;
#pragma unroll 4
        for (uint32_t w = w0 + lane; w < w1; w += 32u) c += __popc(term_word(bm, w, a.n_terms));
        c = __reduce_add_sync(kFull, c);
        if (lane == 0) s_wcnt[warp] = c;
        __syncthreads();
        uint32_t* dst = a.terms + before + __reduce_add_sync(kFull, lane < warp ? s_wcnt[lane] : 0u);
        for (uint32_t wb = w0; wb < w1; wb += 32u) {
            const uint32_t w = wb + lane;
            uint32_t v = w < w1 ? term_word(bm, w, a.n_terms) : 0u;
            if (!__any_sync(kFull, v != 0u)) continue;
            const uint32_t n = __popc(v);
            uint32_t x = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, x, o);
                if (lane >= uint32_t(o)) x += y;
            }
            uint32_t* d = dst + (x - n);
            for (; v; v &= v - 1u) *d++ = w * 32u + uint32_t(__ffs(v)) - 1u;
            dst += __shfl_sync(kFull, x, 31);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// list-union, merge variant
// ---------------------------------------------------------------------------
// Blocks [lo, lo + cnt) of a list that overlap the ids [lo_id, hi_id):
// three loads from the list's directory when it has one, else two binary
// searches over the block bounds. dj0/dj1 are the directory rows of lo_id
// and of the unclipped tile end.
__device__ __forceinline__ void tile_block_range(const IndexView& ix, uint32_t term, uint32_t lo_id, uint32_t hi_id,
                                                 uint32_t dj0, uint32_t dj1, uint32_t& lo, uint32_t& cnt) {
    const uint32_t b0 = __ldg(ix.term_blk + term), b1 = __ldg(ix.term_blk + term + 1);
    const uint32_t dofs = __ldg(ix.term_dir + term);
    uint32_t hi;
    if (dofs != kNone) {
        lo = __ldg(ix.dir + dofs + dj0);
        hi = __ldg(ix.dir + dofs + dj1);  // first block ending at or after the tile end
        if (hi < b1 && __ldg(ix.blk_first + hi) < hi_id) ++hi;  // it straddles the tile end
    } else {
        lo = lower_bound_g(ix.blk_last, b0, b1, lo_id);
        hi = lower_bound_g(ix.blk_first, lo, b1, hi_id);
    }
    cnt = hi > lo ? hi - lo : 0u;
}

// slot s of the chunk's prefix array with s_pref[s] <= f < s_pref[s+1]
template <int NT>
__device__ __forceinline__ uint32_t find_slot(const uint32_t* s_pref, uint32_t f) {
    uint32_t a0 = 0, a1 = NT;
    while (a1 - a0 > 1) {
        const uint32_t m = (a0 + a1) >> 1;
        if (s_pref[m] <= f) a0 = m; else a1 = m;
    }
    return a0;
}

// list-union, streamed variant of the dense merge, for batches too small for
// the dense group kernel: a thread ORs one 16-byte column of a query's dense
// bitmaps, eight rows in flight, and writes it; no shared memory, no barrier.
// Bound by HBM / L2 (every named row read; column-major item order, so the
// queries that share a row read it from L2). Rows come longest list first: a
// warp whose columns are all ones reads no more. Half-warps whose 64 words
// came out all ones mark them for the scatter kernel.
// The merge kernel did this with a quarter of its threads at 256-word tiles:
// seven queries of the serving mix on c1 135 to 186 us, one query 17 to 26.
// Four CTAs per SM leave the registers that keep all eight loads in flight: 70
// us for seven queries (398 MB of distinct rows: 5.7 TB/s), 92 with the 38
// registers the compiler takes by itself; 16 rows in flight were no faster.
// ACC: OR into the output with atomics (other calls may do so at the same
// time). V: uint4, or uint32_t where rows are not 16-byte aligned.
__device__ __forceinline__ void or_in(uint4& a, uint4 b) { a.x |= b.x; a.y |= b.y; a.z |= b.z; a.w |= b.w; }
__device__ __forceinline__ void or_in(uint32_t& a, uint32_t b) { a |= b; }
__device__ __forceinline__ bool full_vec(uint4 a) { return (a.x & a.y & a.z & a.w) == ~0u; }
__device__ __forceinline__ bool full_vec(uint32_t a) { return a == ~0u; }

constexpr uint32_t kStreamThreads = 256;
template <typename V, bool ACC>
__global__ void __launch_bounds__(kStreamThreads, 4) dense_stream_kernel(IndexView ix, DenseStreamArgs a) {
    wait_previous();
    constexpr uint32_t KT = 8, VW = sizeof(V) / 4u;
    const uint64_t n_v = (a.n_words + VW - 1u) / VW;  // columns (the last may be partial)
    const uint32_t n_cb = uint32_t((n_v + kStreamThreads - 1u) / kStreamThreads);
    const uint64_t items = uint64_t(n_cb) * a.n_q;
    const uint64_t st = ix.dense_stride / VW;
    for (uint64_t item = blockIdx.x; item < items; item += gridDim.x) {
        const uint32_t cb = uint32_t(item / a.n_q), q = uint32_t(item - uint64_t(cb) * a.n_q);
        const uint32_t nd = a.q_ndense[q];
        if (ACC && nd == 0) continue;
        const uint64_t j = uint64_t(cb) * kStreamThreads + threadIdx.x;
        const bool in = j < n_v;
        V acc = V();
        const uint4* dl = reinterpret_cast<const uint4*>(a.q_dense16 + a.q_dstart[q]);  // eight rows each
        const V* base = reinterpret_cast<const V*>(ix.dense) + (in ? j : 0u);
        // the list is read eight rows ahead (a single query of c1's kind on 2^22
        // ads 39.6 -> 37.6 us, the marks' words at once in the scatter with it)
        uint4 nr = nd ? dl[0] : make_uint4(0u, 0u, 0u, 0u);
        for (uint32_t k = 0; k < nd; k += KT) {
            const uint4 r = nr;
            if (k + KT < nd) nr = dl[k / KT + 1u];
            const uint32_t row[KT] = {r.x & 0xffffu, r.x >> 16, r.y & 0xffffu, r.y >> 16,
                                      r.z & 0xffffu, r.z >> 16, r.w & 0xffffu, r.w >> 16};
            V x[KT];
#pragma unroll
            for (uint32_t e = 0; e < KT; ++e)  // past the list: its first row of the eight again
                x[e] = __ldg(base + uint64_t(k + e < nd ? row[e] : row[0]) * st);
#pragma unroll
            for (uint32_t e = 0; e < KT; ++e) or_in(acc, x[e]);
            if (__all_sync(kFull, full_vec(acc) || !in)) break;
        }
        const uint32_t ones = __ballot_sync(kFull, in && full_vec(acc));
        if (a.sat && VW == 4u && (lane_id() & 15u) == 0 && (ones >> lane_id() & 0xffffu) == 0xffffu) {
            const uint32_t t = uint32_t(j / 16u);  // tile-of-64
            atomicOr(a.sat + uint64_t(q) * a.sat_stride + (t >> 5), 1u << (t & 31u));
        }
        if (!in) continue;
        uint32_t* dst = a.out + uint64_t(q) * a.out_stride + j * VW;
        const uint32_t* w = reinterpret_cast<const uint32_t*>(&acc);
        const uint64_t left = a.n_words - j * VW;
        if (!ACC && left >= VW) {
            *reinterpret_cast<V*>(dst) = acc;
        } else {
#pragma unroll
            for (uint32_t e = 0; e < VW; ++e)
                if (e < left) {
                    if (!ACC) dst[e] = w[e];
                    else if (w[e]) atomicOr(dst + e, w[e]);
                }
        }
    }
}

// list-union, merge variant, for lists without dense bitmaps that HYBRID and
// TILE queries merge per tile (the dense ones are in the output already): the
// queries the plan kernel listed, tile by tile; blocks that overlap the tile
// are decoded a warp each into the tile in shared memory.
// ACC: start from an empty tile and OR it into the caller's bitmap with
// atomics (other calls may do so at the same time).
template <int W, int NW, bool ACC>
__global__ void __launch_bounds__(NW * 32) tile_union_kernel(IndexView ix, TileArgs a) {
    constexpr int NT = NW * 32;
    constexpr uint32_t SPAN = uint32_t(W) * 32u;
    extern __shared__ __align__(16) uint32_t tile[];  // W words, dynamic (up to 64 KB)
    __shared__ __align__(16) uint4 stage[NW][32];
    __shared__ uint32_t s_lo[NT];
    __shared__ uint32_t s_pref[NT + 1];
    __shared__ uint32_t s_warp[32];
    const uint32_t tid = threadIdx.x, warp = warp_id();
    wait_previous();
    const uint32_t n_q = *a.n_tile_list;
    const uint64_t items = uint64_t(n_q) * a.n_tiles;
    uint4* tile4 = reinterpret_cast<uint4*>(tile);
    for (uint64_t item = blockIdx.x; item < items; item += gridDim.x) {
        // tile-major order: the CTAs resident together work on one region of
        // the ad space for many queries, so the blocks of lists those queries
        // share are read from L2
        const uint32_t t = uint32_t(item / n_q);
        const uint32_t q = a.tile_list[uint32_t(item - uint64_t(t) * n_q)];
        const uint32_t lo_id = t * SPAN;
        const uint32_t hi_id = (uint64_t(lo_id) + SPAN > ix.n_ads) ? ix.n_ads : lo_id + SPAN;
        const uint32_t dj0 = lo_id >> kDirShift;
        uint32_t dj1 = uint32_t((uint64_t(lo_id) + SPAN) >> kDirShift);
        if (dj1 > ix.dir_n - 1) dj1 = ix.dir_n - 1;
        const uint64_t qb = a.q_off[q], qe = a.q_off[q + 1];
        uint32_t* dst = a.out + uint64_t(q) * a.out_stride + uint64_t(t) * W;
        const uint64_t left = a.n_words - uint64_t(t) * W;
        const uint32_t nw = left < uint64_t(W) ? uint32_t(left) : uint32_t(W);
        for (uint32_t i = tid; i < uint32_t(W); i += NT) tile[i] = (!ACC && i < nw) ? dst[i] : 0u;
        __syncthreads();
        for (uint64_t c0 = qb; c0 < qe; c0 += NT) {
            const uint64_t i = c0 + tid;
            uint32_t lo = 0, cnt = 0;
            const uint32_t cls = i < qe ? __ldg(a.tile_cls + i) : kNone;  // two kernels back
            if (cls != kNone) tile_block_range(ix, cls, lo_id, hi_id, dj0, dj1, lo, cnt);
            uint32_t total;
            const uint32_t ex = block_excl_scan<NT>(cnt, s_warp, &total);
            s_lo[tid] = lo;
            s_pref[tid] = ex;
            if (tid == NT - 1) s_pref[NT] = ex + cnt;
            __syncthreads();
            // decode the blocks: warp w takes a contiguous share of the flat
            // block range, finds its first (slot, block) once and walks on,
            // keeping the next block's loads in flight
            const uint32_t per = (total + NW - 1) / NW;
            uint32_t f = warp * per;
            const uint32_t fend = f + per < total ? f + per : total;
            if (f < fend) {
                uint32_t s = find_slot<NT>(s_pref, f);
                uint32_t j = f - s_pref[s];
                Fetched nxt = fetch_block(ix, s_lo[s] + j);
                while (f < fend) {
                    const Fetched cur = nxt;
                    if (++f < fend) {
                        if (++j == s_pref[s + 1] - s_pref[s]) {  // next list with blocks in this tile
                            j = 0;
                            do {
                                ++s;
                            } while (s_pref[s + 1] == s_pref[s]);
                        }
                        nxt = fetch_block(ix, s_lo[s] + j);
                    }
                    uint32_t id[4], cnt_b;
                    decode_fetched(cur, stage[warp], id, cnt_b);
                    or_tile(tile, lo_id, SPAN, id, cnt_b);
                }
            }
            __syncthreads();
        }
        if constexpr (ACC) {
            for (uint32_t i = tid; i < nw; i += NT)
                if (tile[i]) atomicOr(dst + i, tile[i]);
        } else if (a.vec_ok) {
            uint4* d4 = reinterpret_cast<uint4*>(dst);
            for (uint32_t j = tid; j * 4u + 3u < nw; j += NT) d4[j] = tile4[j];
            for (uint32_t i = (nw & ~3u) + tid; i < nw; i += NT) dst[i] = tile[i];
        } else {
            for (uint32_t i = tid; i < nw; i += NT) dst[i] = tile[i];
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// list-union, dense group variant: one CTA per SM walks 64- or 32-word
// tiles; for each tile, a 2-D TMA copy stages that tile's slice of every
// dense bitmap in shared memory once (double-buffered where two stages fit:
// the next tile's copy is in flight while this one is merged), then every
// non-probe query of the batch ORs its dense slices from shared memory and
// writes its tile (the merge kernel later adds the lists without dense
// bitmaps that a query merges). Dense bitmaps shared by many queries are
// read from L2 / HBM once per tile instead of once per query and tile.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], "
        "[%4];" ::"r"(smem_addr(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_addr(bar))
        : "memory");
}

constexpr uint32_t kGroupThreads = 1024;

// What one lane ORs per row: one word of a 32-word tile, two of a 64-word one.
template <uint32_t GW> struct GroupWord;
template <> struct GroupWord<32> { typedef uint32_t T; };
template <> struct GroupWord<64> { typedef uint2 T; };
__device__ __forceinline__ uint32_t orw(uint32_t a, uint32_t b) { return a | b; }
__device__ __forceinline__ uint2 orw(uint2 a, uint2 b) { return make_uint2(a.x | b.x, a.y | b.y); }
template <typename T> __device__ __forceinline__ T zero_word();
template <> __device__ __forceinline__ uint32_t zero_word<uint32_t>() { return 0u; }
template <> __device__ __forceinline__ uint2 zero_word<uint2>() { return make_uint2(0u, 0u); }
__device__ __forceinline__ bool all_ones(uint32_t a) { return a == ~0u; }
__device__ __forceinline__ bool all_ones(uint2 a) { return (a.x & a.y) == ~0u; }
// OR of a lane's words (word w and on) into the output, by atomics: other
// queries may share the bitmap
__device__ __forceinline__ void or_words(uint32_t* o, uint32_t a, uint64_t w, uint64_t n_words) {
    if (a && w < n_words) atomicOr(o, a);
}
__device__ __forceinline__ void or_words(uint32_t* o, uint2 a, uint64_t w, uint64_t n_words) {
    if (a.x && w < n_words) atomicOr(o, a.x);
    if (a.y && w + 1u < n_words) atomicOr(o + 1, a.y);
}
// true when the warp's whole tile slice is set: no further row can change it
template <typename T>
__device__ __forceinline__ bool tile_full(T acc) { return __all_sync(kFull, all_ones(acc)); }

// Row `woff` (a word offset, row * GW) of a stage, at this lane's column
// (B = stage + lane * GW / 32 words)
template <typename T>
__device__ __forceinline__ T ld_row(const uint8_t* B, uint32_t woff) {
    return *reinterpret_cast<const T*>(B + (woff << 2));
}
template <typename T>
__device__ __forceinline__ T or2w(const uint8_t* B, uint32_t v) {
    return orw(ld_row<T>(B, v & 0xffffu), ld_row<T>(B, v >> 16));
}
// OR of the 8 rows named by the 16-bit word offsets in v
template <typename T>
__device__ __forceinline__ T or8w(const uint8_t* B, uint4 v) {
    return orw(orw(orw(ld_row<T>(B, v.x & 0xffffu), ld_row<T>(B, v.x >> 16)),
                   orw(ld_row<T>(B, v.y & 0xffffu), ld_row<T>(B, v.y >> 16))),
               orw(orw(ld_row<T>(B, v.z & 0xffffu), ld_row<T>(B, v.z >> 16)),
                   orw(ld_row<T>(B, v.w & 0xffffu), ld_row<T>(B, v.w >> 16))));
}
// OR over a list of nd word offsets (padded to a multiple of 8 with the
// zero row), 16 at a time: per row one extract, one address, one shared load.
// The lists are in ascending bitmap order, which is longest list first, so a
// tile of a dense query saturates early; the warp stops once every bit of
// its slice is set (about 30 % of the row reads on config c1).
template <typename T>
__device__ __forceinline__ T or_list_words(const uint8_t* B, const uint4* ol, uint32_t nd) {
    T acc = zero_word<T>();
    uint32_t k = 0;
    for (; k + 16u <= nd; k += 16u) {
        acc = orw(acc, orw(or8w<T>(B, ol[k >> 3]), or8w<T>(B, ol[(k >> 3) + 1])));
        if (tile_full(acc)) return acc;
    }
    if (k + 8u <= nd) {
        acc = orw(acc, or8w<T>(B, ol[k >> 3]));
        k += 8u;
    }
    // the last 0 .. 7 rows, without the list's padding
    const uint32_t r = nd - k;
    if (r) {
        uint4 v = ol[k >> 3];
        if (r & 4u) {
            acc = orw(acc, orw(or2w<T>(B, v.x), or2w<T>(B, v.y)));
            v.x = v.z;
            v.y = v.w;
        }
        if (r & 2u) {
            acc = orw(acc, or2w<T>(B, v.x));
            v.x = v.y;
        }
        if (r & 1u) acc = orw(acc, ld_row<T>(B, v.x & 0xffffu));
    }
    return acc;
}
// Shared memory (dynamic, 1024-byte aligned base): two stages of n_rows x
// GW words (rows = dense bitmaps + the zero row), then per such query
// its list's offset and length, the queue of those queries, and the
// lists themselves when they fit (else they are read from global memory): the
// plan kernel writes them as 16-bit row word offsets (row * GW). GW = 64 halves the
// index work per word (each lane ORs two words per row) where two stages of
// 64-word rows fit.
// ACC: OR into the output with atomics (bitmaps may be shared, rows need no
// alignment) instead of overwriting it.
template <uint32_t GW, bool ACC>
__global__ void __launch_bounds__(kGroupThreads, 1)
    dense_group_kernel(const __grid_constant__ CUtensorMap tmap_full, const __grid_constant__ CUtensorMap tmap_last,
                       DenseGroupArgs a) {
    typedef typename GroupWord<GW>::T T;
    constexpr uint32_t kLaneWords = GW / 32u;
    static_assert(kGroupMaxBoxes * kGroupBoxRows * GW < 65536u, "16-bit word offsets");
    extern __shared__ uint8_t g_raw[];
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ uint32_t s_next[2];
    __shared__ uint32_t s_ndq;
    __shared__ uint32_t s_warp[32];
    uint8_t* base = g_raw + ((1024u - (smem_addr(g_raw) & 1023u)) & 1023u);
    const uint32_t stage_bytes = (a.n_rows * GW * 4u + 1023u) & ~1023u;
    const bool dbl = a.stages == 2u;  // two stages: the next tile's copy overlaps this tile's merge
    uint32_t* stage0 = reinterpret_cast<uint32_t*>(base);
    uint32_t* s_meta = reinterpret_cast<uint32_t*>(base + a.stages * stage_bytes);  // n_q: list offset / 8 << 16 | nd
    uint16_t* s_qlist = reinterpret_cast<uint16_t*>(s_meta + a.n_q);               // queries with work
    uint4* s_lists = reinterpret_cast<uint4*>(base + a.stages * stage_bytes + ((6u * a.n_q + 15u) & ~15u));
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    constexpr uint32_t kNW = kGroupThreads / 32u;
    wait_previous();
    uint32_t t = blockIdx.x;
    if (t >= a.n_tiles) return;
    const uint32_t n_q = a.d_n_q ? min(*a.d_n_q, a.n_q) : a.n_q;
    const uint32_t full_boxes = (a.n_rows - 1u) / kGroupBoxRows;  // boxes of 256 rows before the last
    auto issue = [&](uint32_t tile, uint32_t st) {  // thread 0 only
        fence_proxy_async();  // earlier reads of this stage (ordered by the barrier) before the copy
        mbar_expect_tx(&bar[st], a.n_rows * GW * 4u);
        uint32_t* dst = stage0 + st * (stage_bytes / 4u);
        for (uint32_t j = 0; j < full_boxes; ++j)
            tma_load_2d(dst + j * kGroupBoxRows * GW, &tmap_full, int(tile * GW), int(j * kGroupBoxRows), &bar[st]);
        tma_load_2d(dst + full_boxes * kGroupBoxRows * GW, &tmap_last, int(tile * GW), int(full_boxes * kGroupBoxRows),
                    &bar[st]);
    };
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
        s_next[0] = s_next[1] = 0;
        issue(t, 0);  // the first tile's copy overlaps the list staging below
    }
    // stage those queries' lists (the same for every tile): offsets
    // by a block scan over the queries, at most two per thread
    uint32_t len[2], cnt[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t q = tid * 2u + r;
        // when ORing into the output, queries without dense bitmaps have nothing to add
        const bool dq = q < n_q && !(ACC && a.q_ndense[q] == 0u);
        len[r] = dq ? ((a.q_ndense[q] + 7u) & ~7u) : 0u;
        cnt[r] = dq ? 1u : 0u;
    }
    uint32_t tot_len, tot_cnt;
    const uint32_t off0 = block_excl_scan<kGroupThreads>(len[0] + len[1], s_warp, &tot_len);
    const uint32_t rk0 = block_excl_scan<kGroupThreads>(cnt[0] + cnt[1], s_warp, &tot_cnt);
    const bool in_smem = tot_len <= a.list_cap;
    {
        uint32_t off = off0, rk = rk0;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t q = tid * 2u + r;
            if (q < a.n_q) s_meta[q] = cnt[r] ? ((off >> 3) << 16) | a.q_ndense[q] : 0xffffffffu;
            if (cnt[r]) s_qlist[rk] = uint16_t(q);
            off += len[r];
            rk += cnt[r];
        }
    }
    if (tid == 0) s_ndq = tot_cnt;
    __syncthreads();
    if (in_smem) {
        for (uint32_t i = warp; i < tot_cnt; i += kNW) {  // a warp per query, 16 bytes per lane
            const uint32_t q = s_qlist[i];
            const uint32_t m = s_meta[q];
            const uint4* src = reinterpret_cast<const uint4*>(a.q_dense16 + a.q_dstart[q]);
            uint4* dst = s_lists + (m >> 16);
            for (uint32_t j = lane; j < ((m & 0xffffu) + 7u) / 8u; j += 32u) dst[j] = src[j];
        }
    }
    __syncthreads();
    const uint32_t n_dq = s_ndq;
    uint32_t phase = 0;  // bit s: parity of stage s's next completion
    for (uint32_t it = 0; t < a.n_tiles; ++it, t += gridDim.x) {
        const uint32_t st = dbl ? (it & 1u) : 0u;
        const bool more = t + gridDim.x < a.n_tiles;
        const uint32_t par = (phase >> st) & 1u;
        const bool ok = mbar_wait_bounded(&bar[st], par, a.spin_limit);
        if (__syncthreads_or(!ok)) {
            // The copy into this stage is the only one in flight: the next
            // tile's copy is issued only after a wait succeeds. It gets one
            // more bounded interval to land before the CTA (and its shared
            // memory) goes; a copy still pending after that is abandoned
            // with the error bit set.
            if (tid == 0) atomicOr(a.err, kErrTmaTimeout);
            mbar_wait_bounded(&bar[st], par, a.spin_limit);
            return;
        }
        phase ^= 1u << st;
        // the other stage was released by the barrier that ended the previous
        // tile: its refill overlaps this tile's merge
        if (tid == 0 && more && dbl) issue(t + gridDim.x, st ^ 1u);
        const uint32_t* S = stage0 + st * (stage_bytes / 4u);
        const uint8_t* B = reinterpret_cast<const uint8_t*>(S + lane * kLaneWords);
        const uint64_t w = uint64_t(t) * GW + lane * kLaneWords;
        for (;;) {
            uint32_t i = 0;
            if (lane == 0) i = atomicAdd(&s_next[st], 1u);
            i = __shfl_sync(kFull, i, 0);
            if (i >= n_dq) break;
            const uint32_t q = s_qlist[i];
            const uint32_t m = s_meta[q];
            const uint32_t nd = m & 0xffffu;
            const T acc = in_smem ? or_list_words<T>(B, s_lists + (m >> 16), nd)
                                  : or_list_words<T>(B, reinterpret_cast<const uint4*>(a.q_dense16 + a.q_dstart[q]), nd);
            if (a.sat && tile_full(acc) && lane == 0)
                atomicOr(a.sat + uint64_t(q) * a.sat_stride + (t >> 5), 1u << (t & 31u));
            if constexpr (ACC) {
                or_words(a.out + uint64_t(a.out_slot ? a.out_slot[q] : q) * a.out_stride + w, acc, w, a.n_words);
                continue;
            }
            uint32_t* o = a.out + uint64_t(q) * a.out_stride + w;
            if constexpr (GW == 64u) {
                if (w + 1u < a.n_words) *reinterpret_cast<uint2*>(o) = acc;  // 8-byte aligned (checked at launch)
                else if (w < a.n_words) o[0] = acc.x;
            } else {
                if (w < a.n_words) o[0] = acc;
            }
        }
        __syncthreads();  // this stage is read; the next iteration may refill it
        if (tid == 0) {
            s_next[st] = 0;
            // one stage: the next tile's copy starts now that every warp is
            // done with this one (the arrive in issue() publishes the reset)
            if (!dbl && more) issue(t + gridDim.x, 0u);
        }
    }
}

// ---------------------------------------------------------------------------
// list-union, scatter variant (load-balanced over the short lists' blocks)
// ---------------------------------------------------------------------------
// Lean decode of one block by one warp, from payload words read straight into
// registers: lane l takes gap slots 4l .. 4l+3, that is ids 4l+1 .. 4l+4, and
// the last lane's fourth position (a block has at most 127 gaps) stands for
// the block's first id. Only for bits <= 16: the lane's four gaps then lie in
// the 64 bits from bit 4 * bits * l, three words at most.
struct GapWords {
    uint32_t x0, x1, x2;
};
__device__ __forceinline__ GapWords load_gaps(const IndexView& ix, uint32_t unit, uint32_t meta) {
    const uint32_t bits = meta & 63u, gaps = (meta >> 8) & 127u;
    GapWords g{0u, 0u, 0u};
    // a lane whose first slot exists reads at most two words past the block's
    // last one: inside the payload's padding unit
    if (4u * lane_id() < gaps) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(ix.payload + unit) + ((4u * bits * lane_id()) >> 5);
        g.x0 = __ldg(w);
        g.x1 = __ldg(w + 1);
        g.x2 = __ldg(w + 2);
    }
    return g;
}
__device__ __forceinline__ void gaps_to_ids(uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3, uint32_t first,
                                            uint32_t (&id)[4]) {
    const uint32_t lane = lane_id();
    const uint32_t p0 = v0 + 1u, p1 = p0 + v1 + 1u, p2 = p1 + v2 + 1u, run = p2 + v3 + 1u;
    uint32_t x = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, x, o);
        if (lane >= uint32_t(o)) x += y;
    }
    const uint32_t base = first + (x - run);
    id[0] = base + p0;
    id[1] = base + p1;
    id[2] = base + p2;
    id[3] = lane == 31u ? first : base + run;
}
// ids of this lane's four positions; position k is valid when 4 * lane + k <
// gaps, and lane 31's fourth always is
__device__ __forceinline__ void decode_gaps(const GapWords& g, uint32_t first, uint32_t meta, uint32_t (&id)[4]) {
    const uint32_t lane = lane_id(), bits = meta & 63u, mask = (1u << bits) - 1u;
    const uint32_t off = (4u * bits * lane) & 31u;
    uint32_t lo = __funnelshift_r(g.x0, g.x1, off), hi = __funnelshift_r(g.x1, g.x2, off);
    const uint32_t v0 = lo & mask, v1 = __funnelshift_r(lo, hi, bits) & mask;
    lo = __funnelshift_rc(lo, hi, 2u * bits);
    hi = __funnelshift_rc(hi, 0u, 2u * bits);
    const uint32_t v2 = lo & mask, v3 = __funnelshift_r(lo, hi, bits) & mask;
    gaps_to_ids(v0, v1, v2, v3, first, id);
}
// The same for any width, with each gap's two words read on their own: lists
// whose gaps do not fit 16 bits are short or very uneven.
__device__ __noinline__ void decode_wide(const IndexView& ix, uint32_t unit, uint32_t first, uint32_t meta,
                                         uint32_t (&id)[4]) {
    const uint32_t bits = meta & 63u, gaps = (meta >> 8) & 127u;
    const uint32_t mask = bits >= 32u ? kFull : (1u << bits) - 1u;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(ix.payload + unit);
    uint32_t v[4];
#pragma unroll
    for (uint32_t e = 0; e < 4u; ++e) {
        const uint32_t s = 4u * lane_id() + e, pos = s * bits;
        v[e] = s < gaps ? __funnelshift_r(__ldg(w + (pos >> 5)), __ldg(w + (pos >> 5) + 1), pos & 31u) & mask : 0u;
    }
    gaps_to_ids(v[0], v[1], v[2], v[3], first, id);
}

// last i in [0, n) with at(i) <= key, by the whole warp (32 probes a step);
// at(0) <= key, at ascending
template <typename At, typename Key>
__device__ __forceinline__ uint32_t warp_last_le(At at, uint32_t n, Key key) {
    uint32_t lo = 0;
    while (n > 1u) {
        const uint32_t step = (n + 31u) / 32u, i = lane_id() * step;
        const bool le = i < n && at(lo + i) <= key;
        const uint32_t k = uint32_t(__popc(__ballot_sync(kFull, le))) - 1u;
        lo += k * step;
        n = n - k * step < step ? n - k * step : step;
    }
    return lo;
}

// Load-balanced warps over the short lists' blocks. A warp takes a chunk of up
// to 32 consecutive blocks of the flat block order (queries, then their term
// slots, then the slots' blocks) and works in two parts:
//  * a lane per block: find the block's query and term slot, read its bounds
//    and descriptor, and test its id range against the saturation marks of its
//    bitmap. Blocks in all-ones tiles only are dropped here, before any of
//    their payload is read;
//  * a warp per remaining block: decode (the next block's payload loads in
//    flight) and OR, one atomic per word a lane's ids touch; a block of which
//    some tiles are all ones skips the ORs into those.
// Bound: the atomics' way to L2 (see bin_kernel). Walking the blocks one by
// one (slot arithmetic, bound and descriptor loads by the whole warp, gaps
// staged in shared memory) took about 300 instructions per block of 128 ids
// and a chain of ~20 loads per chunk: one query's few hundred blocks 16.5 us
// where they now take 4 (c0), 32 queries' 94 thousand 49 instead of 55.
// KEYED: every term slot has an output bitmap of its own.
template <int NW, bool KEYED>
__global__ void __launch_bounds__(NW * 32, 6) scatter_kernel(IndexView ix, ScatterArgs a) {
    __shared__ __align__(16) uint4 s_blk[NW][32];  // {payload unit, first id, meta | kMixed, output bitmap}
    __shared__ uint32_t s_row[NW][32];             // row of saturation marks
    constexpr uint32_t kMixed = 0x80000000u;       // some of the block's tiles are all ones
    const uint32_t warp = warp_id(), lane = lane_id();
    wait_previous();
    const uint32_t n_q = a.d_n_q ? min(*a.d_n_q, a.n_q) : a.n_q;
    if (n_q == 0) return;
    const uint64_t total = a.q_light_pref[n_q];
    const uint64_t nwt = uint64_t(gridDim.x) * NW;
    // few blocks: fewer per warp, so that every warp has some
    const uint64_t per = (total + nwt - 1) / nwt;
    const uint32_t chunk = per < a.chunk_blocks ? uint32_t(per) : a.chunk_blocks;
    const uint32_t tshift = a.sat_shift + 5u;  // id -> tile
    for (uint64_t f0 = (uint64_t(blockIdx.x) * NW + warp) * chunk; f0 < total; f0 += nwt * chunk) {
        // ---- a lane per block ----
        const bool mine = lane < chunk && f0 + lane < total;
        const uint64_t f = mine ? f0 + lane : f0;
        uint32_t q = warp_last_le([&](uint32_t i) { return a.q_light_pref[i]; }, n_q, f0);
        uint64_t pq = a.q_light_pref[q];
        for (uint64_t nx; (nx = a.q_light_pref[q + 1]) <= f; pq = nx) ++q;
        const uint32_t r = uint32_t(f - pq);
        uint64_t slot = 0;
        uint2 sl = make_uint2(0u, 0u);  // the slot's first block: flat in its query, and in the index
        for (uint32_t todo = kFull; todo;) {
            const int lead = __ffs(todo) - 1;
            const uint32_t ql = __shfl_sync(kFull, q, lead);
            const uint32_t rl = __shfl_sync(kFull, r, lead);
            const uint64_t qb = a.q_off[ql];
            const uint32_t n = uint32_t(a.q_off[ql + 1] - qb);
            uint32_t base = warp_last_le([&](uint32_t i) { return a.term_slot[qb + i].x; }, n, rl);
            // 32 slots at a time: rank of each of this query's lanes among their prefixes
            for (uint32_t left = __ballot_sync(kFull, (todo >> lane & 1u) && q == ql);; base += 31u) {
                const uint2 p = base + lane < n ? a.term_slot[qb + base + lane] : make_uint2(kFull, 0u);
                uint32_t at = 0;
#pragma unroll
                for (uint32_t h = 16; h; h >>= 1) {
                    const uint32_t y = __shfl_sync(kFull, p.x, at + h);
                    if (y <= r) at += h;
                }
                const uint32_t px = __shfl_sync(kFull, p.x, at), py = __shfl_sync(kFull, p.y, at);
                const bool in = left >> lane & 1u;
                const bool done = in && at < 31u;
                if (done) {
                    slot = qb + base + at;
                    sl = make_uint2(px, py);
                }
                const uint32_t d = __ballot_sync(kFull, done);
                left &= ~d;
                todo &= ~d;
                if (!left) break;
            }
        }
        const uint32_t b = sl.y + (r - sl.x);
        const uint32_t first = __ldg(ix.blk_first + b);
        const uint2 desc = __ldg(ix.blk_desc + b);
        const uint32_t out_i = KEYED ? a.key_slot[slot] : a.out_slot ? a.out_slot[q] : q;
        uint32_t meta = desc.y;
        bool live = mine;
        if (a.sat) {
            const uint32_t row = min(q, a.sat_last);
            const uint32_t* sat = a.sat + uint64_t(row) * a.sat_stride;
            const uint32_t t0 = first >> tshift, t1 = __ldg(ix.blk_last + b) >> tshift;
            const uint32_t w0 = t0 >> 5, w1 = t1 >> 5;
            bool all = true, some = false;
            // the first and the last word of marks at once: most blocks have no other
            const uint32_t va = sat[w0], vb = sat[w1];
            if (w1 - w0 < 32u) {
                uint32_t ma = kFull << (t0 & 31u), mb = kFull >> (31u - (t1 & 31u));
                if (w0 == w1) ma = mb = ma & mb;
                all = (va & ma) == ma && (vb & mb) == mb;
                some = ((va & ma) | (vb & mb)) != 0u;
                for (uint32_t w = w0 + 1u; w < w1; ++w) {
                    const uint32_t v = sat[w];
                    all &= v == kFull;
                    some |= v != 0u;
                }
            } else {  // a wide range is not checked as a whole
                all = false;
                some = true;
            }
            live = mine && !all;
            if (some) meta |= kMixed;
            s_row[warp][lane] = row;
        }
        __syncwarp();
        s_blk[warp][lane] = make_uint4(desc.x, first, meta, out_i);
        __syncwarp();
        // ---- a warp per block ----
        uint32_t todo = __ballot_sync(kFull, live);
        if (!todo) continue;
        uint32_t k = uint32_t(__ffs(todo)) - 1u;
        uint4 nb = s_blk[warp][k];
        GapWords ng = load_gaps(ix, nb.x, nb.z);
        while (todo) {
            const uint4 cb = nb;
            const GapWords cg = ng;
            const uint32_t ck = k;
            todo &= todo - 1u;
            if (todo) {
                k = uint32_t(__ffs(todo)) - 1u;
                nb = s_blk[warp][k];
                ng = load_gaps(ix, nb.x, nb.z);
            }
            uint32_t* out = a.out + uint64_t(cb.w) * a.out_stride;
            const uint32_t* sat = cb.z & kMixed ? a.sat + uint64_t(s_row[warp][ck]) * a.sat_stride : nullptr;
            uint32_t id[4];
            if ((cb.z & 63u) > 16u) decode_wide(ix, cb.x, cb.y, cb.z, id);
            else decode_gaps(cg, cb.y, cb.z, id);
            const uint32_t gaps = (cb.z >> 8) & 127u;
            uint32_t m[4];
#pragma unroll
            for (uint32_t e = 0; e < 4u; ++e) m[e] = 1u << (id[e] & 31u);
            if (gaps != 127u) {  // warp-uniform: a list's last block
#pragma unroll
                for (uint32_t e = 0; e < 4u; ++e)
                    if (4u * lane + e >= gaps && !(e == 3u && lane == 31u)) m[e] = 0u;
            }
            if (sat) {
#pragma unroll
                for (uint32_t e = 0; e < 4u; ++e) {
                    const uint32_t t = id[e] >> tshift;
                    if (m[e] && (sat[t >> 5] >> (t & 31u) & 1u)) m[e] = 0u;
                }
            }
            // ids of one word become one atomic
#pragma unroll
            for (uint32_t e = 0; e < 3u; ++e) {
                if ((id[e] ^ id[e + 1]) < 32u) {
                    m[e + 1] |= m[e];
                    m[e] = 0u;
                }
            }
#pragma unroll
            for (uint32_t e = 0; e < 4u; ++e)
                if (m[e]) atomicOr(out + (id[e] >> 5), m[e]);
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// list-union, binned variant
// ---------------------------------------------------------------------------
// The plain ids of the lists in plain_term, a warp per block.
__global__ void __launch_bounds__(256) plain_ids_kernel(IndexView ix, const uint32_t* plain_off, uint32_t* plain) {
    const uint64_t nw = uint64_t(gridDim.x) * 8u;
    for (uint64_t b = uint64_t(blockIdx.x) * 8u + warp_id(); b < ix.n_blocks; b += nw) {
        const uint32_t t = __ldg(ix.blk_term + b), p = __ldg(ix.term_plain + t);
        if (p == kNone) continue;
        const uint2 d = __ldg(ix.blk_desc + b);
        const uint32_t first = __ldg(ix.blk_first + b), gaps = d.y >> 8;
        uint32_t id[4];
        if ((d.y & 63u) > 16u) decode_wide(ix, d.x, first, d.y, id);
        else decode_gaps(load_gaps(ix, d.x, d.y), first, d.y, id);
        uint32_t* dst = plain + uint64_t(__ldg(plain_off + p)) * 4u + (b - __ldg(ix.term_blk + t)) * ABF_BLOCK_POSTINGS;
#pragma unroll
        for (uint32_t e = 0; e < 4u; ++e) {
            const uint32_t s = 4u * lane_id() + e;  // gap slot: the id after it
            if (s < gaps) dst[s + 1u] = id[e];
            else if (s == ABF_BLOCK_POSTINGS - 1u) dst[0] = first;
        }
    }
}

// The plan kernel's tables: per term {first block, postings, dense bitmap,
// plain list}, and what the planner's features add up (cbytes: compressed
// bytes, null: left as they are).
__global__ void __launch_bounds__(256) term_info_kernel(IndexView ix, uint4* info, TermFeat* feat,
                                                        const uint32_t* cbytes) {
    const double inv_ads = 1.0 / double(ix.n_ads);
    for (uint32_t t = blockIdx.x * 256u + threadIdx.x; t < ix.n_terms; t += gridDim.x * 256u) {
        const uint32_t len = ix.term_len[t];
        info[t] = make_uint4(ix.term_blk[t], len, ix.term_dense[t], ix.n_plain ? ix.term_plain[t] : kNone);
        if (cbytes) feat[t] = TermFeat{log1p(-fmin(double(len) * inv_ads, 0.999999)), cbytes[t], 0u};
    }
}

// position in the plain ids of each list's first id at or past every tile start
__global__ void __launch_bounds__(256) plain_dir_kernel(IndexView ix, const uint32_t* plain_term,
                                                        const uint32_t* plain_off, uint32_t* dir) {
    const uint64_t n = uint64_t(ix.n_plain) * ix.plain_dir_n;
    for (uint64_t i = uint64_t(blockIdx.x) * 256u + threadIdx.x; i < n; i += uint64_t(gridDim.x) * 256u) {
        const uint32_t p = uint32_t(i / ix.plain_dir_n), j = uint32_t(i - uint64_t(p) * ix.plain_dir_n);
        const uint32_t len = __ldg(ix.term_len + plain_term[p]), a0 = plain_off[p] * 4u;
        const uint64_t key = uint64_t(j) << kBinShift;
        dir[i] = a0 + (key >= ix.n_ads ? len : lower_bound_g(ix.plain + a0, 0u, len, uint32_t(key)));
    }
}

// A lane's global atomic is a 32-byte sector of its own on the way to L2: an
// SM sends about one per clock, so the scatter kernel stops at ~300 G
// postings/s however few instructions it takes, and where the batch's bitmaps
// exceed L2 each such sector is read from and written to HBM. Shared-memory
// atomics go at about ten lanes a clock. So in large batches the lists of mid
// length (plain ids, no dense bitmap) are merged per tile: a CTA takes one
// (tile, query, part) item at a time from a ticket counter, loads its 16,384
// words of the bitmap (the group kernel's output), looks up each list's ids in
// the tile (a thread per list), cuts them into chunks of at most 256 (a thread
// per chunk), ORs the chunks (a warp per chunk, eight ids a lane) and writes
// the tile back. Tiles-of-64 that are all ones already are neither read nor
// written. Items run tile by tile, so that the ids that queries share are read
// from L2. A query with more than its share of ids is cut into parts by its
// lists; their tiles start at zero and are ORed into the output by coalesced
// atomics.
// 512 queries of config c1: 550 us (333 of them the tiles' round trip through
// HBM), and the scatter kernel's share falls from 1,269 to 110; 2,048 queries
// of config c2: 2.65 and 0.47 ms where the scatter took 9.72. The same from
// the packed blocks (bounds, decode and range tests per block and tile, ~160
// instructions for 128 ids) took 868 us on c1; testing every id's mark before
// its shared atomic 649; without the shared atomics it takes as long as with.
template <bool ACC>
__global__ void __launch_bounds__(kBinThreads, kBinCtasPerSm) bin_kernel(IndexView ix, BinArgs a) {
    constexpr uint32_t W = kBinWords, NT = kBinThreads, NW = NT / 32u;
    constexpr uint32_t kSub = W / 64u;  // tiles-of-64 of an item, one mark each
    constexpr uint32_t kChunk = 256u;   // ids a warp ORs at a time
    extern __shared__ __align__(16) uint32_t tile[];
    __shared__ uint32_t s_lo[NT], s_n[NT], s_pref[NT + 1], s_warp[32], s_sat[kSub / 32u];
    __shared__ uint2 s_chunk[NT];                 // {position of the first id, ids}
    __shared__ uint64_t s_qb[2];                  // of the current and the next item: first slot of the query,
    __shared__ uint32_t s_it[2][6];                // {item left?, tile, query, part, parts, lists of the query}
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    wait_previous();
    const uint32_t n_q = a.d_n_q ? min(*a.d_n_q, a.n_q) : a.n_q;
    if (n_q == 0) return;
    const uint32_t n_parts = a.parts_pref[n_q];
    if (n_parts == 0) return;
    const uint64_t items = uint64_t(n_parts) * a.n_tiles;
    uint4* tile4 = reinterpret_cast<uint4*>(tile);
    uint8_t* tile_b = reinterpret_cast<uint8_t*>(tile);
    // warp 0 claims an item and looks it up, one item ahead of the CTA's work
    auto claim = [&](uint32_t slot) {
        uint32_t item = 0;
        if (lane == 0) item = atomicAdd(a.ticket, 1u);
        item = __shfl_sync(kFull, item, 0);
        if (item < items) {
            const uint32_t t = item / n_parts, g = item - t * n_parts;
            const uint32_t q = warp_last_le([&](uint32_t i) { return a.parts_pref[i]; }, n_q, g);
            const uint32_t p0 = a.parts_pref[q], p1 = a.parts_pref[q + 1];
            if (lane == 0) {
                s_qb[slot] = a.q_off[q];
                s_it[slot][1] = t;
                s_it[slot][2] = q;
                s_it[slot][3] = g - p0;
                s_it[slot][4] = p1 - p0;
                s_it[slot][5] = a.q_nbin[q];
            }
        }
        if (lane == 0) s_it[slot][0] = item < items ? 1u : 0u;
    };
    if (warp == 0) claim(0);
    __syncthreads();
    for (uint32_t cur = 0;; cur ^= 1u) {
        if (!s_it[cur][0]) return;
        const uint32_t t = s_it[cur][1], q = s_it[cur][2], part = s_it[cur][3], parts = s_it[cur][4];
        const uint64_t qb = s_qb[cur];
        const uint32_t nm = (s_it[cur][5] + parts - 1u - part) / parts;  // this part's lists: part, part + parts, ..
        const bool own = !ACC && parts == 1u;  // nobody else ORs into this tile
        uint32_t* dst = a.out + uint64_t(a.out_slot ? a.out_slot[q] : q) * a.out_stride + uint64_t(t) * W;
        const uint64_t left = a.n_words - uint64_t(t) * W;
        const uint32_t nw = left < uint64_t(W) ? uint32_t(left) : W;
        // marks of the tile; a tile that is all ones needs nothing
        bool full = true;
        if (tid < kSub / 32u) {
            const uint32_t* sat = a.sat + uint64_t(min(q, a.sat_last)) * a.sat_stride;
            uint32_t v = 0;
            if (a.sat_shift == 6u) {
                const uint32_t w = t * (kSub / 32u) + tid;
                if (w < a.sat_stride) v = sat[w];
            } else {  // marks of 32-word tiles: both halves
                for (uint32_t h = 0; h < 2u; ++h) {
                    const uint32_t w = (t * (kSub / 32u) + tid) * 2u + h;
                    const uint32_t x = w < a.sat_stride ? sat[w] : 0u;
                    for (uint32_t b = 0; b < 16u; ++b) v |= ((x >> (2u * b) & 3u) == 3u ? 1u : 0u) << (h * 16u + b);
                }
            }
            s_sat[tid] = v;
            const uint32_t n = (nw + 63u) / 64u;  // marks in use
            const uint32_t used = tid * 32u >= n ? 0u : n - tid * 32u >= 32u ? kFull : (1u << (n - tid * 32u)) - 1u;
            full = (v & used) == used;
        }
        const bool skip = __syncthreads_and(full);
        if (warp == 0) claim(cur ^ 1u);
        if (skip) {
            __syncthreads();
            continue;
        }
        // the tile's words come in while the lists are looked up. Thread tid's
        // 16-byte slots are tid + NT * k, in tiles-of-64 tid / 16 + 32 * k: bit
        // tid / 16 of mark word k
        const uint32_t mbit = 1u << (tid >> 4);
        static_assert(NT == 512 && kSub == 256, "mark word k covers the slots tid + NT * k");
        if (own && a.vec_ok && nw == W) {
#pragma unroll
            for (uint32_t k = 0; k < kSub / 32u; ++k)
                if (!(s_sat[k] & mbit)) cp_async16(tile4 + tid + NT * k, dst + (tid + NT * k) * 4u);
        } else if (own) {
            for (uint32_t i = tid; i < W; i += NT) tile[i] = i < nw ? dst[i] : 0u;
        } else {
#pragma unroll
            for (uint32_t k = 0; k < kSub / 32u; ++k) tile4[tid + NT * k] = make_uint4(0u, 0u, 0u, 0u);
        }
        for (uint32_t c0 = 0; c0 < nm; c0 += NT) {
            uint32_t lo = 0, n = 0;
            if (c0 + tid < nm) {
                const uint32_t* d = ix.plain_dir +
                                    uint64_t(a.bin_list[qb + part + uint64_t(c0 + tid) * parts]) * ix.plain_dir_n + t;
                lo = __ldg(d);
                n = __ldg(d + 1) - lo;
            }
            uint32_t total;
            const uint32_t ex = block_excl_scan<int(NT)>((n + kChunk - 1u) / kChunk, s_warp, &total);
            s_lo[tid] = lo;
            s_n[tid] = n;
            s_pref[tid] = ex;
            if (tid == NT - 1u) s_pref[NT] = ex + (n + kChunk - 1u) / kChunk;
            cp_async_wait_all();
            __syncthreads();  // also: the tile is loaded
            for (uint32_t f0 = 0; f0 < total; f0 += NT) {
                const uint32_t m = min(NT, total - f0);
                if (tid < m) {
                    const uint32_t s = find_slot<int(NT)>(s_pref, f0 + tid), k = (f0 + tid - s_pref[s]) * kChunk;
                    s_chunk[tid] = make_uint2(s_lo[s] + k, min(kChunk, s_n[s] - k));
                }
                __syncthreads();
                // the next chunk's ids are in flight while one is ORed
                constexpr uint32_t E = kChunk / 32u;
                uint32_t nx[E], nn = 0;
                auto fetch = [&](uint32_t i) {
                    const uint2 c = s_chunk[i];
                    const uint32_t* src = ix.plain + c.x + lane;
                    nn = c.y;
#pragma unroll
                    for (uint32_t e = 0; e < E; ++e)
                        if (lane + 32u * e < c.y) nx[e] = __ldg(src + 32u * e);
                };
                if (warp < m) fetch(warp);
                for (uint32_t i = warp; i < m; i += NW) {
                    uint32_t x[E];
                    const uint32_t cn = nn;
#pragma unroll
                    for (uint32_t e = 0; e < E; ++e) x[e] = nx[e];
                    if (i + NW < m) fetch(i + NW);
                    // a tile starts at a multiple of 2^19 ads: the byte of an
                    // id's word in it is (id >> 3) mod 64 K, less two bits
                    auto put = [&](uint32_t e) {
                        atomicOr(reinterpret_cast<uint32_t*>(tile_b + (x[e] >> 3 & (W * 4u - 4u))), 1u << (x[e] & 31u));
                    };
                    if (cn == kChunk) {
#pragma unroll
                        for (uint32_t e = 0; e < E; ++e) put(e);
                    } else {
#pragma unroll
                        for (uint32_t e = 0; e < E; ++e)
                            if (lane + 32u * e < cn) put(e);
                    }
                }
                __syncthreads();
            }
        }
        if (own) {
            if (a.vec_ok && nw == W) {
#pragma unroll
                for (uint32_t k = 0; k < kSub / 32u; ++k)
                    if (!(s_sat[k] & mbit)) reinterpret_cast<uint4*>(dst)[tid + NT * k] = tile4[tid + NT * k];
            } else {
                for (uint32_t i = tid; i < nw; i += NT) dst[i] = tile[i];
            }
        } else if (nw == W) {
#pragma unroll 8
            for (uint32_t i = tid; i < W; i += NT) {
                const uint32_t v = tile[i];
                if (v) atomicOr(dst + i, v);
            }
        } else {
            for (uint32_t i = tid; i < nw; i += NT)
                if (tile[i]) atomicOr(dst + i, tile[i]);
        }
        __syncthreads();  // the tile and the marks are read, the next item is there
    }
}

// ---------------------------------------------------------------------------
// bitmap-probe
// ---------------------------------------------------------------------------
// The scan of blk_term is small beside the hit blocks: a query names long
// lists, whose blocks are neighbours, so few warps' shares hold most hits and
// their chains of descriptor, payload and atomics decide. 128 blocks per warp
// and step left six of eight warps of a 256-block chunk idle; 32 per step and
// the next hit's fetch under the current one's decode took 31 queries on 65,536
// terms x 2^20 ads from 850 to 244 us, 40 on 1,000 x 50,001 from 918 to 280.
template <int NW>
__global__ void __launch_bounds__(NW * 32) probe_kernel(IndexView ix, ProbeArgs a) {
    __shared__ __align__(128) uint32_t sbm[kProbeSmemWords];
    __shared__ __align__(16) uint4 stage[NW][32];
    __shared__ __align__(8) uint64_t bar;
    const uint32_t tid = threadIdx.x, lane = lane_id(), warp = warp_id();
    wait_previous();
    // the device counter also counts queries demoted past the slot capacity
    uint32_t n_probe = a.n_probe_host;
    if (a.d_n_probe && *a.d_n_probe < n_probe) n_probe = *a.d_n_probe;
    if (a.only_if && *a.only_if == 0u) return;
    if (n_probe == 0 || ix.n_blocks == 0) return;
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    uint32_t phase = 0;
    const uint64_t cb = a.chunk_blocks;
    const uint64_t n_chunks = (ix.n_blocks + cb - 1) / cb;
    for (uint64_t chunk = blockIdx.x; chunk < n_chunks; chunk += gridDim.x) {
        const uint64_t c0 = chunk * cb;
        const uint64_t c1 = c0 + cb < ix.n_blocks ? c0 + cb : ix.n_blocks;
        const uint32_t t0 = __ldg(ix.blk_term + c0), t1 = __ldg(ix.blk_term + c1 - 1);
        const uint32_t w0 = (t0 >> 5) & ~3u;
        uint32_t w1 = ((t1 >> 5) + 4u) & ~3u;
        if (w1 > a.qbm_words) w1 = a.qbm_words;
        const uint32_t span = w1 > w0 ? w1 - w0 : 0u;
        for (uint32_t g0 = 0; g0 < n_probe; g0 += kProbeGroup) {
            const uint32_t G = n_probe - g0 < kProbeGroup ? n_probe - g0 : kProbeGroup;
            const bool staged = a.staged_ok && span > 0 && (span & 3u) == 0 && span * G <= kProbeSmemWords;
            if (staged) {
                __syncthreads();  // everyone is done with the previous slice
                if (tid == 0) {
                    fence_proxy_async();
                    mbar_expect_tx(&bar, span * 4u * G);
                    for (uint32_t g = 0; g < G; ++g)
                        bulk_g2s(sbm + g * span, a.qbm + uint64_t(g0 + g) * a.qbm_stride + w0, span * 4u, &bar);
                }
                const bool ok = mbar_wait_bounded(&bar, phase, a.spin_limit);
                if (__syncthreads_or(!ok)) {
                    // one more bounded interval for the copies to land before
                    // the CTA's shared memory is released; copies still
                    // pending after it are abandoned with the error bit set
                    if (tid == 0) atomicOr(a.err, kErrTmaTimeout);
                    mbar_wait_bounded(&bar, phase, a.spin_limit);
                    return;
                }
                phase ^= 1u;
            }
            bool held = false;
            uint32_t held_q = 0;
            Fetched f{};
            auto emit = [&](const Fetched& g, uint32_t qm) {
                uint32_t id[4], cnt;
                decode_fetched(g, stage[warp], id, cnt);
                for (; qm; qm &= qm - 1u) {
                    const uint32_t slot = g0 + uint32_t(__ffs(qm)) - 1u;
                    const uint32_t o = a.out_slot ? a.out_slot[slot] : slot;
                    or_global(a.out + uint64_t(o) * a.out_stride, ix.n_ads, id, cnt);
                }
            };
            for (uint64_t base = c0 + uint64_t(warp) * 32u; base < c1; base += uint64_t(NW) * 32u) {
                const uint64_t idx = base + lane;
                const uint32_t term = idx < c1 ? __ldg(ix.blk_term + idx) : kFull;
                uint32_t hit = 0;
                if (term != kFull) {
                    const uint32_t wd = term >> 5, bit = term & 31u;
                    if (wd < a.qbm_words) {
                        for (uint32_t g = 0; g < G; ++g) {
                            const uint32_t word = staged ? sbm[g * span + (wd - w0)]
                                                         : a.qbm[uint64_t(g0 + g) * a.qbm_stride + wd];
                            hit |= ((word >> bit) & 1u) << g;
                        }
                    }
                }
                for (uint32_t lanes = __ballot_sync(kFull, hit != 0u); lanes; lanes &= lanes - 1u) {
                    const uint32_t src = __ffs(lanes) - 1u;
                    const uint32_t qm = __shfl_sync(kFull, hit, src);
                    const Fetched next = fetch_block(ix, uint32_t(base + src));
                    if (held) emit(f, held_q);
                    f = next;
                    held_q = qm;
                    held = true;
                }
            }
            if (held) emit(f, held_q);
        }
    }
}

// ---------------------------------------------------------------------------
// compaction: one pass (chunk popcount, decoupled look-back, id writes)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t masked_word(const uint32_t* bm, uint64_t w, uint64_t n_bits) {
    uint32_t v = bm[w];
    const uint64_t lo = w * 32u;
    if (lo + 32u > n_bits) v &= (n_bits > lo) ? ((1u << uint32_t(n_bits - lo)) - 1u) : 0u;
    return v;
}

__device__ __forceinline__ uint64_t ld_status(const uint64_t* p) {
    return *reinterpret_cast<const volatile unsigned long long*>(p);
}
// A status word carries its own value, and no other write of a work item is
// read by another CTA while the kernel runs, so publishing needs no fence:
// one atomic exchange at L2, where the look-back's volatile loads read it.
__device__ __forceinline__ void st_status(uint64_t* p, uint64_t v) {
    atomicExch(reinterpret_cast<unsigned long long*>(p), static_cast<unsigned long long>(v));
}

// Decoupled look-back, run by one whole warp for work item `item` whose own
// id count is `agg`: publishes the count, then reads the status words of the
// earlier items 32 at a time (lane k reads item - 1 - k of the window),
// waits until none of them is empty, and adds up the counts back to the
// nearest item that has published its inclusive prefix; publishes its own
// inclusive prefix and returns the exclusive one in *excl. Items are claimed
// in ascending order by running CTAs, each of which publishes its count
// before it looks back, so every wait ends; a wait that still sees an empty
// word after `limit` polls gives up and returns false.
__device__ bool lookback_prefix(uint64_t* status, uint64_t item, uint32_t agg, uint32_t limit, uint64_t* excl) {
    const uint32_t lane = lane_id();
    if (item == 0) {
        if (lane == 0) st_status(status, kFlagIncl | agg);
        *excl = 0;
        return true;
    }
    if (lane == 0) st_status(status + item, kFlagAgg | agg);
    uint64_t prefix = 0;
    uint64_t end = item;  // the window is items [end - 32, end)
    uint32_t spins = 0;
    for (;;) {
        const bool in_range = end > uint64_t(lane);
        const uint64_t sw = in_range ? ld_status(status + (end - 1u - lane)) : kFlagIncl;  // before item 0: 0
        if (__any_sync(kFull, (sw >> 62) == 0u)) {
            if (++spins > limit) {
                *excl = prefix;
                return false;
            }
            __nanosleep(64);
            continue;
        }
        const uint32_t incl = __ballot_sync(kFull, (sw >> 62) == 2u);
        const uint32_t upto = incl ? uint32_t(__ffs(incl)) - 1u : 31u;  // nearest inclusive word in the window
        uint64_t v = lane <= upto ? (sw & kValMask) : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
        prefix += v;
        if (incl) break;
        end -= 32u;
    }
    if (lane == 0) st_status(status + item, kFlagIncl | (prefix + agg));
    *excl = prefix;
    return true;
}

// One CTA per (bitmap, 1024-word chunk) at a time, items taken in ascending
// order from a ticket counter. Each of the 4 warps owns 8 consecutive units
// of 32 words, held in registers (lane l: word l of each unit); the chunk's
// id count is published and its output offset found by a decoupled
// look-back before the CTA starts it, and then every warp expands its units
// on its own into ascending ids (three expansions by the unit's id count,
// below). The bitmap is read once: there is no separate counting pass.
//
// U: units per warp. 8 where there are chunks for half the CTA slots of a full
// GPU; else 2 or 1, so that a single bitmap is spread over more SMs: one query
// on c0 (32 chunks of 8 units per warp, 256 of one) 9.8 -> 5.7 us, on c1 (512,
// 2,048 of two) 18 -> 16.
//
// What bounds it depends on the density. 64 bitmaps of 2^22 ads, memset and
// launch included, us and TB/s: empty 53; one bit in 64 85, 0.6; in 8 112, 1.5;
// in 4 130, 2.3; half 146, 3.9; three in four 157, 5.3; 15 in 16 189, 5.5; full
// 201, 5.5. From three in four on it is the copies' way out (5.5 TB/s at this
// size, 5.9 in the 26.9 GB of 512 queries on c1); below, the chunks' own way
// through claim, load, count and look-back (53 us for 8,192) and the expansion,
// which takes longer the fuller the words are.

// bulk copy shared -> global (TMA engine), completion tracked per thread
__device__ __forceinline__ void bulk_s2g(void* gdst, const void* ssrc, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(smem_addr(ssrc)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

constexpr uint32_t kIdBuf = 1024 + 32;  // one unit's ids plus the part of a 128-byte line before them

// Ids of one unit into dst[0 .. tot): lane l holds word l of the unit in v
// and the ids of the lower lanes' words in ex; id0 = first id of the unit +
// lane. Three expansions, by the unit's id count t:
//  * t >= kPairMin: two bits per lane -- lanes 0-15 take bits 2j, 2j+1 of
//    the even word, lanes 16-31 those of the odd word, so one pair of
//    shuffles serves two words; a lane stores at most two ids per step.
//  * t < kPairMin: each lane writes the ids of its own word, lowest bit
//    first, for as many steps as the fullest word of the unit has bits;
//    no shuffles, and a sparse unit costs steps in proportion to its bits.
//  * t == 1024 (every bit set) is handled by the caller without bit work.
// Measured on bitmaps with the per-query densities of config c1: 6 % less
// time than one lane per bit for every dense unit and a shuffle loop over
// the non-zero words for the rest, and 2x at 25 % density.
constexpr uint32_t kPairMin = 384;

__device__ __forceinline__ void st_shared(uint32_t addr, uint32_t v) {
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v));
}

// at: shared address of the first id of this lane's word
__device__ __forceinline__ void expand_pairs(uint32_t v, uint32_t at, uint32_t id0) {
    const uint32_t lane = lane_id();
    const uint32_t half = lane >> 4, j = lane & 15u;
    const uint32_t below = (1u << (2u * j)) - 1u;               // bits under this lane's pair
    uint32_t id = id0 - lane + half * 32u + 2u * j;             // id of bit 2j of word `half`
#pragma unroll 4
    for (uint32_t i = 0; i < 16u; ++i, id += 64u) {
        const uint32_t word = __shfl_sync(kFull, v, 2u * i + half);
        const uint32_t a = __shfl_sync(kFull, at, 2u * i + half) + 4u * __popc(word & below);
        const uint32_t b2 = word >> (2u * j);
        if (b2 & 1u) st_shared(a, id);
        if (b2 & 2u) st_shared(a + 4u * (b2 & 1u), id + 1u);
    }
}

__device__ __forceinline__ void expand_lane_word(uint32_t v, uint32_t at, uint32_t id0) {
    const uint32_t lane = lane_id();
    const uint32_t wb = id0 - lane + 32u * lane;  // id of bit 0 of this lane's word
    const uint32_t steps = __reduce_max_sync(kFull, uint32_t(__popc(v)));
    for (uint32_t i = 0; i < steps; ++i, at += 4u) {
        if (v) {
            st_shared(at, wb + uint32_t(__ffs(v)) - 1u);
            v &= v - 1u;
        }
    }
}

// One warp claims the next work item and makes it ready for the CTA: the
// chunk's words into buf (lane l: word 32 m + l), each warp slice's id count
// into s_wtot, the decoupled look-back's exclusive prefix into *s_prefix.
// The claim is followed at once by the loads and the count's publication, so
// later items' look-backs never wait long on it.
template <uint32_t kWarpUnits>
__device__ void prepare_chunk(const CompactArgs& a, uint64_t items, uint64_t n_words, uint32_t* buf,
                              unsigned long long* s_item, unsigned long long* s_prefix, uint32_t* s_wtot) {
    constexpr uint32_t kUnits = kWarpUnits * kCompactWarps;
    const uint32_t lane = lane_id();
    unsigned long long n = 0;
    if (lane == 0) n = atomicAdd(a.ticket, 1ull);
    n = __shfl_sync(kFull, n, 0);
    if (lane == 0) *s_item = n;
    if (n >= items) return;
    const uint32_t q = uint32_t(n / a.n_chunks);
    const uint32_t c = uint32_t(n - uint64_t(q) * a.n_chunks);
    const uint32_t* bm = a.bm + uint64_t(q) * a.stride;
    const uint64_t wbase = uint64_t(c) * (kUnits * 32u);
#pragma unroll 8
    for (uint32_t m = 0; m < kUnits; ++m) {
        const uint64_t wi = wbase + m * 32u + lane;
        if (wi + 1u < n_words) cp_async4(buf + m * 32u + lane, bm + wi);
        else buf[m * 32u + lane] = wi < n_words ? masked_word(bm, wi, a.n_bits) : 0u;
    }
    cp_async_wait_all();
    __syncwarp();
    uint32_t t = 0;
#pragma unroll
    for (uint32_t w = 0; w < kCompactWarps; ++w) {
        uint32_t cw = 0;
#pragma unroll
        for (uint32_t k = 0; k < kWarpUnits; ++k) cw += __popc(buf[(w * kWarpUnits + k) * 32u + lane]);
        cw = __reduce_add_sync(kFull, cw);
        if (lane == 0) s_wtot[w] = cw;
        t += cw;
    }
    uint64_t excl = 0;
    const bool ok = lookback_prefix(a.status, n, t, a.spin_limit, &excl);
    if (lane == 0) {
        if (!ok) atomicOr(a.err, kErrScanTimeout);
        *s_prefix = excl;
        if (a.id_offsets) {
            if (c == 0) a.id_offsets[q] = excl;
            if (n + 1 == items) a.id_offsets[a.n_q] = excl + t;
        }
        if (a.id_counts && t) atomicAdd(reinterpret_cast<unsigned long long*>(a.id_counts + q), t);
    }
}

// The CTA works on one item while the first of its warps to finish prepares
// the next one in its own id buffer (claim, loads, count, look-back), so the
// claim's round trip, the loads and the look-back overlap the other warps'
// expansion instead of stalling the whole CTA.
template <uint32_t kWarpUnits>
__global__ void __launch_bounds__(kCompactWarps * 32, 48 / kCompactWarps) compact_kernel(CompactArgs a) {
    __shared__ __align__(16) uint32_t s_buf[kCompactWarps][kIdBuf];
    __shared__ uint32_t s_wtot[kCompactWarps];
    __shared__ unsigned long long s_item, s_prefix;
    __shared__ uint32_t s_src, s_first;
    static_assert(kCompactChunkWords <= kIdBuf, "a chunk fits one id buffer");
    const uint32_t lane = lane_id(), warp = warp_id();
    uint32_t* buf = s_buf[warp];
    const uint32_t buf_addr = smem_addr(buf);
    const uint64_t n_words = (a.n_bits + 31) / 32;
    const uint64_t items = uint64_t(a.n_q) * a.n_chunks;
    wait_previous();
    if (warp == 0) prepare_chunk<kWarpUnits>(a, items, n_words, buf, &s_item, &s_prefix, s_wtot);
    if (threadIdx.x == 0) {
        s_src = 0;
        s_first = 0;
    }
    __syncthreads();
    for (;;) {
        const uint64_t item = s_item;
        if (item >= items) break;
        const uint32_t q = uint32_t(item / a.n_chunks);
        const uint32_t c = uint32_t(item - uint64_t(q) * a.n_chunks);
        const uint64_t wbase = uint64_t(c) * (kWarpUnits * 32u * kCompactWarps) + uint64_t(warp) * (kWarpUnits * 32u);
        const uint32_t* src = s_buf[s_src] + warp * (kWarpUnits * 32u);
        uint32_t v[kWarpUnits], tot[kWarpUnits];
#pragma unroll
        for (uint32_t k = 0; k < kWarpUnits; ++k) {
            v[k] = src[k * 32u + lane];
            tot[k] = __reduce_add_sync(kFull, uint32_t(__popc(v[k])));
        }
        uint64_t o0 = s_prefix + __reduce_add_sync(kFull, lane < warp ? s_wtot[lane] : 0u);
        // The warp's ids leave by bulk copies of whole 128-byte lines (2 % less
        // time on c1 than 16-byte ends per unit: 4,638 -> 4,588 us for 512
        // queries, 26.9 GB; without expanding anything the same copies take
        // 4,430, without copying the rest takes 3,780): buf holds words of the output from a line's start on, of which the first
        // `from` are not this slice's; what does not fill a line is carried to
        // the next unit in a register (lane l: word l).
        uint32_t slice = 0;
#pragma unroll
        for (uint32_t k = 0; k < kWarpUnits; ++k) slice += tot[k];
        const bool fits = o0 + slice <= a.capacity && (reinterpret_cast<uintptr_t>(a.ids) & 3u) == 0;
        uint32_t fill = (uint32_t(reinterpret_cast<uintptr_t>(a.ids) >> 2) + uint32_t(o0)) & 31u, from = fill, carry = 0;
        uint32_t* line = a.ids + o0 - fill;
        // every warp holds its words and offset: the chunk's buffer and the
        // next item's slots may be reused
        __syncthreads();
#pragma unroll 1
        for (uint32_t k = 0; k < kWarpUnits; ++k) {
            // a rolled loop keeps one copy of the expansion code (the
            // instruction cache holds it): the current unit is always in
            // v[0], the later ones move down one register per step
            const uint32_t vk = v[0], t = tot[0];
#pragma unroll
            for (uint32_t j = 0; j + 1 < kWarpUnits; ++j) {
                v[j] = v[j + 1];
                tot[j] = tot[j + 1];
            }
            if (t == 0) continue;
            const uint32_t cnt = __popc(vk);
            uint32_t x = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, x, o);
                if (lane >= uint32_t(o)) x += y;
            }
            const uint32_t ex = x - cnt;
            const uint32_t id0 = uint32_t((wbase + k * 32u) * 32u) + lane;
            if (fits) {
                if (lane == 0) bulk_wait_read_all();  // the previous unit's copy has read the buffer
                __syncwarp();
                if (lane < fill) buf[lane] = carry;
                const uint32_t end = fill + t;
                if (t == 1024u) {
                    // every bit set: buf[x] = first id of the unit + x - fill
                    const uint32_t b0 = id0 - lane - fill, m0 = (fill + 3u) / 4u;
                    uint4* b4 = reinterpret_cast<uint4*>(buf);
                    for (uint32_t m = m0 + lane; m < end / 4u; m += 32u) {
                        const uint32_t y = b0 + 4u * m;
                        b4[m] = make_uint4(y, y + 1u, y + 2u, y + 3u);
                    }
                    if (lane < 3u) {  // the words short of a vector at either end
                        const uint32_t h = fill + lane, e = (end & ~3u) + lane;
                        if (h < 4u * m0) buf[h] = b0 + h;
                        if (e < end) buf[e] = b0 + e;
                    }
                } else if (t >= kPairMin) {
                    expand_pairs(vk, buf_addr + 4u * (fill + ex), id0);
                } else {
                    expand_lane_word(vk, buf_addr + 4u * (fill + ex), id0);
                }
                fence_proxy_async();  // these shared writes before the async-proxy read
                __syncwarp();
                const uint32_t full = end & ~31u;
                if (full) {
                    const uint32_t lo = from ? 32u : 0u;
                    if (lane == 0 && full > lo) {
                        bulk_s2g(line + lo, buf + lo, (full - lo) * 4u);
                        bulk_commit();
                    }
                    if (from && lane >= from) line[lane] = buf[lane];  // the slice's first, partial line
                    from = 0;
                    line += full;
                }
                fill = end - full;
                if (lane < fill) carry = buf[full + lane];
            } else {
                // an output too short for the slice: every id is checked
                uint64_t o = o0 + ex;
                for (uint32_t m = vk; m; m &= m - 1u, ++o)
                    if (o < a.capacity) a.ids[o] = id0 - lane + 32u * lane + uint32_t(__ffs(m)) - 1u;
            }
            o0 += t;
        }
        if (fits && lane >= from && lane < fill) line[lane] = carry;  // the last, partial line
        // the first warp done prepares the next item in its own buffer
        uint32_t first = 0;
        if (lane == 0) first = atomicAdd(&s_first, 1u);
        first = __shfl_sync(kFull, first, 0);
        if (first == 0) {
            if (lane == 0) bulk_wait_read_all();  // its last copy has read the buffer
            __syncwarp();
            prepare_chunk<kWarpUnits>(a, items, n_words, buf, &s_item, &s_prefix, s_wtot);
            if (lane == 0) s_src = warp;
        }
        __syncthreads();
        if (threadIdx.x == 0) s_first = 0;
    }
    if (lane == 0) bulk_wait_all();
}

// ---------------------------------------------------------------------------
// self-test of the bounded waits
// ---------------------------------------------------------------------------
// CTA 0 arms an mbarrier for 16 bytes that no copy delivers and waits on it
// with mbar_wait_bounded; CTA 1 looks back from item 1 at status[0], which
// nothing publishes, with lookback_prefix. No asynchronous copy is ever
// issued, so nothing is in flight when the CTAs leave.
__global__ void __launch_bounds__(32) wait_selftest_kernel(uint64_t* status2, uint32_t* err, uint32_t limit) {
    __shared__ __align__(8) uint64_t bar;
    if (blockIdx.x == 0) {
        if (threadIdx.x == 0) {
            mbar_init(&bar, 1);
            fence_mbar_init();
            mbar_expect_tx(&bar, 16u);
        }
        __syncwarp();
        const bool ok = mbar_wait_bounded(&bar, 0u, limit);
        if (__any_sync(kFull, !ok) && threadIdx.x == 0) atomicOr(err, kErrTmaTimeout);
    } else {
        uint64_t excl = 0;
        const bool ok = lookback_prefix(status2, 1u, 7u, limit, &excl);
        if (!ok && threadIdx.x == 0) atomicOr(err, kErrScanTimeout);
    }
}

inline int grid_for(uint64_t items, int sm_count, uint32_t per_sm) {
    uint64_t g = uint64_t(sm_count) * (per_sm ? per_sm : 1u);
    if (items < g) g = items;
    return int(g ? g : 1);
}

}  // namespace

IndexView view_of(const abf_index* ix) {
    IndexView v;
    v.payload = reinterpret_cast<const uint4*>(ix->dev.payload);
    v.blk_first = ix->dev.blk_first;
    v.blk_last = ix->dev.blk_last;
    v.blk_desc = reinterpret_cast<const uint2*>(ix->dev.blk_desc);
    v.blk_term = ix->dev.blk_term;
    v.term_blk = ix->dev.term_blk;
    v.term_len = ix->dev.term_len;
    v.term_dense = ix->dev.term_dense;
    v.dense = ix->dev.dense;
    v.term_dir = ix->dev.term_dir;
    v.dir = ix->dev.dir;
    v.term_feat = ix->dev.term_feat;
    v.term_plain = ix->dev.term_plain;
    v.term_info = reinterpret_cast<const uint4*>(ix->dev.term_info);
    v.plain = ix->dev.plain;
    v.plain_dir = ix->dev.plain_dir;
    v.plain_dir_n = ix->derived.plain_dir_n;
    v.n_plain = ix->dev.plain ? ix->derived.n_plain() : 0u;
    v.dense_stride = ix->derived.dense_stride;
    v.dir_n = ix->derived.dir_n;
    v.n_dense = ix->derived.n_dense;
    v.n_terms = ix->n_terms;
    v.n_ads = ix->n_ads;
    v.n_blocks = ix->n_blocks;
    return v;
}

uint32_t compact_chunks(uint64_t n_bits, uint32_t units) {
    const uint64_t n_words = (n_bits + 31) / 32, chunk = units * 32u * kCompactWarps;
    return uint32_t((n_words + chunk - 1) / chunk);
}

uint32_t compact_units(uint64_t n_q, uint64_t n_bits) {
    if (n_q * compact_chunks(n_bits, 8) >= kCompactFew) return 8;
    return n_q * compact_chunks(n_bits, 2) >= kCompactFew ? 2 : 1;
}

cudaError_t launch_plan(const IndexView& v, const PlanArgs& a, cudaStream_t s) {
    if (a.n_q == 0) return cudaSuccess;
    // with a device count the bound may be far above it: a few waves of CTAs
    const uint32_t most = a.d_n_q ? 148u * 16u : 65535u * 16u;
    count_launch();
    const uint32_t grid = a.n_q < most ? a.n_q : most;
    auto with = [&](auto given) {
        if (a.n_inline > sizeof(given.t) / 4u) return cudaErrorInvalidValue;
        given.n = a.n_inline;
        std::memcpy(given.t, a.inline_terms, a.n_inline * 4u);
        return launch_after(plan_kernel<sizeof(given.t) / 4u>, grid, 256, 0, s, v, a, given);
    };
    if (!a.inline_terms) return launch_after(plan_kernel<0>, grid, 256, 0, s, v, a, InlineTerms<0>{});
    return a.n_inline <= kInlineSmall ? with(InlineTerms<kInlineSmall>()) : with(InlineTerms<kInlineLarge>());
}

cudaError_t launch_queue_scan(const QueueArgs& a, cudaStream_t s) {
    count_launch();
    return launch_after(queue_scan_kernel, 1, 1024, 0, s, a);
}

cudaError_t launch_key_runs(const KeyRunsArgs& a, cudaStream_t s) {
    count_launch();
    return launch_after(key_runs_kernel, 1, 1024, 0, s, a);
}

cudaError_t launch_term_lists(const TermListArgs& a, cudaStream_t s) {
    if (a.n_q == 0) return cudaSuccess;
    count_launch(2);
    const cudaError_t e = launch_after(term_count_kernel, a.n_q, kTermThreads, 0, s, a);
    return e != cudaSuccess ? e : launch_after(term_list_kernel, a.n_q, kTermThreads, 0, s, a);
}

template <int W, int NW, bool ACC>
static cudaError_t tile_launch(const IndexView& v, const TileArgs& a, int grid, cudaStream_t s) {
    constexpr int smem = W * 4;
    if (smem > 48 * 1024) {
        // opt in to more than 48 KB of dynamic shared memory, once per device
        // (so that later launches, also under stream capture, make no
        // host-side attribute call)
        static std::atomic<uint64_t> done{0};
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const uint64_t bit = 1ull << (dev & 63);
        if (!(done.load() & bit)) {
            e = cudaFuncSetAttribute(tile_union_kernel<W, NW, ACC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
            if (e != cudaSuccess) return e;
            done.fetch_or(bit);
        }
    }
    return launch_after(tile_union_kernel<W, NW, ACC>, uint32_t(grid), NW * 32, smem, s, v, a);
}

template <int W>
static cudaError_t tile_dispatch_w(const IndexView& v, const TileArgs& a, uint32_t nw, int grid, cudaStream_t s) {
    switch (nw) {
        case 1: return a.accumulate ? tile_launch<W, 1, true>(v, a, grid, s) : tile_launch<W, 1, false>(v, a, grid, s);
        case 2: return a.accumulate ? tile_launch<W, 2, true>(v, a, grid, s) : tile_launch<W, 2, false>(v, a, grid, s);
        case 4: return a.accumulate ? tile_launch<W, 4, true>(v, a, grid, s) : tile_launch<W, 4, false>(v, a, grid, s);
        default: return a.accumulate ? tile_launch<W, 8, true>(v, a, grid, s) : tile_launch<W, 8, false>(v, a, grid, s);
    }
}

namespace {
template <typename V, bool ACC>
cudaError_t stream_launch(const IndexView& v, const DenseStreamArgs& a, int sm_count, cudaStream_t s) {
    const uint64_t cols = (a.n_words + sizeof(V) / 4u - 1u) / (sizeof(V) / 4u);
    const uint64_t items = (cols + kStreamThreads - 1u) / kStreamThreads * a.n_q;
    return launch_after(dense_stream_kernel<V, ACC>, uint32_t(grid_for(items, sm_count, 64)), kStreamThreads, 0, s, v, a);
}
}  // namespace

cudaError_t launch_dense_stream(const IndexView& v, const DenseStreamArgs& a, int sm_count, cudaStream_t s) {
    if (a.n_q == 0 || a.n_words == 0) return cudaSuccess;
    count_launch();
    if (a.vec_ok)
        return a.accumulate ? stream_launch<uint4, true>(v, a, sm_count, s) : stream_launch<uint4, false>(v, a, sm_count, s);
    return a.accumulate ? stream_launch<uint32_t, true>(v, a, sm_count, s) : stream_launch<uint32_t, false>(v, a, sm_count, s);
}

cudaError_t launch_tile_union(const IndexView& v, const TileArgs& a, const abf_tuning& t, int sm_count,
                              cudaStream_t s) {
    const uint64_t items = uint64_t(a.n_q) * a.n_tiles;
    if (items == 0) return cudaSuccess;
    const uint32_t nw = t.warps_per_tile ? t.warps_per_tile : 8u;
    // ctas_per_sm counts 8-warp CTAs; narrower CTAs are packed proportionally
    const uint32_t per_sm = (t.ctas_per_sm ? t.ctas_per_sm : 2u) * (nw >= 8u ? 1u : 8u / nw);
    const int grid = grid_for(items, sm_count, per_sm);
    cudaError_t e;
    switch (t.tile_words) {
        case 256: e = tile_dispatch_w<256>(v, a, nw, grid, s); break;
        case 512: e = tile_dispatch_w<512>(v, a, nw, grid, s); break;
        case 2048: e = tile_dispatch_w<2048>(v, a, nw, grid, s); break;
        case 4096: e = tile_dispatch_w<4096>(v, a, nw, grid, s); break;
        case 8192: e = tile_dispatch_w<8192>(v, a, nw, grid, s); break;
        case 16384: e = tile_dispatch_w<16384>(v, a, nw, grid, s); break;
        default: e = tile_dispatch_w<1024>(v, a, nw, grid, s); break;
    }
    count_launch();
    return e;
}

namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encoder() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return EncodeTiledFn(nullptr);
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}
}  // namespace

cudaError_t encode_dense_tmap(const IndexView& v, uint32_t gw, void* out) {
    static_assert(sizeof(CUtensorMap) == 128, "tensor map size");
    EncodeTiledFn fn = encoder();
    if (!fn || !v.dense || v.n_dense == 0 || (gw != 32u && gw != 64u)) return cudaErrorNotSupported;
    // dims: words of a bitmap (innermost), bitmaps; rows past n_dense read as
    // zeros. Two descriptors: boxes of 256 bitmaps, and one box for the rest
    // plus the zero row, so a stage holds exactly n_dense + 1 rows.
    const uint32_t rows = v.n_dense + 1u;
    const uint32_t last = rows - (rows - 1u) / kGroupBoxRows * kGroupBoxRows;
    const cuuint64_t dims[2] = {cuuint64_t(v.dense_stride), cuuint64_t(v.n_dense)};
    const cuuint64_t strides[1] = {cuuint64_t(v.dense_stride) * 4u};
    const cuuint32_t es[2] = {1, 1};
    for (int k = 0; k < 2; ++k) {
        const cuuint32_t box[2] = {gw, k == 0 ? kGroupBoxRows : last};
        const CUresult r = fn(reinterpret_cast<CUtensorMap*>(out) + k, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2,
                              const_cast<uint32_t*>(v.dense), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    }
    return cudaSuccess;
}

uint32_t dense_group_list_cap(uint32_t n_rows, uint32_t n_q, uint32_t gw, uint32_t stages) {
    const uint64_t stage = (uint64_t(n_rows) * gw * 4u + 1023u) & ~1023ull;
    const uint64_t used = 1024u + stages * stage + ((6ull * n_q + 15u) & ~15ull);
    return used >= kGroupSmemBytes ? 0u : uint32_t((kGroupSmemBytes - used) / 2u) & ~7u;
}

namespace {
template <uint32_t GW, bool ACC>
cudaError_t launch_group_w(const CUtensorMap (&m)[2], const DenseGroupArgs& a, int sm_count, cudaStream_t s) {
    static std::atomic<uint64_t> done{0};  // devices whose attribute is set
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (!(done.load() >> dev & 1ull)) {
        e = cudaFuncSetAttribute(dense_group_kernel<GW, ACC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 int(kGroupSmemBytes));
        if (e != cudaSuccess) return e;
        done.fetch_or(1ull << dev);
    }
    const uint32_t grid = a.n_tiles < uint32_t(sm_count) ? a.n_tiles : uint32_t(sm_count);
    return launch_after(dense_group_kernel<GW, ACC>, grid, kGroupThreads, kGroupSmemBytes, s, m[0], m[1], a);
}
}  // namespace

cudaError_t launch_dense_group(const void* tmaps, uint32_t gw, const DenseGroupArgs& a, int sm_count,
                               cudaStream_t s) {
    if (a.n_q == 0 || a.n_tiles == 0) return cudaSuccess;
    if (a.n_rows < 2 || a.n_rows > kGroupMaxBoxes * kGroupBoxRows || a.n_q > kGroupMaxQueries)
        return cudaErrorInvalidValue;
    const uint64_t stage = (uint64_t(a.n_rows) * gw * 4u + 1023u) & ~1023ull;
    if ((a.stages != 1u && a.stages != 2u) ||
        1024u + a.stages * stage + ((6ull * a.n_q + 15u) & ~15ull) > kGroupSmemBytes)
        return cudaErrorInvalidValue;
    CUtensorMap m[2];
    std::memcpy(m, tmaps, sizeof(m));
    cudaError_t e;
    if (gw == 64u) e = a.accumulate ? launch_group_w<64, true>(m, a, sm_count, s) : launch_group_w<64, false>(m, a, sm_count, s);
    else if (gw == 32u) e = a.accumulate ? launch_group_w<32, true>(m, a, sm_count, s) : launch_group_w<32, false>(m, a, sm_count, s);
    else return cudaErrorInvalidValue;
    count_launch();
    return e;
}

cudaError_t launch_scatter(const IndexView& v, const ScatterArgs& a, const abf_tuning& t, int sm_count,
                           cudaStream_t s) {
    if (a.n_q == 0) return cudaSuccess;
    // one wave of resident CTAs (6 of 8 warps per SM) at most
    const int grid = grid_for(~0ull, sm_count, std::min<uint32_t>(t.ctas_per_sm ? t.ctas_per_sm * 2u : 6u, 6u));
    count_launch();
    return launch_after(a.key_slot ? scatter_kernel<8, true> : scatter_kernel<8, false>, uint32_t(grid), 256, 0, s, v, a);
}

namespace {
template <bool ACC>
cudaError_t launch_bin_acc(const IndexView& v, const BinArgs& a, int sm_count, cudaStream_t s) {
    static std::atomic<uint64_t> done{0};  // devices whose attribute is set
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (!(done.load() >> (dev & 63) & 1ull)) {
        e = cudaFuncSetAttribute(bin_kernel<ACC>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBinWords * 4u));
        if (e != cudaSuccess) return e;
        done.fetch_or(1ull << (dev & 63));
    }
    return launch_after(bin_kernel<ACC>, uint32_t(sm_count) * kBinCtasPerSm, kBinThreads, kBinWords * 4u, s, v, a);
}
}  // namespace

cudaError_t launch_term_info(const IndexView& v, uint4* info, TermFeat* feat, const uint32_t* cbytes, int sm_count,
                             cudaStream_t s) {
    term_info_kernel<<<sm_count * 8, 256, 0, s>>>(v, info, feat, cbytes);
    count_launch();
    return cudaGetLastError();
}

cudaError_t launch_plain_ids(const IndexView& v, const uint32_t* plain_term, const uint32_t* plain_off, uint32_t* plain,
                             uint32_t* plain_dir, int sm_count, cudaStream_t s) {
    if (v.n_plain == 0) return cudaSuccess;
    plain_ids_kernel<<<sm_count * 8, 256, 0, s>>>(v, plain_off, plain);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    plain_dir_kernel<<<sm_count * 8, 256, 0, s>>>(v, plain_term, plain_off, plain_dir);
    count_launch(2);
    return cudaGetLastError();
}

cudaError_t launch_bin(const IndexView& v, const BinArgs& a, int sm_count, cudaStream_t s) {
    if (a.n_q == 0 || a.n_tiles == 0) return cudaSuccess;
    const cudaError_t e = a.accumulate ? launch_bin_acc<true>(v, a, sm_count, s) : launch_bin_acc<false>(v, a, sm_count, s);
    count_launch();
    return e;
}

cudaError_t launch_probe(const IndexView& v, const ProbeArgs& a, const abf_tuning& t, int sm_count, cudaStream_t s) {
    if (v.n_blocks == 0) return cudaSuccess;
    const uint64_t n_chunks = (v.n_blocks + a.chunk_blocks - 1) / a.chunk_blocks;
    const int grid = grid_for(n_chunks, sm_count, t.ctas_per_sm ? t.ctas_per_sm : 4u);
    count_launch();
    return launch_after(probe_kernel<8>, uint32_t(grid), 256, 0, s, v, a);
}

cudaError_t launch_compact(const CompactArgs& a, int sm_count, uint32_t ctas_per_sm, cudaStream_t s) {
    const uint64_t items = uint64_t(a.n_q) * a.n_chunks;
    if (items == 0) return cudaSuccess;
    if (!a.zeroed) {
        // the ticket beside the look-back words saves a memset
        const bool both = static_cast<void*>(a.ticket + 1) == static_cast<void*>(a.status);
        cudaError_t e = cudaMemsetAsync(both ? static_cast<void*>(a.ticket) : a.status, 0, (items + both) * sizeof(uint64_t), s);
        if (e == cudaSuccess && !both) e = cudaMemsetAsync(a.ticket, 0, sizeof(unsigned long long), s);
        if (e == cudaSuccess && a.id_counts) e = cudaMemsetAsync(a.id_counts, 0, uint64_t(a.n_q) * sizeof(uint64_t), s);
        if (e != cudaSuccess) return e;
    }
    // ctas_per_sm counts CTAs of 8 warps: the same resident warps whatever the CTA size
    const uint32_t per_sm = (ctas_per_sm ? ctas_per_sm : 6u) * 8u / kCompactWarps;
    count_launch();
    const auto kernel = a.units == 8u ? compact_kernel<8> : a.units == 2u ? compact_kernel<2> : compact_kernel<1>;
    return launch_after(kernel, uint32_t(grid_for(items, sm_count, per_sm)), kCompactWarps * 32, 0, s, a);
}

cudaError_t launch_wait_selftest(uint64_t* status2, uint32_t* err, uint32_t spin_limit, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(status2, 0, 2 * sizeof(uint64_t), s);
    if (e != cudaSuccess) return e;
    wait_selftest_kernel<<<2, 32, 0, s>>>(status2, err, spin_limit);
    count_launch();
    return cudaGetLastError();
}

}  // namespace abf
