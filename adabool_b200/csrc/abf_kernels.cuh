// Kernel argument blocks and launchers of libadabool (sm_100a).
//
// Kernels (all integer, HBM/L2 bound):
//   plan_kernel        per query: resolve the path (given, the learned
//                      planner's inline, or the fixed rule), split lists into
//                      merged (long) and scattered (short), prefix the short
//                      lists' block counts, claim a bitmap-probe slot and
//                      write the probe query's term bitmap
//   queue_scan_kernel  exclusive scan of the per-query scattered block counts
//   dense_stream_kernel  list-union, dense bitmaps of small batches: every
//                      thread ORs one 16-byte column of a query's rows
//   dense_group_kernel list-union, dense bitmaps of large batches: every row
//                      staged once per tile, ORed per query in shared memory
//   tile_union_kernel  list-union, merge variant: one CTA owns a tile of one
//                      query's output bitmap in shared memory, decodes every
//                      block of the long lists without dense bitmaps that
//                      overlaps the tile and ORs with shared-memory atomics
//   scatter_kernel     list-union, scatter variant: load-balanced warps decode
//                      the short lists' blocks and OR into the global bitmap
//                      with lane-combined atomicOr
//   bin_kernel         list-union, binned variant: the mid-length lists of large
//                      batches, from plain ids, per 16,384-word tile in shared
//                      memory
//   plain_ids / plain_dir_kernel  the plain ids, when an index is uploaded
//   probe_kernel       bitmap-probe: scans every block of the index, stages
//                      the probe queries' term-bitmap slices in shared memory
//                      with bulk async copies (TMA engine), tests each block's
//                      term and scatters hit blocks into their queries
//   term_count / term_list_kernel  query term bitmaps -> term lists, for the
//                      bitmap-probe operators (the list-union kernels then
//                      merge them; the scan answers what does not fit)
//   key_runs_kernel    runs of consecutive keys with one output bitmap
//   compact_kernel     compaction: bitmap -> ascending uint32 ids in one pass
//                      (chunk popcounts, decoupled look-back prefix, id
//                      writes)
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include "abf_internal.h"

namespace abf {

constexpr uint32_t kNoHeavy = 0xffffffffu;   // heavy_min meaning "merge no list"
constexpr uint32_t kDenseOnly = 0xfffffffeu; // heavy_min meaning "merge only the dense-bitmap lists"
// warps per compaction CTA; a chunk (256 words per warp) fits one warp's id
// buffer, where the warp that prepares it stages it
constexpr uint32_t kCompactWarps = 4;
constexpr uint32_t kCompactChunkWords = kCompactWarps * 256;  // bitmap words per compaction work item
constexpr uint32_t kCompactFew = 888;  // fewer items than this (6 per SM): shorter chunks
// look-back words that a batch with shorter chunks can need: less than
// kCompactFew items turn into at most eight times as many
constexpr uint32_t kCompactFewStatus = 8u * kCompactFew;
constexpr uint32_t kProbeGroup = 32;          // probe queries tested per pass

// device error codes (workspace flag)
constexpr uint32_t kErrScanTimeout = 1u;
constexpr uint32_t kErrTmaTimeout = 2u;
constexpr uint32_t kErrTermRange = 4u;

// Polls of a bounded device wait (look-back status word, mbarrier) before it
// gives up, sets its error bit and returns. A look-back poll sleeps ~64 ns,
// an mbarrier poll is one try_wait (which itself suspends for a
// hardware-defined interval), so the default allows well over a second.
constexpr uint32_t kDefaultSpinLimit = 1u << 22;

struct QueueArgs {
    const uint64_t* q_light_cnt;
    uint64_t* q_light_pref;   // n_q + 1
    uint32_t n_q;
    const uint32_t* d_n_q;    // optional device count of queries (at most n_q)
    // optional (q_bblk): the bin kernel's work split, see BinArgs
    const uint32_t* q_bblk;
    const uint32_t* q_nbin;
    uint32_t* parts_pref;     // out: n_q + 1
    uint32_t* ticket;         // out: zeroed
    uint32_t n_tiles;
    uint32_t slots;           // CTAs of the bin kernel that run at a time
    // optional: where this word is set (or the plan kernel says so), the
    // queries' term slots overlap and nothing of them may be followed: no
    // blocks, parts, listed or dense lists
    const uint32_t* overlap;
    uint32_t* n_tile_list;
    uint32_t* q_ndense;
};

// Terms of a single query given to the plan kernel with its arguments: no
// upload, no staging buffer to wait for (one query on c0 28.7 -> 24.2 us). Two sizes, as a launch copies them
// whole; with the other arguments the larger one stays below 4 KB.
constexpr uint32_t kInlineSmall = 112, kInlineLarge = 800;
template <uint32_t N>
struct InlineTerms {
    uint32_t n;
    uint32_t t[N];
};
template <>
struct InlineTerms<0> {};

// queries whose scan the plan kernel's last CTA runs: in steps of 256, a step
// costs it ~0.6 us, a launch of the scan kernel ~3 us
constexpr uint32_t kScanInPlan = 2048;

struct PlanArgs {
    // with inline terms (n_q 1): the CTA writes them and their offsets here
    // first, and zeroes the batch's counters at ctl (ctl_words)
    const uint32_t* inline_terms;  // host pointer, read at launch; null: terms and q_off are filled
    uint32_t n_inline;
    uint32_t* ctl;
    uint32_t ctl_words;
    const uint32_t* terms;
    const uint64_t* q_off;
    uint32_t n_q;
    const uint8_t* paths;     // per-query abf_path or null
    uint32_t path_uniform;    // abf_path when paths is null
    uint32_t hybrid_min;      // HYBRID merge threshold (postings)
    const float* planner;     // installed planner parameters (ABF_PLANNER_PARAMS) or null: with
                              // them, ABF_PATH_AUTO queries take the MLP's choice
    uint64_t n_postings;      // index postings (a planner feature)
    float probe_min_frac;     // fixed rule: probe when touched blocks / all blocks > this
    uint32_t fixed_hybrid_min;  // fixed rule otherwise: HYBRID when a list has >= this many
                                // postings (0: never), else UNION
    uint2* term_slot;         // out: per term slot, exclusive prefix (in its query) of scattered blocks
                              // and the list's first block
    uint64_t* q_light_cnt;    // out: per query scattered blocks
    uint32_t* probe_list;     // out: probe slot -> query
    uint32_t* n_probe;        // in/out: zeroed before launch
    uint32_t probe_cap;
    uint32_t* probe_bm;       // optional: probe slot s's term bitmap at probe_bm + s * probe_stride
    uint64_t probe_stride;    // words; written (zeroed, then the query's terms) by the query's CTA
    uint8_t* path_out;        // out (optional): resolved path per query
    uint64_t max_terms;       // term slots of the scratch arrays; queries past it get no work
    uint32_t* err;            // device error flag (optional)
    uint32_t* overlap;        // out (optional, without `done`, zeroed before launch): set when a query ends before
                              // it begins and others follow, so that theirs may be slots of earlier ones
    // optional: queries that (also) merge lists without dense bitmaps, in any
    // order; n_tile_list is zeroed before launch
    uint32_t* tile_list;
    uint32_t* n_tile_list;
    int dense_in_tile;        // 1: dense-bitmap lists go to the merge kernel, 0: scattered too
    uint32_t* tile_cls;       // out: per term slot, what the merge kernel does with it
                              // (kNone: nothing, else the term)
    // optional per-query dense-bitmap lists (all three set, or q_dense16 null):
    // the query's distinct dense bitmap indices in ascending order, as 16-bit
    // values from q_dense16 + q_dstart[q] (16-byte aligned), padded to a
    // multiple of 8 with the index n_dense (an all-zero row for the TMA path)
    uint16_t* q_dense16;      // out: max_terms + 8 * n_q + 16 entries
    uint32_t dense_shift;     // entries are index << this (the group kernel's row word offsets: 6 or 5)
    uint32_t* q_dstart;       // out: per query
    uint32_t* q_ndense;       // out: per query, distinct dense bitmaps
    const uint32_t* d_n_q;    // optional device count of queries (at most n_q)
    // optional binning (bin_list set): lists with plain ids go to the bin
    // kernel in queries where they hold at least bin_min_blocks blocks in all,
    // and else those that the path merges (HYBRID, TILE)
    uint32_t* bin_list;       // out: from slot q_off[q] on, their plain list indices
    uint32_t* q_nbin;         // out: per query, such lists
    uint32_t* q_bblk;         // out: per query, their blocks
    uint32_t bin_min_blocks;
    // optional: what later kernels of the batch find zeroed, per query
    uint32_t* sat;            // sat_stride words of saturation marks
    uint32_t sat_stride;
    uint64_t* status;         // n_chunks compaction look-back words
    uint32_t n_chunks;
    uint64_t* id_counts;
    // optional: the CTA that finishes last runs the scan over the queries
    uint32_t* done;           // CTAs finished: zero before the launch, and again when it ends
    QueueArgs queue;
    const uint32_t* mixed_from;  // optional device word: queries from this one on have keys of several
                              // output bitmaps, and bin none
    uint32_t no_dense_from;   // queries from this one on scatter their dense-bitmap lists too
                              // (0: none do; only with dense_in_tile)
};

// Consecutive keys with the same bitmap index form one run, which the kernels
// above then treat as a query. Of keys in no order (fewer than eight per run),
// those past the first `cap` runs are cut into chunks of kKeyChunk instead,
// whatever their bitmaps.
constexpr uint32_t kKeyChunk = 1024;  // keys that a planning CTA takes in one step
struct KeyRunsArgs {
    const uint32_t* qidx;
    uint32_t n_keys;
    uint32_t cap;
    uint64_t* off;            // out: first key of each run or chunk, then n_keys (n_keys + 1 entries)
    uint32_t* slot;           // out: the run's bitmap index
    uint32_t* n_runs;         // out: runs and chunks, and the first chunk (kNone: none)
};

// Term bitmaps -> term lists (ascending), one list per bitmap, packed.
struct TermListArgs {
    const uint32_t* qbm;      // qbm_stride words apart
    uint64_t qbm_stride;
    uint32_t qbm_words;       // readable words per bitmap
    uint32_t n_q;
    uint32_t n_terms;         // bits at and past it are ignored
    uint32_t cap;             // room in terms; if the lists do not fit, all come out empty and *overflow is 1
    uint32_t* cnt;            // scratch: n_q
    uint32_t* terms;          // out
    uint64_t* off;            // out: n_q + 1
    uint32_t* overflow;       // out: 0 or 1
    uint32_t* zero;           // n_zero (< 512) counters that the next kernels find zeroed
    uint32_t n_zero;
    uint32_t* err;            // optional error flag, set to err_value
    uint32_t err_value;
};

struct TileArgs {
    const uint32_t* tile_cls;  // per term slot, from the plan kernel
    const uint64_t* q_off;
    uint32_t n_q;              // most queries that can be listed
    uint32_t n_tiles;
    uint32_t* out;             // holds the queries' dense bitmaps' OR already
    uint64_t out_stride;      // words between query bitmaps
    uint64_t n_words;         // words of one bitmap
    int accumulate;           // 1: OR into the existing bitmap with atomics, 0: load, add, store
    int vec_ok;               // out 16-byte aligned and out_stride % 4 == 0
    const uint32_t* tile_list;  // the plan kernel's list of the queries to visit, and its length
    const uint32_t* n_tile_list;
};

// dense stream kernel: the dense bitmaps of every query, for small batches
struct DenseStreamArgs {
    const uint16_t* q_dense16;
    const uint32_t* q_dstart;
    const uint32_t* q_ndense;
    uint32_t n_q;
    uint32_t* out;
    uint64_t out_stride;
    uint64_t n_words;
    int accumulate;            // 1: OR into the output with atomics, 0: overwrite
    int vec_ok;                // out 16-byte aligned and out_stride % 4 == 0
    uint32_t* sat;             // optional, zeroed: marks of all-ones tiles-of-64 (only with vec_ok)
    uint32_t sat_stride;
};

// dense group kernel: one pass per 32- or 64-word tile over all queries
constexpr uint32_t kGroupBoxRows = 256;   // dense bitmaps per TMA box
constexpr uint32_t kGroupMaxBoxes = 3;    // up to 767 dense bitmaps plus the zero row
constexpr uint32_t kGroupMaxQueries = 2048;
constexpr uint32_t kGroupSmemBytes = 226u * 1024u;  // dynamic shared memory of the group kernel

struct DenseGroupArgs {
    const uint16_t* q_dense16;
    const uint32_t* q_dstart;
    const uint32_t* q_ndense;
    uint32_t n_q;              // <= kGroupMaxQueries
    uint32_t n_rows;           // n_dense + 1 (the last row reads as zeros)
    uint32_t list_cap;         // list entries (16-bit row word offsets) that fit in shared memory
    uint32_t stages;           // 2: double-buffered tile copies; 1: one stage, refilled after each tile
    uint32_t n_tiles;          // ceil(n_words / tile words)
    uint32_t* out;
    uint64_t out_stride;
    uint64_t n_words;
    uint32_t* err;
    uint32_t spin_limit;       // polls of an mbarrier wait before it gives up
    uint32_t* sat;             // optional, zeroed before launch: bit t of query q's sat_stride words
    uint32_t sat_stride;       //   is set when tile t of its bitmap came out all ones
    const uint32_t* d_n_q;     // optional device count of queries (at most n_q)
    int accumulate;            // 1: OR into the output with atomics (bitmaps may be shared), 0: overwrite
    const uint32_t* out_slot;  // query -> output bitmap index (null: identity)
};

// bin kernel: tiles of kBinWords words
constexpr uint32_t kBinWords = (1u << kBinShift) / 32u;
constexpr uint32_t kBinThreads = 512;
constexpr uint32_t kBinCtasPerSm = 3;
struct BinArgs {
    const uint32_t* bin_list;  // per query: plain list indices, from slot q_off[q] on
    const uint64_t* q_off;
    const uint32_t* q_nbin;
    const uint32_t* parts_pref;  // exclusive prefix (n_q + 1) of the parts that each query's lists are cut into
    uint32_t* ticket;          // item counter, zero
    uint32_t n_q;
    const uint32_t* d_n_q;     // optional device count of queries (at most n_q)
    uint32_t n_tiles;
    uint32_t* out;
    uint64_t out_stride;
    const uint32_t* out_slot;  // query -> output bitmap index (null: identity)
    uint64_t n_words;
    int accumulate;            // 1: bitmaps may be shared, OR with atomics always
    int vec_ok;                // out 16-byte aligned and out_stride % 4 == 0
    const uint32_t* sat;       // the dense group kernel's marks (see ScatterArgs)
    uint32_t sat_stride;
    uint32_t sat_shift;
    uint32_t sat_last;
};

struct ScatterArgs {
    const uint64_t* q_off;
    const uint2* term_slot;
    const uint64_t* q_light_pref; // n_q + 1
    uint32_t n_q;
    const uint32_t* out_slot;  // query -> output bitmap index (null: identity)
    const uint32_t* key_slot;  // instead: term slot -> output bitmap index
    uint32_t* out;
    uint64_t out_stride;
    uint32_t chunk_blocks;     // consecutive blocks a warp takes at a time (at most 32)
    const uint32_t* sat;       // optional: the dense group kernel's saturated-tile bits
    uint32_t sat_stride;       //   (words per query); an OR into a word of such a tile
    uint32_t sat_shift;        //   is skipped; tile = word >> sat_shift
    uint32_t sat_last;         // queries past this one share its row of marks (all zero then: no marks)
    const uint32_t* d_n_q;     // optional device count of queries (at most n_q)
};

struct ProbeArgs {
    const uint32_t* qbm;       // probe term bitmaps, qbm_stride words apart
    uint64_t qbm_stride;
    uint32_t qbm_words;        // readable words per bitmap
    int staged_ok;             // qbm 16-byte aligned and stride % 4 == 0
    const uint32_t* d_n_probe; // device count, clamped to n_probe_host (null: n_probe_host)
    uint32_t n_probe_host;     // probe bitmaps available
    const uint32_t* out_slot;  // probe slot -> output bitmap index (null: identity)
    uint32_t* out;
    uint64_t out_stride;
    uint32_t chunk_blocks;     // multiple of 128
    uint32_t* err;
    uint32_t spin_limit;       // polls of an mbarrier wait before it gives up
    const uint32_t* only_if;   // optional: the kernel does nothing while this device word is 0
};

// Compaction of n_q bitmaps into one packed id array. Work item i is chunk
// i % n_chunks of bitmap i / n_chunks; items are claimed in ascending order
// from a ticket counter, and each publishes its id count in status[i] so
// that later items find their output offset by looking back.
struct CompactArgs {
    const uint32_t* bm;
    uint64_t stride;           // words between bitmaps
    uint32_t n_q;
    uint64_t n_bits;           // ids >= n_bits are dropped
    uint32_t n_chunks;         // per bitmap
    uint32_t units;            // 32-word units per warp of a chunk (8, 2 or 1; see compact_units)
    uint64_t* status;          // n_q * n_chunks look-back words, zeroed before launch
    unsigned long long* ticket;  // item counter, zeroed before launch
    uint32_t* ids;
    uint64_t capacity;
    uint64_t* id_offsets;      // optional n_q + 1
    uint64_t* id_counts;       // optional n_q, accumulated (zeroed before launch)
    uint32_t* err;
    uint32_t spin_limit;       // polls of a look-back wait before it gives up
    int zeroed;                // status, ticket and id_counts are zero already
};

IndexView view_of(const abf_index* ix);
uint32_t compact_chunks(uint64_t n_bits, uint32_t units = 8);
uint32_t compact_units(uint64_t n_q, uint64_t n_bits);

cudaError_t launch_plan(const IndexView& v, const PlanArgs& a, cudaStream_t s);
// two 2-D TMA descriptors (2 x 128 bytes into out) of the dense bitmaps:
// gw-word (32 or 64) x 256-bitmap boxes, and one box for the remaining
// bitmaps plus the zero row; cudaErrorNotSupported when the driver has no
// encoder
cudaError_t encode_dense_tmap(const IndexView& v, uint32_t gw, void* out);
// list entries (16-bit row word offsets) the group kernel can stage in shared
// memory with gw-word tiles and `stages` stages (0: the stages do not fit)
uint32_t dense_group_list_cap(uint32_t n_rows, uint32_t n_q, uint32_t gw, uint32_t stages);
cudaError_t launch_dense_group(const void* tmaps, uint32_t gw, const DenseGroupArgs& a, int sm_count,
                               cudaStream_t s);
cudaError_t launch_dense_stream(const IndexView& v, const DenseStreamArgs& a, int sm_count, cudaStream_t s);
cudaError_t launch_queue_scan(const QueueArgs& a, cudaStream_t s);
cudaError_t launch_key_runs(const KeyRunsArgs& a, cudaStream_t s);
cudaError_t launch_term_lists(const TermListArgs& a, cudaStream_t s);
cudaError_t launch_tile_union(const IndexView& v, const TileArgs& a, const abf_tuning& t, int sm_count,
                              cudaStream_t s);
cudaError_t launch_scatter(const IndexView& v, const ScatterArgs& a, const abf_tuning& t, int sm_count,
                           cudaStream_t s);
cudaError_t launch_term_info(const IndexView& v, uint4* info, TermFeat* feat, const uint32_t* cbytes, int sm_count,
                             cudaStream_t s);
// ids and positions of the plain lists (IndexView::plain, plain_dir) from the blocks
cudaError_t launch_plain_ids(const IndexView& v, const uint32_t* plain_term, const uint32_t* plain_off, uint32_t* plain,
                             uint32_t* plain_dir, int sm_count, cudaStream_t s);
cudaError_t launch_bin(const IndexView& v, const BinArgs& a, int sm_count, cudaStream_t s);
cudaError_t launch_probe(const IndexView& v, const ProbeArgs& a, const abf_tuning& t, int sm_count,
                         cudaStream_t s);
// planner (abf_planner.cu)
cudaError_t launch_planner(const IndexView& v, const float* params, const uint32_t* terms, const uint64_t* q_off,
                           uint32_t n_q, uint32_t hybrid_min, uint64_t n_postings, float* feat, float* pred,
                           uint8_t* paths, cudaStream_t s);
cudaError_t launch_mlp_forward(const float* p, const float* x, uint32_t n, float* y, cudaStream_t s);
cudaError_t launch_mlp_grad(const float* p, const float* x, const float* t, const float* mask, uint32_t n, float* g,
                            float* loss2, cudaStream_t s);
cudaError_t launch_adam(float* p, const float* g, float* m, float* v, uint32_t step, float lr, float b1, float b2,
                        float eps, cudaStream_t s);

// clears status / ticket / id_counts on the stream, then one compaction launch
cudaError_t launch_compact(const CompactArgs& a, int sm_count, uint32_t ctas_per_sm, cudaStream_t s);

// Self-test of the bounded waits: one CTA arms an mbarrier for 16 bytes that
// no copy delivers, another looks back at a status word that no item
// publishes (status2[0], zeroed here); both run the same wait code as the
// path kernels with the given poll limit, give up, set kErrTmaTimeout /
// kErrScanTimeout in *err and return.
cudaError_t launch_wait_selftest(uint64_t* status2, uint32_t* err, uint32_t spin_limit, cudaStream_t s);

// A launch that may come up while the kernel before it on the stream finishes
// (see wait_previous). With the counters, marks and look-back words zeroed by
// the plan kernel instead of memsets, the scan in its last CTA and one upload,
// a single query has 6 nodes on the stream instead of 13: 56 -> 33 us on c0,
// 95 -> 68 on c1 with the planner.
template <typename... P, typename... A>
inline cudaError_t launch_after(void (*kernel)(P...), uint32_t grid, uint32_t threads, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace abf
