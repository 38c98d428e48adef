// Internal interface between the C ABI layer (capi.cu) and the kernels.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace shapex {

// LSD radix sort of 64-bit keys in 9-bit digits: 7 passes cover the 63 bits of
// a Morton code; the 8th (bit 63 alone) is trivial for codes and skipped.
constexpr int kSortBits = 9;
constexpr int kSortBins = 1 << kSortBits;
constexpr int kSortPasses = 8;
constexpr int kSortThreads = 512;
constexpr int kSortIpt = 8;
constexpr int kSortTile = kSortThreads * kSortIpt;  // 4096 keys per tile
constexpr int kDedupThreads = 256;
constexpr int kDedupIpt = 16;
constexpr int kDedupTile = kDedupThreads * kDedupIpt;
constexpr int kScanThreads = 256;
constexpr int kScanIpt = 16;
constexpr int kScanTile = kScanThreads * kScanIpt;
constexpr int kLeafThreads = 256;
constexpr int kLeafIpt = 8;
constexpr int kLeafTile = kLeafThreads * kLeafIpt;
// Search hierarchy: leaves of at most kLeafMax points, kFan nodes under each
// inner node, at most kMaxLevels levels (32^6 leaves).
constexpr int kLeafMax = 32;
constexpr int kFan = 32;
constexpr int kMaxLevels = 6;

// Query counters: fp64 solves, nodes visited, buckets scanned, candidates,
// merge steps, inserts.
enum { CNT_FP64 = 0, CNT_NODES, CNT_BUCKETS, CNT_CANDIDATES, CNT_MERGE, CNT_INSERTS, CNT_LEARNED_MISS,
       CNT_CELL_WARPS, CNT_CELL_FALLBACK, CNT_CELL_LOOKUPS, CNT_CELL_POINTS, kQueryCounters };

// Small device-resident state of one build (zeroed at the start of each build).
struct DevState {
    // what a query clears and the host reads after it
    uint32_t err;
    uint32_t work;  // next work item of a persistent search launch
    uint32_t items;  // entries of a search's list of work items, from its front
    uint32_t parts;  // and from its back
    unsigned long long counters[kQueryCounters];  // in the order of se_stats
    // what the host reads after a build
    unsigned long long u;      // unique codes
    unsigned long long n_oct;  // octree nodes
    float min_coord, max_coord, range;
    int32_t root_level;
    // search hierarchy: level l holds level_count[l] nodes from level_off[l] on;
    // the top level is the first of at most kFan nodes
    int32_t top_level;
    uint32_t level_off[kMaxLevels];
    uint32_t level_count[kMaxLevels];
    // build scratch
    uint32_t min_ord;  // ordered-uint encodings (f2ord) of the bbox min / max
    uint32_t max_ord;
    int32_t n_active;                       // non-trivial sort passes
    int32_t pass_active[kSortPasses];
    int32_t pass_parity[kSortPasses];
    uint32_t tile_counter[15];              // dynamic tile ids: sort passes, dedup, octree scan, leaves; encode's blocks
    uint32_t disorder;                      // given keys were not in order
    uint32_t hist[kSortPasses][kSortBins];       // per-digit histograms of the codes
    uint32_t digit_off[kSortPasses][kSortBins];  // exclusive digit offsets
};
constexpr size_t kQueryStateBytes = offsetof(DevState, u);          // err, work, counters
constexpr size_t kHostStateBytes = offsetof(DevState, level_off);   // what the host reads

// Codes of at most 63 bits take this many digit passes.
constexpr int sort_passes(int code_bits) { return (code_bits + kSortBits - 1) / kSortBits; }
constexpr int kCodePasses = sort_passes(63);

// Scratch of one build that must start at zero, in 32-bit words: the octree
// scan's look-back (64-bit), the hierarchy's arrival counters, the look-backs
// of the leaf scan and of dedup, and last those of the sort passes.
struct ScratchLayout {
    int64_t oct, arrivals, leaves, dedup, sort, sort_pass;
    explicit ScratchLayout(int64_t n) {
        const int64_t tiles = (n + kSortTile - 1) / kSortTile;
        oct = 0;
        arrivals = 2 * ((n + kScanTile - 1) / kScanTile);
        leaves = arrivals + n / 512 + 16;  // one counter per hierarchy node of level 2 and up
        dedup = leaves + (n + kLeafTile - 1) / kLeafTile;
        sort = dedup + (n + kDedupTile - 1) / kDedupTile;
        sort_pass = kSortBins * tiles;
    }
    int64_t words(int passes) const { return sort + passes * sort_pass; }
};

// Byte layout of OT::OTNode (reference src/Octree.hpp:19-36), 56 bytes.
struct OtNode {
    int32_t children[8];
    float corner[3];
    float cell_size;
    int32_t child_node_mask;
    int32_t child_leaf_mask;
};
static_assert(sizeof(OtNode) == 56, "OTNode layout");

// Search hierarchy node: the box of its points. A leaf (level 0) is a maximal
// Morton subtree of at most min(leaf_bucket, 32) points: lo.w holds its first
// point and hi.w its point count (int bits). Node i of level l covers nodes
// [32 i, 32 i + 32) of level l - 1.
struct __align__(16) SNode {
    float4 lo;
    float4 hi;
};
// Nodes of the hierarchy over n points, at most (every leaf holds a point).
__host__ __device__ constexpr int64_t hierarchy_nodes(int64_t n) {
    int64_t total = n;
    for (int64_t c = n; c > kFan;) {
        c = (c + kFan - 1) / kFan;
        total += c;
    }
    return total;
}
struct BuildBufs {
    int64_t cap;  // capacity in points
    const float* x;
    const float* y;
    const float* z;
    uint64_t* keys0;
    uint64_t* keys1;
    uint32_t* scratch;   // ScratchLayout(cap).words(kCodePasses)
    uint64_t* codes;     // unique sorted codes
    float4* pts4;        // decoded points, padded for 16-byte loads
    float* pts3;         // decoded points, AoS xyz
    // radix tree as exported (RT::Nodes)
    int32_t* left_child;
    int32_t* parent;
    uint8_t* prefix_n;
    uint8_t* has_leaf_left;
    uint8_t* has_leaf_right;
    // radix tree with the full root range, for the learned radius features
    int32_t* sparent;
    int32_t* leaf_parent;
    int32_t* range_end;
    // search hierarchy
    int32_t* leaf_start;  // first point of each leaf
    SNode* snodes;        // hierarchy_nodes(cap) entries
    // octree
    int32_t* oct_counts;
    int32_t* oct_offsets;  // cap + 1
    void* oct_nodes;       // se_otnode[oct_cap]
    int64_t oct_cap;
    DevState* st;
};

struct BuildParams {
    int64_t n;
    int code_bits;
    int root_compat;
    int build_octree;
    int bucket;
    int build_radix = 1;  // 0: no radix tree (the search does not need it)
    int spin_limit = kSpinLimit;  // polls before a look-back wait gives up
    int stall_first_tile = 0;     // test hook: the first sort tile never publishes its prefix
};

// Stage events of one build: [0] start, then after bbox, encode, sort, dedup,
// radix tree, search boxes, octree.
constexpr int kBuildEvents = 8;
constexpr int kFrontMax = 8192;

// Enqueue the whole build on `s`. Reads x/y/z from bufs; results stay on the
// device. `ev` (kBuildEvents events, may be null) are recorded between stages;
// *launches receives the number of kernels launched. Of a cloud of at most
// kFrontMax points events 2 to 4 are not recorded: one kernel does stages 0 to 3.
cudaError_t enqueue_build(const BuildBufs& b, const BuildParams& p, cudaStream_t s, int num_sms, cudaEvent_t* ev,
                          int* launches);
// Enqueue only the octree stage (used to redo it after a capacity regrow).
cudaError_t enqueue_octree(const BuildBufs& b, const BuildParams& p, cudaStream_t s, int* launches);

// ---- learned search-radius proposal (mlp.cu) --------------------------------
constexpr int kMlpF = 32;  // features per point
constexpr int kMlpH = 64;  // hidden width
// FP32 master parameters, one flat array.
struct MlpLayout {
    static constexpr int W1 = 0;                   // [kMlpF][kMlpH], input-major
    static constexpr int B1 = W1 + kMlpF * kMlpH;  // [kMlpH]
    static constexpr int W2 = B1 + kMlpH;          // [kMlpH][kMlpH], input-major
    static constexpr int B2 = W2 + kMlpH * kMlpH;  // [kMlpH]
    static constexpr int W3 = B2 + kMlpH;          // [kMlpH]
    static constexpr int B3 = W3 + kMlpH;          // scalar
    static constexpr int N = B3 + 1;
};
constexpr int kMlpParams = MlpLayout::N;

cudaError_t enqueue_features(const BuildBufs& b, int64_t u, int code_bits, int64_t start, int64_t count, float* out,
                             cudaStream_t s);
cudaError_t enqueue_predict_radius(const BuildBufs& b, const float* params, float margin, int64_t u, int code_bits,
                                   int64_t start, int64_t count, float* r2_out, float* yhat_out, cudaStream_t s);
cudaError_t enqueue_mlp_forward(const float* params, const float* X, int64_t n, float* yhat, float* h1, float* h2,
                                cudaStream_t s);
// Adds the gradient of a batch to grads and its loss to *loss (both start at zero).
cudaError_t enqueue_mlp_grad(const float* params, const float* X, const float* y, int64_t n, float tau, float* grads,
                             float* loss, cudaStream_t s, int num_sms);
// One Adam step; leaves grads at zero.
cudaError_t enqueue_adam(float* params, float* grads, float* m, float* v, float lr, int step, cudaStream_t s);

// Sort n 64-bit keys in place in `keys` (ascending) with the onesweep passes;
// `tmp` (n keys), `lookback` (kSortBins words per 4096-key tile) and `st` are scratch.
cudaError_t enqueue_sort_keys(uint64_t* keys, uint64_t* tmp, int64_t n, uint32_t* lookback, DevState* st,
                              cudaStream_t s, int num_sms);

// Foreign queries in the order of their places among the tree's codes: keys
// hold the place (30 bits, scaled to the top of them) from bit kOrderShift up
// and the query's number in the low 30 bits, sorted by as many of the place's
// leading bits as the number of queries calls for.
constexpr int kOrderShift = 33;
struct QueryOrder {
    uint64_t* keys0;
    uint64_t* keys1;
    uint32_t* lookback;  // kSortBins words per 4096-key tile
    DevState* st;
};
// *order receives the sorted keys (keys0 or keys1), *items the search's work
// items in the other buffer (their number goes into b.st->items), *shift the
// scale of the places, *launches the number of kernels launched.
cudaError_t enqueue_query_order(const BuildBufs& b, const QueryOrder& o, const float* queries, int64_t n, int64_t u,
                                int code_bits, const uint64_t** order, const uint64_t** items, int* shift,
                                cudaStream_t s, int num_sms, int* launches);
// Queries per warp of a search of `count` queries, and whether foreign ones are
// put in order (those that are not come one to a warp).
int queries_per_warp(int64_t count, int num_sms, bool foreign);
bool order_foreign(int64_t count, int64_t u, int k, int num_sms);
// Trees of at most this many points: foreign queries are taken as given, as many
// to a warp as the tree's own points (every warp reads all of the tree anyway).
// 100k queries, k = 1: of a tree of 5 points 103 us in order, 56 as given; of 100
// points 118 and 64 us.
constexpr int64_t kTinyTree = 256;
// Whether a search of `count` of the tree's own points lists its work items
// first (one more kernel; the list takes b.scratch). Not where other clouds fill
// the GPU beside it (device_count).
bool list_points(int64_t count, int k, int num_sms);
// A work item of sorted foreign queries: the first of them in the low half, how
// many in the high half. Places that the queries of one warp may span: as many
// as the foreign rule allows, and as many as of the tree's own points (which
// share nearly everything). 250k queries near a 2M-point scene, k = 8: 1046 us
// without seed windows for those that span less, 721 us with windows up to 256
// places, 674 us up to 512 (4096 cost more than they save). The second bound at
// 1024 makes 50k queries 694 us, at 64 every seventh tree point as a query (50k)
// 373 us; as now 400 and 293 us.
constexpr int kWindowSpan = 512;
constexpr int kTogetherSpan = 256;

struct QueryParams {
    int k;
    int64_t start;      // first query (self queries)
    int64_t count;      // number of queries
    int64_t u;          // tree points
    const float* ext_queries;  // AoS xyz external queries or nullptr (self queries)
    const uint64_t* order = nullptr;  // external queries: their order (enqueue_query_order), or nullptr: as given
    const uint64_t* items = nullptr;  // with order: the work items
    int order_shift = 0;
    int32_t* out_idx;   // count*k or nullptr
    float* out_d2;      // count*k or nullptr
    float* out_normals; // count*3 or nullptr
    float vx, vy, vz;
    float eigengap_fp64;
    int code_bits;
    int seed_halo;
    const float* learned_r2;  // per query: starting bound from the learned radius, or nullptr
    int learned_skip_seed;    // with learned_r2: skip the Morton-window seed
    int device_count;         // 1: query all u points of the build, u read on the device; `count`
                              // is then an upper bound used only to size the grid
    int compat;               // 1: the reference's approximate octree search and FP32 covariance
    int64_t n_octree;         // octree nodes (compat search)
    int step_limit = 0;       // > 0: node visits per warp before the walk gives up (test hook)
    // learned cell scan: the code-range table of this build (null: the learned
    // attempt walks the tree with the cap), its per-axis shift, and the most
    // points a warp scans before it falls back to the walk
    const uint32_t* cell_lut = nullptr;
    int lut_shift = 0;
    int cell_pmax = 0;
    int cell_span = 3;
    // persistent batch launches: resident blocks per SM (0: as many as fit)
    // and warps per block (0: the per-k default; 2 or 4)
    int batch_blocks_per_sm = 0;
    int batch_warps_per_block = 0;
};

// Code-range table of a build for the learned cell scan: lut[j] = the number
// of unique codes below j << (3 * (bits per axis - level)), j = 0 .. 8^level
// (lut[8^level] = u). Level between 1 and the bits per axis.
cudaError_t enqueue_cell_lut(const BuildBufs& b, int code_bits, int level, uint32_t* lut, cudaStream_t s,
                             int num_sms);

cudaError_t enqueue_query(const BuildBufs& b, const QueryParams& q, cudaStream_t s, int num_sms);

// One cloud of a batched query: its own points, search hierarchy and build
// state (u is read there on the device), its output, and the index of its
// first 32-query item in the launch.
struct BatchCloud {
    const float4* pts;
    const SNode* snodes;
    DevState* st;
    float* out_normals;
    int64_t item0;
};

// Normals of many clouds that share q.k in one persistent launch (grid = the
// kernel's resident blocks on every SM). `clouds` is a device array of
// n_clouds entries, `counter` a device word this call resets. q supplies k,
// viewpoint, eigengap threshold and seed halo.
// u and the error word of every cloud of a batch (states st[0..n)) into
// u_out / err_out.
cudaError_t enqueue_batch_collect(const DevState* st, int n, unsigned long long* u_out, uint32_t* err_out,
                                  cudaStream_t s);

cudaError_t enqueue_query_batch(const BatchCloud* clouds, int n_clouds, int64_t n_items, unsigned long long* counter,
                                const QueryParams& q, cudaStream_t s, int num_sms);
// Reference-compatible search over the OTNode array (enqueue_query forwards
// to it when q.compat is set).
cudaError_t enqueue_query_compat(const BuildBufs& b, const QueryParams& q, cudaStream_t s, int num_sms);

}  // namespace shapex
