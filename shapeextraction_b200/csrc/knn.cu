// Exact kNN over the search hierarchy, fused with covariance, 3x3 symmetric
// eigensolve and orientation (sm_100a).
//
// Replaces, from the reference (paths relative to its project root):
//   knnSearchKernel<k> + nodeBoxDistance + PriorityQueue
//       src/Octree.hpp:136-212, src/Octree.cu:326-352, src/dequeue.hpp
//   findCovariancesKernel<k>            src/NormalEstimation.hpp:96-156
//   cusolverDnSsyevjBatched             src/NormalEstimation.hpp:235-301
//   normalsFromEigenVectors             src/NormalEstimation.hpp:158-192
//
// One warp serves up to 32 consecutive queries (Morton-ordered, so spatially
// coherent); lane i owns query i. Each lane keeps the k smallest squared
// distances offered to it as a sorted list in registers, whose last entry is
// its pruning bound, and the (distance, index) candidates within the bound in
// shared memory. The warp first offers the Morton window around its queries,
// then walks the search hierarchy: 32 nodes are tested at once against the box
// of the warp's queries, nearest first, and each that passes by all 32
// queries. Points come in runs of at most 32, staged in shared memory; each
// lane's hits are a bit mask, from which they are appended to its candidates.
// When a lane's slots are full, all lanes merge their fresh distances into
// their lists and drop the candidates beyond their bounds. The k nearest are
// the candidates left at the end, sorted by (distance, index). Pruning uses the
// box distance with the same rounding chain as the point distance, so the
// result is exact, ties broken by point index.
//
// Before, the lists held (distance, index) keys and took one insertion per
// buffered candidate. Distances alone merge eight at a time through min/max
// networks in half the registers, and nothing is gathered twice: 2M scene,
// k = 16, search 2.69 -> 2.29 ms; 20M precision mix 18.0 -> 15.5 ms; 1M lists of
// 32 3.14 -> 2.05 ms. What holds it now is latency and issue: of the 4M precision
// mix 64% of the issue slots are busy, fixed-latency waits 2.6 per issue, waits
// for global loads 1.35, for shared ones 0.9.

#include <cfloat>
#include <climits>
#include <cstdint>
#include <type_traits>
#include <utility>

#include "pipeline.cuh"
#include "eig3.cuh"

namespace shapex {

namespace {

// Per-k tile shape, measured on B200 (2M scene): candidate slots (8 bytes per
// lane and slot, shared memory) against resident warps. Fewer slots mean more
// merges and prunes, fewer warps leave the fixed-latency stalls uncovered, and
// registers beyond the budget spill. k = 16: 28 slots x 24 warps 2281 us, 32 x
// 22 2288 (20M precision mix 15.47 ms; kept), 36 x 20 2328, 24 x 28 2787;
// k = 8: 22 x 28 1434 us, 22 x 24 1477, 18 x 24 1480, 20 x 20 1578; k = 32
// (1M): 48 x 16 2049 us, 56 x 14 2105, 52 x 14 2177, 44 x 18 2230. Blocks of
// two warps: with four, 22 warps do not divide; one each costs 1 KB of reserved
// shared memory per warp (2371 us).
template <int K>
struct KnnCfg {
    static constexpr int buf = K <= 8 ? 22 : (K <= 16 ? 32 : (K <= 24 ? 40 : 48));  // candidate slots per lane
    static constexpr int threads = 64;                                                // block size
    static constexpr int warps = threads / 32;
    static constexpr int min_blocks = K <= 8 ? 14 : (K <= 16 ? 11 : (K <= 24 ? 9 : 8));  // resident blocks per SM asked of ptxas
};
constexpr int kMaxHalo = 48;            // seed points on each side of a warp's queries
constexpr unsigned FULL = 0xffffffffu;

// (squared distance, index) packed so that one unsigned compare orders by
// distance then index; distances are >= 0, so their IEEE bits are monotonic.
__device__ __forceinline__ unsigned long long pack_key(float d, int64_t i) {
    return ((unsigned long long)__float_as_uint(d) << 32) | (uint32_t)i;
}
constexpr unsigned long long kEmptyKey = (0x7f800000ull << 32) | 0xffffffffull;  // (+inf, max index)
__device__ __forceinline__ int32_t key_idx(unsigned long long k) { return (int32_t)(uint32_t)k; }
__device__ __forceinline__ float key_d(unsigned long long k) { return __uint_as_float((uint32_t)(k >> 32)); }

// v[i] for a run-time i, as a masked OR over all entries, so that the list
// stays in registers (a direct v[i] would move it to local memory).
template <int K>
__device__ __forceinline__ float pick(const float (&v)[K], int i) {
    uint32_t acc = 0;
#pragma unroll
    for (int j = 0; j < K; ++j) acc |= j == i ? __float_as_uint(v[j]) : 0u;
    return __uint_as_float(acc);
}

__device__ __forceinline__ void exchange(float& a, float& b) {  // a <= b afterwards
    const float t = fminf(a, b);
    b = fmaxf(a, b);
    a = t;
}
__device__ __forceinline__ void exchange(unsigned long long& a, unsigned long long& b) {
    const bool sw = b < a;
    const unsigned long long t = sw ? b : a;
    b = sw ? a : b;
    a = t;
}

// Ascending sort of N values in registers: Batcher's odd-even merge exchange
// (Knuth, TAOCP vol. 3, Algorithm 5.2.2M): 19 exchanges for 8 values, 63 for
// 16, 191 for 32. The network is a compile-time list of wire pairs.
template <int N>
struct SortNet {
    int n = 0;
    int lo[N * N / 2] = {}, hi[N * N / 2] = {};
    __host__ __device__ constexpr SortNet() {
        for (int p = 1; p < N; p <<= 1)
            for (int k = p; k >= 1; k >>= 1)
                for (int j = k % p; j + k < N; j += 2 * k)
                    for (int i = j; i < j + k && i + k < N; ++i)
                        if (i / (2 * p) == (i + k) / (2 * p)) {
                            lo[n] = i;
                            hi[n++] = i + k;
                        }
    }
};
// A bitonic merge of N wires, N not necessarily a power of two: the network
// of the next power of two with its lowest wires held at minus infinity, so
// that their exchanges fall away.
template <int N>
struct MergeNet {
    int n = 0;
    int lo[N * 5] = {}, hi[N * 5] = {};
    __host__ __device__ constexpr MergeNet() {
        int P = 1;
        while (P < N) P <<= 1;
        for (int h = P / 2; h >= 1; h >>= 1)
            for (int i = P - N; i + h < P; ++i)
                if ((i & h) == 0) {
                    lo[n] = i - (P - N);
                    hi[n++] = i + h - (P - N);
                }
    }
};
template <class Net, class T, int N, size_t... I>
__device__ __forceinline__ void run_net(T (&v)[N], std::index_sequence<I...>) {
    constexpr Net net;
    (exchange(v[std::integral_constant<int, net.lo[I]>::value], v[std::integral_constant<int, net.hi[I]>::value]), ...);
}
template <class T, int N>
__device__ __forceinline__ void sort_values(T (&v)[N]) {
    run_net<SortNet<N>>(v, std::make_index_sequence<SortNet<N>().n>());
}

constexpr int kBatch = 8;  // candidates merged into a list at once

// The k smallest squared distances offered to one query so far, ascending, in
// registers; their last is the pruning bound. The points they belong to are
// not carried along: the lane's buffer of candidate indices keeps every point
// within the bound, and the k nearest are taken from it at the end. With
// EXACT = false the list is longer than k and the bound is entry k-1.
//
// Distances alone are 32 bits, so an exchange of the merge network is a min
// and a max, where (distance, index) keys took six instructions on the
// half-rate ALU pipe, and the list takes half the registers.
template <int K, bool EXACT>
struct Nearest {
    float d[K];
    float tau;  // d[k - 1]
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int j = 0; j < K; ++j) d[j] = INFINITY;
        tau = INFINITY;
    }
    __device__ __forceinline__ void set_bound(int k) { tau = EXACT ? d[K - 1] : pick(d, k - 1); }
    __device__ __forceinline__ void sort_filled(int k) {
        sort_values(d);
        set_bound(k);
    }
    // The K lowest of the list and the batch c: the list's tail against the
    // sorted batch reversed leaves the K lowest as a sequence that rises and
    // then falls (Batcher 1968), which a bitonic merge sorts.
    __device__ __forceinline__ void merge(float (&c)[kBatch], int k) {
        sort_values(c);
#pragma unroll
        for (int t = 0; t < kBatch && t < K; ++t) d[K - 1 - t] = fminf(d[K - 1 - t], c[t]);
        run_net<MergeNet<K>>(d, std::make_index_sequence<MergeNet<K>().n>());
        set_bound(k);
    }
};

// Per-warp shared scratch. pts[0, 24): a staged run of 32 points; pts[24, 64):
// while the warp walks the hierarchy, the order keys of the levels above the
// current one; pts[64, 96): the lanes' queries and bounds. The cell scan uses
// a larger pts in its own way. d and idx: each lane's candidates, [slot][lane]
// so that a warp's accesses to one slot fall in distinct banks.
template <int B, bool CELLS = false>
struct WarpSmem {
    float4 pts[CELLS ? 128 : 96];
    float d[B][32];
    int32_t idx[B][32];
    uint32_t count[kQueryCounters];  // the warp's work counters, added to the build state's when it ends
    uint32_t whole, items;           // work items of the launch: those from the front of a list, all
    float4 box_lo, box_hi;           // the box of the warp's active queries
    __device__ __forceinline__ uint32_t* level_keys(int l) {  // l >= 1
        return reinterpret_cast<uint32_t*>(&pts[24]) + 32 * (l - 1);
    }
    __device__ __forceinline__ float4* query() { return pts + 64; }  // x, y, z, bound (-1: idle lane)
};
static_assert(24 + (kMaxLevels - 1) * 8 <= 64, "order keys fit behind the staged run");

// Ordered widest first so that the struct packs into 128 bytes: one more
// padded word (144 bytes) made ptxas give the k = 32 kernels 161-163
// registers instead of 142, one resident block per SM fewer.
struct QArgs {
    int64_t start, count, u;
    union {
        const float* ext;      // foreign queries
        const uint64_t* parts;  // the tree's own points: work items (null: warp_queries each)
    };
    int32_t* out_idx;
    float* out_d2;
    float* out_normals;
    union {
        const float* learned_r2;
        const uint64_t* items;  // foreign queries with an order: the work items
    };
    union {
        const uint32_t* cell_lut;   // learned cell scan: code-range table (null: tree walk with the cap)
        const uint64_t* order;      // foreign queries: their order (null: as given)
        const uint64_t* parts_end;  // with `parts` (and no cell scan)
    };
    float vx, vy, vz;
    float gap;
    int k;
    int code_bits;
    int seed_halo;
    int learned_skip_seed;
    int device_count;  // 1: u = count = the build's unique-point count, read on the device (start 0)
    int step_limit;    // > 0: node visits per warp before the walk gives up (test hook)
    union {
        int lut_shift;    // per-axis shift of the table's level (bits per axis - level)
        int order_shift;  // scale of the places in `order`
    };
    union {
        int cell_pmax;  // cell scan: most points per warp before it falls back to the walk
        float close;    // foreign queries as given: extent, in ranges of the tree, of a group taken together (0: none)
    };
    int cell_span;     // cell scan: most cells per axis covering one lane's ball (2..4)
    int warp_queries;  // queries per warp, 1..32
};
static_assert(sizeof(QArgs) <= 128, "QArgs grew past 128 bytes");

struct Counters {
    int cand = 0, ins = 0, merge = 0, buckets = 0, lmiss = 0, cells = 0, cell_fallback = 0, cell_lookups = 0,
        cell_points = 0;
};

// One query: its candidates are slots [0, n) of the lane's columns W.d and
// W.idx, every point offered so far that may be among its k nearest; the
// distances of the first `merged` of them are in the list.
struct Query {
    float x, y, z;
    int k;
    int n, merged;
};

// Merge the distances of every lane's fresh candidates into its list; the warp
// steps through max-over-lanes batches together.
template <int K, bool EXACT, class WS>
__device__ __forceinline__ void merge_fresh(Nearest<K, EXACT>& nn, Query& q, WS& W, int lane, Counters& ct) {
    const int fresh = q.n - q.merged;
    const int most = (int)__reduce_max_sync(FULL, (unsigned)fresh);
    ct.merge += most;
    ct.cand += fresh;
#pragma unroll 1
    for (int j = 0; j < most; j += kBatch) {
        float c[kBatch];
#pragma unroll
        for (int t = 0; t < kBatch; ++t) c[t] = j + t < fresh ? W.d[q.merged + j + t][lane] : INFINITY;
        nn.merge(c, q.k);
    }
    q.merged = q.n;
}

// Drop the candidates beyond every lane's bound (all must be merged). At most
// `room` stay: equal distances can leave more than k, and of those at the
// bound the lowest indices go first, as in the lists.
template <class WS>
__device__ __forceinline__ void prune(Query& q, float tau, int room, WS& W, int lane, Counters& ct) {
    const int most = (int)__reduce_max_sync(FULL, (unsigned)q.n);
    int w = 0;
#pragma unroll 4
    for (int j = 0; j < most; ++j) {
        const float d = W.d[j][lane];
        if (j < q.n && d <= tau) {
            const int32_t i = W.idx[j][lane];
            W.d[w][lane] = d;
            W.idx[w][lane] = i;
            ++w;
        }
    }
    ct.ins += w;
    if (w > room) {  // ties at the bound: keep k candidates
        int ties = q.k;
        for (int j = 0; j < w; ++j) ties -= W.d[j][lane] < tau;
        int32_t last = -1;  // the ties-th lowest index at the bound
        for (int i = 0; i < ties; ++i) {
            int32_t next = INT_MAX;
            for (int j = 0; j < w; ++j) {
                const int32_t at = W.idx[j][lane];
                if (at > last && at < next && W.d[j][lane] == tau) next = at;
            }
            last = next;
        }
        int v = 0;
        for (int j = 0; j < w; ++j) {
            const float d = W.d[j][lane];
            const int32_t at = W.idx[j][lane];
            if (d < tau || at <= last) {
                W.d[v][lane] = d;
                W.idx[v][lane] = at;
                ++v;
            }
        }
        w = v;
    }
    q.n = q.merged = w;
}

// Append every lane's hits among a run of points (bit i of `hits`: point
// `first` + i, at(i) its coordinates) to its candidates, making room on the
// way; a hit that a bound tightened meanwhile excludes is passed over. With
// `settle` all candidates are merged in any case. A prune leaves at most `room`
// candidates.
template <int K, bool EXACT, class WS, class At>
__device__ __forceinline__ void take_hits(uint32_t hits, bool settle, int room, At at, Nearest<K, EXACT>& nn, Query& q, float& tau,
                                          float cap, WS& W, int lane, Counters& ct) {
    constexpr int kBuf = KnnCfg<K>::buf;
    for (;;) {
        const int mine = __popc(hits);
        int rounds = (int)__reduce_max_sync(FULL, (unsigned)mine);
        if (rounds == 0 && !settle) return;
        if (settle || __any_sync(FULL, q.n + mine > kBuf)) {
            settle = false;
            merge_fresh(nn, q, W, lane, ct);
            prune(q, nn.tau, room, W, lane, ct);
            if (tau >= 0.0f) tau = fminf(nn.tau, cap);
            rounds = min(rounds, (int)__reduce_min_sync(FULL, (unsigned)(kBuf - q.n)));
        }
#pragma unroll 1
        for (; rounds > 0; --rounds) {
            if (hits) {
                const int i = __ffs(hits) - 1;
                hits &= hits - 1;
                int32_t idx;
                const float3 p = at(i, idx);
                const float d = dist2(q.x, q.y, q.z, p.x, p.y, p.z);
                if (d <= tau) {
                    W.d[q.n][lane] = d;
                    W.idx[q.n][lane] = idx;
                    ++q.n;
                }
            }
        }
    }
}

// The lanes' hits among points [first, first + cnt) (cnt <= 32) except those in
// [w0, w1) (already offered): bit i of a lane's mask for point first + i within
// its bound. The points are staged in pairs for dist2_pair: floats [4j, 4j + 4)
// hold x and y of points 2j and 2j + 1, floats [64 + 2j, 64 + 2j + 2) their z;
// a slot past cnt holds a NaN x, whose distance passes no bound. Either every
// lane tests all points (two at a time), or, when few lanes need them (`needm`),
// each lane holds one point and the warp steps over those queries, so that the
// cost follows their number.
template <class WS>
__device__ __forceinline__ uint32_t scan_run(int32_t first, int cnt, uint32_t needm, int32_t w0, int32_t w1,
                                             const Query& q, float tau, WS& W, int lane,
                                             const float4* __restrict__ pts) {
    float* f = reinterpret_cast<float*>(W.pts);
    const float4 p = lane < cnt ? __ldg(pts + first + lane) : make_float4(__int_as_float(0x7fc00000), 0.f, 0.f, 0.f);
    {
        const int o = 4 * (lane >> 1) + (lane & 1);
        f[o] = p.x;
        f[o + 2] = p.y;
        f[64 + lane] = p.z;
    }
    __syncwarp();
    uint32_t hits = 0;
    if (2 * __popc(needm) < cnt) {
        while (needm) {
            const int i = __ffs(needm) - 1;
            needm &= needm - 1;
            const float4 o = W.query()[i];
            const uint32_t h = __ballot_sync(FULL, dist2(o.x, o.y, o.z, p.x, p.y, p.z) <= o.w);
            if (lane == i) hits = h;
        }
    } else {
        const uint64_t qqx = twice(q.x), qqy = twice(q.y), qqz = twice(q.z);
#pragma unroll 1
        for (int t = 0; t < cnt; t += 8) {
            uint32_t h = 0;
#pragma unroll
            for (int e = 0; e < 8; e += 2) {
                const ulonglong2 xy = *reinterpret_cast<const ulonglong2*>(f + 2 * (t + e));
                const uint64_t d =
                    dist2_pair(qqx, qqy, qqz, xy.x, xy.y, *reinterpret_cast<const uint64_t*>(f + 64 + t + e));
                if (lo_half(d) <= tau) h |= 1u << e;
                if (hi_half(d) <= tau) h |= 2u << e;
            }
            hits |= h << t;
        }
    }
    if (first < w1 && first + cnt > w0) {  // some were already offered
        const int lo = max(w0 - first, 0), hi = min(w1 - first, 32);
        hits &= ~((0xffffffffu >> (32 - (hi - lo))) << lo);
    }
    return hits;
}

// Position of set bit number n (from 0) of w; w has more than n set bits.
__device__ __forceinline__ int nth_set_bit(uint32_t w, int n) {
    int pos = 0;
#pragma unroll
    for (int width = 16; width >= 1; width >>= 1) {
        const int c = __popc(w & ((1u << width) - 1u));
        if (n >= c) {
            n -= c;
            w >>= width;
            pos += width;
        }
    }
    return pos;
}

// First index in codes[lo, hi) whose code is >= key (hi when none).
__device__ __forceinline__ uint32_t lower_bound_codes(const uint64_t* __restrict__ codes, uint32_t lo, uint32_t hi,
                                                      uint64_t key) {
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(codes + mid) < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Bounds of the decoded coordinates X0..X1 of one axis, for pruning: the
// decode (codeToPoint: fma(X / M, range, min)) is evaluated with a multiply by
// 1/M instead of the division and widened by `pad`, which exceeds the
// difference between the two evaluations (at most range * 2^-22 + max|coord| *
// 2^-23), so every decoded point of the range lies inside [lo, hi].
__device__ __forceinline__ void axis_bounds(uint32_t X0, uint32_t X1, float inv_m, float mn, float range, float pad,
                                            float& lo, float& hi) {
    lo = __fmaf_rn((float)X0 * inv_m, range, mn) - pad;
    hi = __fmaf_rn((float)X1 * inv_m, range, mn) + pad;
}

// Integer code-coordinate box [lo, hi] (per axis, clamped to [0, M]) that
// holds every tree point within squared distance r2 of the tree point whose
// code is `code`: |x_p - x_q| <= R for every point p with dist2 <= r2
// (dist2's rounding costs far less than the 1e-6 added to R), and in code
// units the decode adds at most 1/4 + 2^-23 * M * max|coordinate| / range on
// each side. r2 must be finite and >= 0; a degenerate range gives the whole
// cube.
__device__ __forceinline__ void ball_box(uint64_t code, float r2, uint32_t M, float mn, float range, uint32_t (&lo)[3],
                                         uint32_t (&hi)[3]) {
    const float fbs = (float)M;
    const float R = __fmul_ru(__fsqrt_ru(r2), 1.000001f);
    const float ru = __fmul_ru(R, __fdiv_ru(fbs, range));
    const float big = fmaxf(fabsf(mn), fabsf(mn + range));
    const float slack = __fadd_ru(__fmul_ru(__fmul_ru(1.1920929e-7f, fbs), __fdiv_ru(big, range)), 0.25f);
    const float ext = __fadd_ru(ru, slack) + 1.0f;
    const int64_t e = ext < 4.0e9f ? (int64_t)ceilf(ext) : ((int64_t)1 << 40);  // NaN: whole cube
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        const int64_t X = (int64_t)gather3(code >> ax);
        lo[ax] = (uint32_t)max64(0, X - e);
        hi[ax] = (uint32_t)min64((int64_t)M, X + e);
    }
}

constexpr int kCellBits = 1024;   // cells of a warp's union grid: one bit each, in pts[112, 120)
constexpr int kCellRanges = 64;   // nonempty cells a warp scans: listed in pts[32, 96), order keys after

// Learned attempt as a direct scan of Morton cells, with no tree walk.
//
// Each lane's predicted ball (radius sqrt(cap) around its query) is covered by
// an integer box of code coordinates, widened by the decode rounding, and the
// warp picks the finest level at which every lane's box spans at most
// cell_span cells per axis. The union of the lanes' cells is marked in a
// shared bitmap; each marked cell is the contiguous run of sorted codes under
// its prefix, found with the build's code-range table and a short binary
// search. The nonempty cells are taken nearest first (box distance to the
// warp's first query); a cell that no lane's current bound reaches any more is
// skipped, and the points of the others are packed into 32-point chunks that
// every lane tests against its own bound (dense: no per-lane loops). Every
// point within a lane's cap lies in one of its cells and is offered to it
// unless the lane's bound already excludes the cell's box, so a lane whose
// k-th distance ends within its cap has its exact k best; the caller searches
// the others again. Returns false, having offered nothing, when the warp's
// cells are too many (queries spread across distant regions) or hold more
// than cell_pmax points; the caller then walks the tree with the cap.
template <int K, bool EXACT, class WS>
__device__ __forceinline__ bool cell_scan(Nearest<K, EXACT>& nn, Query& q, WS& W, int lane, Counters& ct,
                                          const float4* __restrict__ pts, const uint64_t* __restrict__ codes,
                                          const QArgs& a, const DevState* st, bool act, int64_t qi, float cap) {
    const float qx = q.x, qy = q.y, qz = q.z;
    const int bpa = a.code_bits / 3;
    const uint32_t M = bitscale_of(a.code_bits);
    const float fbs = (float)M;
    const float mn = st->min_coord, range = st->range;
    const bool ok = act && cap >= 0.0f && cap < INFINITY;  // false for NaN
    uint32_t lo[3] = {0u, 0u, 0u}, hi[3] = {0u, 0u, 0u};
    int s = 0;
    if (ok) {
        ball_box(__ldg(codes + qi), cap, M, mn, range, lo, hi);
        uint32_t dmax = 0;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) dmax = max(dmax, hi[ax] - lo[ax]);
        // the finest level at which the box spans at most cell_span cells per
        // axis: (hi >> s) - (lo >> s) <= (dmax >> s) + 1 <= cell_span - 1
        while ((int)(dmax >> s) > a.cell_span - 2) ++s;
    }
    const uint32_t okm = __ballot_sync(FULL, ok);
    if (!okm) return true;  // no lane has a usable cap: every active lane is searched again
    s = (int)__reduce_max_sync(FULL, (unsigned)(ok ? s : 0));
    uint32_t A[3], g[3];
    for (int tries = 0;; ++tries) {
        uint64_t cells = 1;
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            A[ax] = __reduce_min_sync(FULL, ok ? (lo[ax] >> s) : 0xffffffffu);
            const uint32_t b = __reduce_max_sync(FULL, ok ? (hi[ax] >> s) : 0u);
            g[ax] = b - A[ax] + 1;
            cells *= g[ax];
        }
        if (cells <= (uint64_t)kCellBits) break;
        if (tries == 2 || s >= bpa) {
            ++ct.cell_fallback;
            return false;
        }
        ++s;
    }
    // mark the union of the lanes' cells
    uint32_t* bits = reinterpret_cast<uint32_t*>(&W.pts[112]);  // words [0, 32); inclusive prefixes at [32, 64)
    __syncwarp();
    bits[lane] = 0u;
    __syncwarp();
    if (ok) {
        for (uint32_t z = (lo[2] >> s) - A[2]; z <= (hi[2] >> s) - A[2]; ++z)
            for (uint32_t y = (lo[1] >> s) - A[1]; y <= (hi[1] >> s) - A[1]; ++y)
                for (uint32_t x = (lo[0] >> s) - A[0]; x <= (hi[0] >> s) - A[0]; ++x) {
                    const uint32_t b = (z * g[1] + y) * g[0] + x;
                    atomicOr(&bits[b >> 5], 1u << (b & 31));
                }
    }
    __syncwarp();
    const uint32_t word = bits[lane];
    int incl = __popc(word);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += t;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    uint32_t* pre = bits + 32;
    pre[lane] = (uint32_t)incl;
    __syncwarp();
    // one cell per lane per round: its code range and its order key
    int4* list = reinterpret_cast<int4*>(&W.pts[32]);                         // (first, count, prefix lo, hi)
    uint32_t* okeys = reinterpret_cast<uint32_t*>(&W.pts[32 + kCellRanges]);  // scan order keys
    const uint32_t* lut = a.cell_lut;
    const int ls = a.lut_shift;
    const float inv_m = 1.0f / fbs;
    const float big = fmaxf(fabsf(mn), fabsf(mn + range));
    const float pad = __fadd_ru(__fmul_ru(big, 4.76837158e-7f), __fmul_ru(range, 9.53674316e-7f));  // 2^-21, 2^-20
    // order reference: the warp's first query with a usable cap
    const int ref = __ffs(okm) - 1;
    const float rx = __shfl_sync(FULL, qx, ref), ry = __shfl_sync(FULL, qy, ref), rz = __shfl_sync(FULL, qz, ref);
    int nr = 0;
    int64_t ptotal = 0;
    ct.cell_lookups += total;
    for (int r0 = 0; r0 < total; r0 += 32) {
        const int idx = r0 + lane;
        uint32_t first = 0, cnt = 0;
        uint64_t P = 0;
        float key = 0.0f;
        if (idx < total) {
            int w = 0;  // the word holding marked cell number idx
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1)
                if ((int)pre[w + step - 1] <= idx) w += step;
            const int before = w > 0 ? (int)pre[w - 1] : 0;
            const uint32_t b = (uint32_t)(w * 32 + nth_set_bit(bits[w], idx - before));
            const uint32_t C[3] = {A[0] + b % g[0], A[1] + (b / g[0]) % g[1], A[2] + b / (g[0] * g[1])};
            P = spread3(C[0]) | (spread3(C[1]) << 1) | (spread3(C[2]) << 2);
            uint32_t last;
            if (s >= ls) {
                const int d = 3 * (s - ls);
                first = __ldg(lut + (P << d));
                last = __ldg(lut + ((P + 1) << d));
            } else {
                const uint64_t j = P >> (3 * (ls - s));
                const uint32_t l0 = __ldg(lut + j), l1 = __ldg(lut + j + 1);
                first = lower_bound_codes(codes, l0, l1, P << (3 * s));
                last = lower_bound_codes(codes, first, l1, (P + 1) << (3 * s));
            }
            cnt = last - first;
            float bl[3], bh[3];
#pragma unroll
            for (int ax = 0; ax < 3; ++ax)
                axis_bounds(C[ax] << s, (uint32_t)min64((int64_t)M, ((int64_t)(C[ax] + 1) << s) - 1), inv_m, mn, range,
                            pad, bl[ax], bh[ax]);
            key = box_dist2(rx, ry, rz, bl[0], bl[1], bl[2], bh[0], bh[1], bh[2]);
        }
        const bool keep = cnt > 0;
        const uint32_t km = __ballot_sync(FULL, keep);
        if (keep) {
            const int pos = nr + __popc(km & lanemask_lt());
            if (pos < kCellRanges) {
                list[pos] = make_int4((int)first, (int)cnt, (int)(uint32_t)P, (int)(uint32_t)(P >> 32));
                okeys[pos] = (__float_as_uint(key) & ~0x7fu) | (uint32_t)pos;  // distance bits, entry number
            }
        }
        nr += __popc(km);
        ptotal += (int64_t)__reduce_add_sync(FULL, keep ? min(cnt, 1u << 26) : 0u);
    }
    if (nr > kCellRanges || ptotal > (int64_t)a.cell_pmax) {
        ++ct.cell_fallback;
        return false;
    }
    __syncwarp();
    ++ct.cells;
    ct.cell_points += (int)ptotal;
    // Cells nearest first, so that the bounds tighten early. Lane l holds the
    // order keys of entries l and l + 32. A cell goes on only if some lane's
    // current bound (its k-th distance so far, at most its cap) reaches the
    // cell's box; its points are appended to the staging chunk pts[0, 32)
    // (index in .w), and each full chunk is tested by every lane.
    uint32_t ok0 = lane < nr ? okeys[lane] : 0xffffffffu;
    uint32_t ok1 = lane + 32 < nr ? okeys[lane + 32] : 0xffffffffu;
    int fill = 0;
    bool merged = false;
    // Hits are appended as they come, eight points at a time so that the slots
    // last: with the hits of 32 points in a mask, appended afterwards in as many
    // steps as the lane with most of them has, this search took 6.6 ms on a 2M
    // scene (k = 16), now 3.7 ms.
    auto test_chunk = [&](int n) {
        __syncwarp();
        for (int t0 = 0; t0 < n; t0 += 8) {
            if (__any_sync(FULL, q.n > KnnCfg<K>::buf - 8)) {
                merge_fresh(nn, q, W, lane, ct);
                prune(q, nn.tau, KnnCfg<K>::buf - 8, W, lane, ct);
            }
            const float b2 = ok ? fminf(nn.tau, cap) : -1.0f;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float4 p = W.pts[t0 + e];
                const float d = dist2(qx, qy, qz, p.x, p.y, p.z);
                if (t0 + e < n && d <= b2) {
                    W.d[q.n][lane] = d;
                    W.idx[q.n][lane] = __float_as_int(p.w);
                    ++q.n;
                }
            }
        }
        __syncwarp();
        if (!merged) {  // the nearest points usually hold most of each list: merge them at once
            merged = true;
            merge_fresh(nn, q, W, lane, ct);
            prune(q, nn.tau, KnnCfg<K>::buf - 8, W, lane, ct);
        }
    };
    for (int it = 0; it < nr; ++it) {
        const uint32_t m = __reduce_min_sync(FULL, min(ok0, ok1));
        if (ok0 == m) ok0 = 0xffffffffu;
        if (ok1 == m) ok1 = 0xffffffffu;
        const int4 r = list[m & 0x7fu];
        const uint64_t P = (uint64_t)(uint32_t)r.z | ((uint64_t)(uint32_t)r.w << 32);
        float bl[3], bh[3];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) {
            const uint32_t Cax = gather3(P >> ax);
            axis_bounds(Cax << s, (uint32_t)min64((int64_t)M, ((int64_t)(Cax + 1) << s) - 1), inv_m, mn, range, pad,
                        bl[ax], bh[ax]);
        }
        const bool need = ok && box_dist2(qx, qy, qz, bl[0], bl[1], bl[2], bh[0], bh[1], bh[2]) <= fminf(nn.tau, cap);
        if (!__any_sync(FULL, need)) continue;
        ++ct.buckets;
        for (int off = 0; off < r.y;) {
            const int take = min(r.y - off, 32 - fill);
            if (lane < take) {
                const int32_t pi = r.x + off + lane;
                float4 p = __ldg(pts + pi);
                p.w = __int_as_float(pi);
                W.pts[fill + lane] = p;
            }
            fill += take;
            off += take;
            if (fill == 32) {
                test_chunk(32);
                fill = 0;
            }
        }
    }
    if (fill > 0) test_chunk(fill);
    return true;
}

__device__ __forceinline__ void neu_add(float& s, float& c, float x) {
    const float t = s + x;
    if (fabsf(s) >= fabsf(x)) c += (s - t) + x;
    else c += (x - t) + s;
    s = t;
}

// Normal of one query from its k neighbours, ascending, whose indices are in
// nbr[0], nbr[32], ... (the lane's column of the candidate indices, free once
// the search is done; rolled loops keep the code small for large k):
// centred covariance with compensated FP32 sums, FP32 Jacobi, FP64 redo when
// the relative eigengap (l1 - l0) / l2 is below `gap`, orientation towards
// the viewpoint (src/NormalEstimation.hpp:184-189).
__device__ __forceinline__ void estimate_normal(const int32_t* nbr, int k, const float4* __restrict__ pts,
                                                float qx, float qy, float qz, const QArgs& a, float* out,
                                                DevState* st) {
    float s[3] = {0.f, 0.f, 0.f}, c[3] = {0.f, 0.f, 0.f};
#pragma unroll 4
    for (int j = 0; j < k; ++j) {
        const float4 p = __ldg(pts + nbr[32 * j]);
        neu_add(s[0], c[0], p.x - qx);
        neu_add(s[1], c[1], p.y - qy);
        neu_add(s[2], c[2], p.z - qz);
    }
    const float inv_k = 1.0f / (float)k;
    const float m0 = (s[0] + c[0]) * inv_k, m1 = (s[1] + c[1]) * inv_k, m2 = (s[2] + c[2]) * inv_k;
    float cs[6] = {0, 0, 0, 0, 0, 0}, cc[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 4
    for (int j = 0; j < k; ++j) {
        const float4 p = __ldg(pts + nbr[32 * j]);
        const float r0 = (p.x - qx) - m0, r1 = (p.y - qy) - m1, r2 = (p.z - qz) - m2;
        neu_add(cs[0], cc[0], r0 * r0);
        neu_add(cs[1], cc[1], r0 * r1);
        neu_add(cs[2], cc[2], r0 * r2);
        neu_add(cs[3], cc[3], r1 * r1);
        neu_add(cs[4], cc[4], r1 * r2);
        neu_add(cs[5], cc[5], r2 * r2);
    }
    const float inv_den = 1.0f / (float)(k > 1 ? k - 1 : 1);
    float C[6];
#pragma unroll
    for (int e = 0; e < 6; ++e) C[e] = (cs[e] + cc[e]) * inv_den;
    float w[3], nv[3];
    eig3<float>(C, w, nv);
    float nx = nv[0], ny = nv[1], nz = nv[2];
    const float gap = (w[1] - w[0]) / fmaxf(fabsf(w[2]), FLT_MIN);
    if (!(gap >= a.gap)) {
        // near-degenerate neighbourhood: redo covariance and eigensolve in FP64
        double sd[3] = {0, 0, 0};
#pragma unroll 1
        for (int j = 0; j < k; ++j) {
            const float4 p = __ldg(pts + nbr[32 * j]);
            sd[0] += (double)p.x - (double)qx;
            sd[1] += (double)p.y - (double)qy;
            sd[2] += (double)p.z - (double)qz;
        }
        const double md[3] = {sd[0] / k, sd[1] / k, sd[2] / k};
        double Cd[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 1
        for (int j = 0; j < k; ++j) {
            const float4 p = __ldg(pts + nbr[32 * j]);
            const double r0 = ((double)p.x - (double)qx) - md[0];
            const double r1 = ((double)p.y - (double)qy) - md[1];
            const double r2 = ((double)p.z - (double)qz) - md[2];
            Cd[0] += r0 * r0; Cd[1] += r0 * r1; Cd[2] += r0 * r2;
            Cd[3] += r1 * r1; Cd[4] += r1 * r2; Cd[5] += r2 * r2;
        }
        const double dd = (double)(k > 1 ? k - 1 : 1);
#pragma unroll
        for (int e = 0; e < 6; ++e) Cd[e] /= dd;
        double wd[3], nd[3];
        eig3<double>(Cd, wd, nd);
        nx = (float)nd[0];
        ny = (float)nd[1];
        nz = (float)nd[2];
        atomicAdd(&st->counters[CNT_FP64], 1ull);
    }
    const float dot = (a.vx - qx) * nx + (a.vy - qy) * ny + (a.vz - qz) * nz;
    if (dot < 0.0f) { nx = -nx; ny = -ny; nz = -nz; }
    out[0] = nx;
    out[1] = ny;
    out[2] = nz;
}

__device__ __forceinline__ float warp_min(float v) {
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Walk of the search hierarchy for the warp's active lanes, depth first,
// nearest node first. The 32 children of a node are tested at once, one per
// lane, against the box of the warp's queries (its distance to a child's box
// never exceeds that of any query in it, by the same rounding chain); a child
// within the largest bound of the warp is then tested by every lane against
// its own query and bound. The first test is one pass for 32 nodes where the
// binary tree before it took a visit for every two (2M scene, k = 16: 43 tree
// visits and 12 buckets of about 60 points per warp became 19 visits of 32
// nodes and 21 leaves of about 20 points; search 3.08 -> 2.69 ms; 20M precision mix 20.8 -> 18.0 ms, both with the
// earlier lists). The second keeps warps whose queries lie far apart (their
// box covers what is between) from descending everywhere. Fetching the next
// sibling's box one step ahead was slower (3.01 ms): its registers and moves
// cost more than the load, which mostly hits L1.
// A lane's order key is its child's distance with the lane in the low 5 bits
// (rounded down, so still a lower bound); keys of the levels above wait in
// shared memory.
// Before the walk the warp offers the Morton window [w0, w1) around its
// queries to all of them, except the points [e0, e1) that a lane's list was
// filled with (w0 = w1: no seed). Window runs and leaves go through one copy
// of the scan and merge code: with a copy each, instruction fetch stalls
// doubled.
template <int K, bool EXACT, class WS>
__device__ __forceinline__ void search(Nearest<K, EXACT>& nn, Query& q, WS& W, int lane, Counters& ct,
                                       const float4* __restrict__ pts, const SNode* __restrict__ snodes,
                                       const QArgs& a, DevState* st, bool act, float cap, int32_t u, int32_t w0,
                                       int32_t w1, int32_t e0, int32_t e1, uint32_t& steps) {
    const float qx = q.x, qy = q.y, qz = q.z;
    constexpr uint32_t kNone = 0xffffffffu;
    // Siblings that pass the first test before each is tested by all 32 queries
    // at once. Most warps pass a few of 32; a warp across a Morton jump passes
    // nearly all, and a visit for each makes it the last to end: the 100k-point
    // k = 8 search took 237 us without this test, 168 us with it (24), 176 us at
    // 12. Large clouds, where other warps fill in, pay for it sooner: the 20M
    // precision mix 17.89 ms without, 18.04 at 24, 18.52 at 12.
    constexpr int kMaxLoose = 24;
    W.box_lo = make_float4(warp_min(act ? qx : INFINITY), warp_min(act ? qy : INFINITY), warp_min(act ? qz : INFINITY), 0.f);
    W.box_hi = make_float4(warp_max(act ? qx : -INFINITY), warp_max(act ? qy : -INFINITY), warp_max(act ? qz : -INFINITY), 0.f);
    const uint32_t step_cap = a.step_limit > 0 ? (uint32_t)a.step_limit : (uint32_t)min64(4 * (int64_t)u + 64, 0x7fffffff);
    float tau = act ? fminf(nn.tau, cap) : -1.0f;
    float tau_max = INFINITY;
    W.query()[lane] = make_float4(qx, qy, qz, tau);
    int l = __ldg(&st->top_level);
    const int top = l;
    uint32_t first = 0;                                       // the current siblings: [first, first + 32) of level l,
    const SNode* group = snodes + __ldg(&st->level_off[l]);   // from here on
    // order key of the lane's sibling
    auto order_key = [&]() -> uint32_t {
        const bool valid = first + lane < __ldg(&st->level_count[l]);
        const SNode* n = group + (valid ? lane : 0);
        const float4 lo = __ldg(&n->lo), hi = __ldg(&n->hi);
        const float4 ql = W.box_lo, qh = W.box_hi;
        const float gx = fmaxf(fmaxf(__fsub_rn(lo.x, qh.x), __fsub_rn(ql.x, hi.x)), 0.0f);
        const float gy = fmaxf(fmaxf(__fsub_rn(lo.y, qh.y), __fsub_rn(ql.y, hi.y)), 0.0f);
        const float gz = fmaxf(fmaxf(__fsub_rn(lo.z, qh.z), __fsub_rn(ql.z, hi.z)), 0.0f);
        float d = __fmaf_rn(gx, gx, __fmaf_rn(gy, gy, __fmul_rn(gz, gz)));
        bool reach = valid && d <= tau_max;
        if (__popc(__ballot_sync(FULL, reach)) > kMaxLoose) {
            // the box of the queries may hold much that no query is near:
            // take the distance of the nearest query that reaches the child
            d = INFINITY;
            reach = false;
#pragma unroll 1
            for (int i = 0; i < 32; ++i) {
                const float4 o = W.query()[i];
                const float di = box_dist2(o.x, o.y, o.z, lo.x, lo.y, lo.z, hi.x, hi.y, hi.z);
                if (di <= o.w) {
                    d = fminf(d, di);
                    reach = valid;
                }
            }
        }
        return reach ? (__float_as_uint(d) & ~31u) | (uint32_t)lane : kNone;
    };
    uint32_t key = kNone;
    int32_t next = w0;        // the window's next run
    bool started = false;     // the root's children are in `key`
    for (;;) {
        int32_t f = 0, cnt = 0;
        uint32_t needm = FULL;
        const bool window = next < w1;
        const bool own = window || w0 == w1;  // the lane's own [e0, e1) were offered so far, not the window
        if (window) {
            f = next;
            cnt = min(32, w1 - f);
            next += 32;
        } else {
            if (!started) {
                started = true;
                // nothing beyond the window: the tree has no more to offer
                if (w0 > 0 || w1 < u) {
                    tau_max = warp_max(tau);
                    W.query()[lane].w = tau;
                    __syncwarp();
                    key = order_key();
                    ++steps;
                }
            }
            // the next leaf that some lane needs
            for (;;) {
                const uint32_t m = __reduce_min_sync(FULL, key);
                if (m == kNone || __uint_as_float(m & ~31u) > tau_max) {  // nothing left here: up a level
                    if (l == top) break;
                    ++l;
                    first = (first / kFan) & ~31u;
                    group = snodes + __ldg(&st->level_off[l]) + first;
                    key = W.level_keys(l)[lane];
                    continue;
                }
                if (key == m) key = kNone;
                const float4 lo = __ldg(&group[m & 31u].lo), hi = __ldg(&group[m & 31u].hi);
                const float d = box_dist2(qx, qy, qz, lo.x, lo.y, lo.z, hi.x, hi.y, hi.z);
                needm = __ballot_sync(FULL, d <= tau);
                if (!needm) continue;
                if (l > 0) {
                    if (++steps > step_cap) {
                        if (lane == 0) set_err(&st->err, ERRBIT_SEARCH_LIMIT);
                        break;
                    }
                    W.level_keys(l)[lane] = key;
                    --l;
                    first = (first + (m & 31u)) * kFan;
                    group = snodes + __ldg(&st->level_off[l]) + first;
                    key = order_key();
                    continue;
                }
                f = __float_as_int(lo.w);
                if (f >= w0 && f + __float_as_int(hi.w) <= w1) continue;  // all of it was in the window (none: w1 = 0)
                cnt = __float_as_int(hi.w);
                if (cnt < 1 || cnt > kLeafMax || (uint32_t)f > (uint32_t)u - (uint32_t)cnt) {
                    if (lane == 0) set_err(&st->err, ERRBIT_BOUNDS);
                    cnt = 0;
                }
                break;
            }
            ct.buckets += cnt > 0;
        }
        const bool done = cnt == 0;
        const float before = tau;
        uint32_t hits = 0;
        if (!done)
            hits = scan_run(f, cnt, needm, own ? e0 : w0, own ? e1 : w1, q, tau, W, lane, pts);
        take_hits<K, EXACT>(
            hits, done || (window && next >= w1), done ? K : KnnCfg<K>::buf - 8,
            [&](int i, int32_t& idx) {
                const float* c = reinterpret_cast<const float*>(W.pts);
                const int o = 4 * (i >> 1) + (i & 1);
                idx = f + i;
                return make_float3(c[o], c[o + 2], c[64 + i]);
            },
            nn, q, tau, cap, W, lane, ct);
        __syncwarp();
        if (done) break;
        if (__any_sync(FULL, tau != before)) {
            tau_max = warp_max(tau);
            W.query()[lane].w = tau;
            __syncwarp();
        }
    }
}

// Row `row` of k values, 16 bytes at a time where rows are aligned to that. Into
// pinned host memory single words cross PCIe badly: lists of a 2M scene, k = 16,
// 3.87 ms, now 2.86 ms (into device memory 2.01 and 1.95 ms).
template <int K, class T, class Value>
__device__ __forceinline__ void put_row(T* out, int64_t row, int k, Value value) {
    T* o = out + row * k;
    if constexpr (K % 4 == 0) {
        if (k % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) {
#pragma unroll
            for (int j = 0; j < K; j += 4) {
                struct __align__(16) Four {
                    T v[4];
                };
                if (j < k) *reinterpret_cast<Four*>(o + j) = Four{value(j), value(j + 1), value(j + 2), value(j + 3)};
            }
            return;
        }
    }
#pragma unroll
    for (int j = 0; j < K; ++j)
        if (j < k) o[j] = value(j);
}

// The queries [q0, q0 + nq) of one warp: search, then the outputs.
// CELLS: the learned attempt may run the cell scan (a separate instantiation,
// launched only when the caller turned the cell scan on: compiled into the
// default kernels, its code alone slowed them by about 8%).
template <int K, bool EXACT, bool EXT, bool NORMALS, bool CELLS>
__device__ __forceinline__ void knn_warp(const float4* __restrict__ pts, const SNode* __restrict__ snodes,
                                         const uint64_t* __restrict__ codes, const QArgs& a, DevState* st,
                                         int64_t q0, int nq, WarpSmem<KnnCfg<K>::buf, CELLS>& W, int lane) {
    constexpr int kBuf = KnnCfg<K>::buf;
    static_assert(K + 8 <= kBuf, "k candidates and room for hits");
    const int64_t u = a.device_count ? (int64_t)st->u : a.u;
    const int64_t count = a.device_count ? u : a.count;
    if (q0 >= count) return;  // whole warp
    const int64_t qo = q0 + lane;
    const bool active = lane < nq && qo < count;
    float qx, qy, qz;
    int64_t center;   // tree index of the warp's first query; foreign queries: the lane's place among the codes
    int64_t row = qo;  // of the outputs
    if (EXT) {
        row = active ? qo : q0;
        uint64_t key = 0;
        if (a.order) {
            key = __ldg(a.order + row);
            row = (int64_t)(key & ((1u << 30) - 1));
            if (row >= count) {  // the sort failed
                set_err(&st->err, ERRBIT_BOUNDS);
                row = q0;
            }
        }
        qx = __ldg(a.ext + 3 * row);
        qy = __ldg(a.ext + 3 * row + 1);
        qz = __ldg(a.ext + 3 * row + 2);
        center = a.order ? min64(u, (int64_t)(key >> (kOrderShift + a.order_shift)))
                         : code_position(codes, u, query_to_code(qx, qy, qz, st->min_coord, st->range, a.code_bits));
    } else {
        const float4 p = __ldg(pts + a.start + (active ? qo : q0));
        qx = p.x;
        qy = p.y;
        qz = p.z;
        center = a.start + q0;
    }
    // the seed window: the warp's, around its queries' places. Foreign queries
    // can lie far apart: each lane then only fills its list around its own place.
    int64_t from = center, to = center + nq;
    bool lone = false;
    if (EXT) {
        const int first = (int)__reduce_min_sync(FULL, active ? (unsigned)center : UINT_MAX);
        const int last = (int)__reduce_max_sync(FULL, active ? (unsigned)center : 0u);
        lone = last - first > kWindowSpan;
        from = first - 16;
        to = last + 16;
    }
    const int64_t w0 = lone ? 0 : max64(0, from - a.seed_halo), w1 = lone ? u : min64(u, to + a.seed_halo);

    Nearest<K, EXACT> nn;
    Query q{qx, qy, qz, a.k, 0, 0};
    Counters ct;
    uint32_t steps = 0;
    // With a learned radius, attempt 0 searches with the predicted bound as a
    // cap; a lane whose k-th neighbour lies beyond its cap (the cap pruned
    // points that could belong to its k best) is searched again without it.
    const bool learned = !EXT && a.learned_r2 != nullptr;
    const float cap0 = (learned && active) ? __ldg(a.learned_r2 + qo) : INFINITY;
    bool act = active;
    // Nothing is near a query with a NaN coordinate: no distance passes its
    // bound and none tightens it, so a search would scan the whole tree for it.
    // Nor is anything nearer than the rest to one whose every squared distance
    // overflows: the lowest indices win the tie. The decoded points lie in the
    // cube [lo, hi]^3, whose box distance is no larger than any of theirs.
    auto out_of_range = [&]() {
        const float lo = st->min_coord, hi = __fmaf_rn(1.0f, st->range, lo);
        return box_dist2(qx, qy, qz, lo, lo, lo, hi, hi, hi) == INFINITY;
    };
    if (EXT) act = act && qx == qx && qy == qy && qz == qz && !out_of_range();
    nn.init();
    for (int attempt = learned ? 0 : 1; attempt < 2; ++attempt) {
        if (EXT && !__any_sync(FULL, act)) break;
        const float cap = attempt == 0 ? cap0 : INFINITY;
        const bool seed = attempt == 1 || !a.learned_skip_seed;
        const int64_t sw0 = seed && !lone ? w0 : 0, sw1 = seed && !lone ? w1 : 0;  // points offered by the seed
        if (act) {
            nn.init();
            q.n = q.merged = 0;
        }
        // learned attempt as a cell scan (falls back to the capped tree walk)
        bool scanned = false;
        if constexpr (CELLS)
            scanned = attempt == 0 && a.cell_lut != nullptr &&
                      cell_scan<K, EXACT>(nn, q, W, lane, ct, pts, codes, a, st, act, a.start + (active ? qo : q0),
                                          cap);
        __syncwarp();
        int32_t e0 = 0, e1 = 0;
        if (seed && act) {
            // Seed: K points of the Morton window around the lane's own
            // position fill its list; the search offers the rest of the window.
            const int64_t at = EXT ? center : center + lane;
            e0 = (int32_t)max64(w0, min64(at - (K / 2 - 1), w1 - K));
            e1 = (int32_t)min64(w1, e0 + K);
#pragma unroll
            for (int t = 0; t < K; ++t) {
                nn.d[t] = INFINITY;
                if (e0 + t < e1) {
                    const float4 p = __ldg(pts + e0 + t);
                    nn.d[t] = dist2(qx, qy, qz, p.x, p.y, p.z);
                    W.d[t][lane] = nn.d[t];
                    W.idx[t][lane] = e0 + t;
                }
            }
            nn.sort_filled(a.k);
            q.n = q.merged = e1 - e0;
            ct.cand += q.n;
            if (cap < INFINITY) {  // those beyond a learned cap do not count
#pragma unroll
                for (int t = 0; t < K; ++t) ct.cand -= nn.d[t] > cap && nn.d[t] < INFINITY;
            }
        }
        if (!CELLS || !scanned)
            search<K, EXACT>(nn, q, W, lane, ct, pts, snodes, a, st, act, cap, (int32_t)u, (int32_t)sw0, (int32_t)sw1, e0,
                             e1, steps);
        else {
            merge_fresh(nn, q, W, lane, ct);
            prune(q, nn.tau, K, W, lane, ct);
        }
        if (attempt == 0) {
            // a lane the cell scan could not serve (its cap is +inf or not a
            // number) was offered nothing: search it again as a miss
            const bool unserved = scanned && !(cap >= 0.0f && cap < INFINITY);
            const bool miss = act && (unserved || !(nn.tau <= cap));
            ct.lmiss += miss;
            act = miss;
            if (!__any_sync(FULL, act)) break;
        }
    }
    {
        const unsigned cand = __reduce_add_sync(FULL, (unsigned)ct.cand);
        const unsigned ins = __reduce_add_sync(FULL, (unsigned)ct.ins);
        const unsigned lmiss = __reduce_add_sync(FULL, (unsigned)ct.lmiss);
        if (lane == 0) {
            W.count[CNT_NODES] += steps;
            W.count[CNT_BUCKETS] += ct.buckets;
            W.count[CNT_MERGE] += ct.merge;
            W.count[CNT_CANDIDATES] += cand;
            W.count[CNT_INSERTS] += ins;
            W.count[CNT_LEARNED_MISS] += lmiss;
            if constexpr (CELLS) {
                W.count[CNT_CELL_WARPS] += ct.cells;
                W.count[CNT_CELL_FALLBACK] += ct.cell_fallback;
                W.count[CNT_CELL_LOOKUPS] += ct.cell_lookups;
                W.count[CNT_CELL_POINTS] += ct.cell_points;
            }
        }
    }
    if (!active) return;

    // A query with a NaN coordinate gets points of its window, at distance NaN;
    // one out of range the first points of the tree.
    const bool lost = q.n == 0 && !(EXT && qx == qx && qy == qy && qz == qz);
    if (q.n == 0)
        for (const int64_t first = lost ? w0 : 0, end = lost ? w1 : u; q.n < K && first + q.n < end; ++q.n) {
            W.d[q.n][lane] = INFINITY;
            W.idx[q.n][lane] = (int32_t)(first + q.n);
        }
    // the k nearest in the lists' order: by distance, then by index
    unsigned long long key[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        key[j] = j < q.n ? pack_key(W.d[j][lane], W.idx[j][lane]) : kEmptyKey;
    }
    sort_values(key);
    // fewer than k points in the tree: repeat entry 0 (src/Octree.hpp:181-191)
    int32_t nbr[K];
#pragma unroll
    for (int j = 0; j < K; ++j) {
        if (j > 0 && key[j] == kEmptyKey) key[j] = key[0];
        nbr[j] = key_idx(key[j]);
    }
    if (!NORMALS && a.out_idx) put_row<K>(a.out_idx, row, a.k, [&](int j) { return nbr[j]; });
    if (!NORMALS && a.out_d2)
        put_row<K>(a.out_d2, row, a.k, [&](int j) { return lost ? __int_as_float(0x7fc00000) : key_d(key[j]); });
    if (NORMALS) {
#pragma unroll
        for (int j = 0; j < K; ++j) W.idx[j][lane] = nbr[j];  // this lane's column only
        estimate_normal(&W.idx[0][lane], a.k, pts, qx, qy, qz, a, a.out_normals + 3 * qo, st);
    }
}

// How many of the foreign queries from q0 on, one to a warp as given, the warp
// takes: its one, or, as the first of an aligned group of 32 within a box of
// `close` tree ranges, all of the group (the others then take none), since
// such share nodes, leaves and most candidates. 17,000 queries within a point
// spacing of each other in a 2M-point scene took 138 us (k = 8) and 449 us
// (k = 32) one to a warp, now 50 and 81 us.
__device__ __forceinline__ int foreign_share(const QArgs& a, const DevState* st, int64_t q0, int lane) {
    const int64_t g0 = q0 & ~(int64_t)31;
    const float* q = a.ext + 3 * min64(g0 + lane, a.count - 1);
    const float x = __ldg(q), y = __ldg(q + 1), z = __ldg(q + 2);
    const float extent =
        fmaxf(fmaxf(warp_max(x) - warp_min(x), warp_max(y) - warp_min(y)), warp_max(z) - warp_min(z));
    if (!(extent <= a.close * st->range)) return 1;
    return q0 == g0 ? 32 : 0;
}

// Persistent: the grid is the resident blocks and each warp takes its next
// queries from a counter. With a block per four warps' queries a block kept its
// registers and shared memory until its slowest warp ended, and 15 of 20
// resident warps were active on average: the 2M scene's k = 16 search took
// 2.68 ms, 2.35 ms persistent.
template <int K, bool EXACT, bool EXT, bool NORMALS, bool CELLS>
__global__ void __launch_bounds__(KnnCfg<K>::threads, KnnCfg<K>::min_blocks)
    k_knn(const float4* __restrict__ pts, const SNode* __restrict__ snodes,
                                                     const uint64_t* __restrict__ codes, QArgs a, DevState* st) {
    extern __shared__ __align__(16) unsigned char knn_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    using WS = WarpSmem<KnnCfg<K>::buf, CELLS>;
    WS& W = reinterpret_cast<WS*>(knn_smem)[warp];
    if (lane < kQueryCounters) W.count[lane] = 0;
    __syncwarp();
    const int64_t n = a.device_count ? (int64_t)st->u : a.count;
    const bool listed = EXT ? a.order != nullptr : !CELLS && a.parts != nullptr;
    if (lane == 0) {  // kept here: a register less across the search
        W.whole = listed ? __ldg(&st->items) : (uint32_t)((n + a.warp_queries - 1) / a.warp_queries);
        W.items = listed && !EXT ? W.whole + __ldg(&st->parts) : W.whole;
    }
    __syncwarp();
    uint32_t item = blockIdx.x * KnnCfg<K>::warps + warp;
    while (item < W.items) {
        int64_t q0 = (int64_t)item * a.warp_queries;
        int nq = a.warp_queries;
        if (listed) {
            const uint64_t e = __ldg(EXT ? a.items + item : item < W.whole ? a.parts + item : a.parts_end - 1 - (item - W.whole));
            q0 = (int64_t)(uint32_t)e;
            nq = (int)(e >> 32);
        } else if (EXT && a.close > 0.0f) {
            nq = foreign_share(a, st, q0, lane);
        }
        if (!EXT || nq > 0) knn_warp<K, EXACT, EXT, NORMALS, CELLS>(pts, snodes, codes, a, st, q0, nq, W, lane);
        __syncwarp();
        if (lane == 0) item = gridDim.x * KnnCfg<K>::warps + atomicAdd(&st->work, 1u);
        item = __shfl_sync(FULL, item, 0);
    }
    if (lane < kQueryCounters && W.count[lane]) atomicAdd(&st->counters[lane], (unsigned long long)W.count[lane]);
}

// Persistent kernel over many clouds that share k: each warp takes the next
// 32-query item from a global counter until all are taken. Items are laid out
// cloud by cloud in the order of `clouds` (largest first), so the large clouds
// start first and the small ones fill the tail. Each cloud's size is read on
// the device from its own build state.
// Block shape of the persistent launch: W warps per block, with the
// resident-block target scaled so that ptxas gets the same register budget
// per thread as the per-k default shape (KnnCfg).
template <int K, int W>
struct BatchCfg {
    static constexpr int threads = 32 * W;
    static constexpr int min_blocks =
        (KnnCfg<K>::min_blocks * KnnCfg<K>::warps) / W > 0 ? (KnnCfg<K>::min_blocks * KnnCfg<K>::warps) / W : 1;
};

template <int K, bool EXACT, int NW>
__global__ void __launch_bounds__(BatchCfg<K, NW>::threads, BatchCfg<K, NW>::min_blocks)
    k_knn_batch(const BatchCloud* __restrict__ clouds, int n_clouds,
                                                           int64_t n_items, unsigned long long* counter, QArgs a) {
    extern __shared__ __align__(16) unsigned char knn_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    using WS = WarpSmem<KnnCfg<K>::buf>;
    WS& W = reinterpret_cast<WS*>(knn_smem)[warp];
    if (lane < kQueryCounters) W.count[lane] = 0;
    __syncwarp();
    for (;;) {
        unsigned long long item = 0;
        if (lane == 0) item = atomicAdd(counter, 1ull);
        item = __shfl_sync(FULL, item, 0);
        if (item >= (unsigned long long)n_items) break;
        int lo = 0, hi = n_clouds - 1;  // last cloud whose first item is <= item
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if ((unsigned long long)__ldg(&clouds[mid].item0) <= item) lo = mid;
            else hi = mid - 1;
        }
        const BatchCloud d = clouds[lo];
        QArgs ca = a;
        ca.out_normals = d.out_normals;
        ca.start = 0;
        ca.device_count = 1;
        knn_warp<K, EXACT, false, true, false>(d.pts, d.snodes, nullptr, ca, d.st, ((int64_t)item - d.item0) * 32, 32,
                                               W, lane);
        __syncwarp();
        if (lane < kQueryCounters && W.count[lane]) {
            atomicAdd(&d.st->counters[lane], (unsigned long long)W.count[lane]);
            W.count[lane] = 0;
        }
        __syncwarp();
    }
}

// Work items of the tree's own points [start, start + count): 32 at a time, cut
// where the Morton order jumps and then into `per`. A jump is a gap between adjacent
// points of more than `jump` times the median gap of the 32; the three widest count.
// A warp across a jump walks two regions and what lies between, and a call of a few
// rounds of warps ends with its slowest: normals of 110k points of a scene, k = 8,
// lasted 249 us for one warp of 3438 (99 of 100 end within 120 us, half within 66).
// Over scenes, cubes, mixtures and precision mixes, against none cut (gaps of 5, 6, 8,
// 10, 12, 16 medians): 45k points, k = 8: 0.77, 0.79, 0.84, 0.86, 0.87, 0.92; 110k, k =
// 16: 0.92, 0.92, 0.82, 0.85, 0.87, 0.92; 300k, k = 16: 1.06, 1.01, 0.98, 0.95, 0.96,
// 0.95. A plane or a line has few: 110k points, k = 16, 131 and 66 us uncut, 172 and 86
// at 5, 134 and 72 at 10. (Judged by the codes' common prefixes, 8 bits below the
// median, a line of 200k points was cut everywhere: 158 -> 306 us.)
// Whole items fill the list from its front and parts, which end sooner, from its
// back (room entries on), so that parts are what starts late when not all fit at
// once.
constexpr int kItemBytes = 2;  // of the list, per point: 4 + 32 / 8 - 1 parts of 8 bytes in 32 points
__global__ void __launch_bounds__(256) k_point_items(const float4* __restrict__ pts, int64_t start, int64_t n,
                                                     int per, float jump, uint64_t* __restrict__ items, int64_t room,
                                                     DevState* st) {
    __shared__ uint32_t s_at[2][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const float4 p = __ldg(pts + start + min64(i, n - 1));
    float gap = fmaxf(fmaxf(fabsf(p.x - __shfl_up_sync(FULL, p.x, 1)), fabsf(p.y - __shfl_up_sync(FULL, p.y, 1))),
                      fabsf(p.z - __shfl_up_sync(FULL, p.z, 1)));
    if (lane == 0 || i >= n) gap = 0.0f;
    uint32_t median = 0;  // 16 gaps are at least this, to an eighth (0: fewer, or of equal points)
#pragma unroll
    for (uint32_t b = 1u << 30; b >= 1u << 20; b >>= 1)
        if (__popc(__ballot_sync(FULL, __float_as_uint(gap) >= (median | b))) >= 16) median |= b;
    uint32_t cuts = 0;
    if (median > 0) {
        float most = jump * __uint_as_float(median);
        do {
            cuts = __ballot_sync(FULL, gap > most);
            most *= 2.0f;
        } while (__popc(cuts) > 3);
    }
    cuts |= 1u;
    const int from = 31 - __clz(cuts & (2u * (1u << lane) - 1u));  // where the lane's part begins
    const uint32_t firsts = __ballot_sync(FULL, i < n && ((lane - from) & (per - 1)) == 0);
    const uint32_t later = lane < 31 ? firsts >> (lane + 1) : 0u;
    const int64_t size = later ? __ffs(later) : min64(32, n - (i - lane)) - lane;
    const bool first = (firsts >> lane) & 1u;
    const uint32_t whole = __ballot_sync(FULL, first && size == per), part = firsts & ~whole;
    if (lane == 0) {
        s_at[0][warp] = __popc(whole);
        s_at[1][warp] = __popc(part);
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        uint32_t* at = s_at[threadIdx.x];
        uint32_t total = 0;
        for (int w = 0; w < 8; ++w) {
            const uint32_t c = at[w];
            at[w] = total;
            total += c;
        }
        const uint32_t base = atomicAdd(threadIdx.x == 0 ? &st->items : &st->parts, total);
        for (int w = 0; w < 8; ++w) at[w] += base;
    }
    __syncthreads();
    if (first) {
        const bool w = (whole >> lane) & 1u;
        const int64_t at = w ? s_at[0][warp] + __popc(whole & lanemask_lt())
                             : room - 1 - (s_at[1][warp] + __popc(part & lanemask_lt()));
        items[at] = ((uint64_t)size << 32) | (uint64_t)i;
    }
}

template <int K, bool EXACT, bool EXT, bool NORMALS, bool CELLS = false>
cudaError_t launch_one(const BuildBufs& b, const QArgs& a, unsigned blocks, cudaStream_t s, int num_sms) {
    constexpr int smem = (int)sizeof(WarpSmem<KnnCfg<K>::buf, CELLS>) * KnnCfg<K>::warps;
    cudaError_t e = cudaFuncSetAttribute(k_knn<K, EXACT, EXT, NORMALS, CELLS>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_knn<K, EXACT, EXT, NORMALS, CELLS>, KnnCfg<K>::threads, smem);
    if (e != cudaSuccess) return e;
    const unsigned resident = (unsigned)(per_sm > 0 ? per_sm : 1) * (unsigned)num_sms;
    if (blocks > resident) blocks = resident;
    k_knn<K, EXACT, EXT, NORMALS, CELLS><<<blocks, KnnCfg<K>::threads, smem, s>>>(b.pts4, b.snodes, b.codes, a,
                                                                                   b.st);
    return cudaGetLastError();
}

template <int K, bool EXACT>
cudaError_t launch_k(const BuildBufs& b, const QArgs& a, bool ext, bool normals, cudaStream_t s, int num_sms) {
    // Cut items are more than this; while all warps fit at once none of them may
    // wait for a warp to end (an item that did started 50 us late).
    const int64_t warps = (a.count + a.warp_queries - 1) / a.warp_queries * (!ext && a.parts ? 2 : 1);
    const unsigned blocks = (unsigned)((warps + KnnCfg<K>::warps - 1) / KnnCfg<K>::warps);
    if (ext) return launch_one<K, EXACT, true, false>(b, a, blocks, s, num_sms);
    if (a.cell_lut && !a.parts) {
        if (normals) return launch_one<K, EXACT, false, true, true>(b, a, blocks, s, num_sms);
        return launch_one<K, EXACT, false, false, true>(b, a, blocks, s, num_sms);
    }
    if (normals) return launch_one<K, EXACT, false, true>(b, a, blocks, s, num_sms);
    return launch_one<K, EXACT, false, false>(b, a, blocks, s, num_sms);
}

template <int K, bool EXACT, int NW>
cudaError_t launch_batch_w(const BatchCloud* clouds, int n_clouds, int64_t n_items, unsigned long long* counter,
                           const QArgs& a, cudaStream_t s, int num_sms, int blocks_per_sm) {
    constexpr int threads = BatchCfg<K, NW>::threads;
    constexpr int smem = (int)sizeof(WarpSmem<KnnCfg<K>::buf>) * NW;
    cudaError_t e =
        cudaFuncSetAttribute(k_knn_batch<K, EXACT, NW>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_knn_batch<K, EXACT, NW>, threads, smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) per_sm = 1;
    if (blocks_per_sm > 0 && blocks_per_sm < per_sm) per_sm = blocks_per_sm;
    const int64_t want = (n_items + NW - 1) / NW;
    const int64_t resident = (int64_t)per_sm * num_sms;
    const unsigned blocks = (unsigned)(want < resident ? want : resident);
    e = cudaMemsetAsync(counter, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    k_knn_batch<K, EXACT, NW><<<blocks, threads, smem, s>>>(clouds, n_clouds, n_items, counter, a);
    return cudaGetLastError();
}

// The per-k default block shape, or the other one of 2 and 4 warps.
template <int K, bool EXACT>
cudaError_t launch_batch(const BatchCloud* clouds, int n_clouds, int64_t n_items, unsigned long long* counter,
                         const QArgs& a, cudaStream_t s, int num_sms, int blocks_per_sm, int warps) {
    constexpr int def = KnnCfg<K>::warps;
    constexpr int alt = def == 4 ? 2 : 4;
    if (warps == alt) return launch_batch_w<K, EXACT, alt>(clouds, n_clouds, n_items, counter, a, s, num_sms,
                                                           blocks_per_sm);
    return launch_batch_w<K, EXACT, def>(clouds, n_clouds, n_items, counter, a, s, num_sms, blocks_per_sm);
}

// lut[j] = lower bound of j << sh in the u sorted unique codes, for j in
// [0, n_ent]; the code count u is read on the device from the build state.
__global__ void __launch_bounds__(256) k_cell_lut(const uint64_t* __restrict__ codes, const DevState* st, int sh,
                                                  int64_t n_ent, uint32_t* __restrict__ lut) {
    const uint32_t u = (uint32_t)st->u;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j <= n_ent;
         j += (int64_t)gridDim.x * blockDim.x) {
        lut[j] = j == n_ent ? u : lower_bound_codes(codes, 0u, u, (uint64_t)j << sh);
    }
}

}  // namespace

cudaError_t enqueue_cell_lut(const BuildBufs& b, int code_bits, int level, uint32_t* lut, cudaStream_t s,
                             int num_sms) {
    const int bpa = code_bits / 3;
    if (level < 1 || level > bpa || level > 10) return cudaErrorInvalidValue;
    const int64_t n_ent = (int64_t)1 << (3 * level);
    const int64_t want = (n_ent + 256) / 256;
    const unsigned blocks = (unsigned)(want < (int64_t)num_sms * 16 ? want : (int64_t)num_sms * 16);
    k_cell_lut<<<blocks, 256, 0, s>>>(b.codes, b.st, 3 * (bpa - level), n_ent, lut);
    return cudaGetLastError();
}

__global__ void k_batch_collect(const DevState* __restrict__ st, int n, unsigned long long* __restrict__ u_out,
                                uint32_t* __restrict__ err_out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    u_out[i] = st[i].u;
    err_out[i] = st[i].err;
}

cudaError_t enqueue_batch_collect(const DevState* st, int n, unsigned long long* u_out, uint32_t* err_out,
                                  cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    k_batch_collect<<<(n + 127) / 128, 128, 0, s>>>(st, n, u_out, err_out);
    return cudaGetLastError();
}

cudaError_t enqueue_query_batch(const BatchCloud* clouds, int n_clouds, int64_t n_items, unsigned long long* counter,
                                const QueryParams& q, cudaStream_t s, int num_sms) {
    if (n_clouds <= 0 || n_items <= 0) return cudaSuccess;
    if (q.k < 1 || q.k > 32) return cudaErrorInvalidValue;
    QArgs a{};
    a.k = q.k;
    a.vx = q.vx;
    a.vy = q.vy;
    a.vz = q.vz;
    a.gap = q.eigengap_fp64;
    a.code_bits = q.code_bits;
    a.seed_halo = q.seed_halo < 0 ? 0 : (q.seed_halo > kMaxHalo ? kMaxHalo : q.seed_halo);
    a.device_count = 1;
    a.warp_queries = 32;
    const int bps = q.batch_blocks_per_sm, wpb = q.batch_warps_per_block;
    switch (q.k) {
        case 8: return launch_batch<8, true>(clouds, n_clouds, n_items, counter, a, s, num_sms, bps, wpb);
        case 10: return launch_batch<10, true>(clouds, n_clouds, n_items, counter, a, s, num_sms, bps, wpb);
        case 16: return launch_batch<16, true>(clouds, n_clouds, n_items, counter, a, s, num_sms, bps, wpb);
        case 32: return launch_batch<32, true>(clouds, n_clouds, n_items, counter, a, s, num_sms, bps, wpb);
        default: break;
    }
    if (q.k <= 4) return launch_batch<4, false>(clouds, n_clouds, n_items, counter, a, s, num_sms, bps, wpb);
    if (q.k <= 8) return launch_batch<8, false>(clouds, n_clouds, n_items, counter, a, s, num_sms, bps, wpb);
    if (q.k <= 12) return launch_batch<12, false>(clouds, n_clouds, n_items, counter, a, s, num_sms, bps, wpb);
    if (q.k <= 16) return launch_batch<16, false>(clouds, n_clouds, n_items, counter, a, s, num_sms, bps, wpb);
    if (q.k <= 24) return launch_batch<24, false>(clouds, n_clouds, n_items, counter, a, s, num_sms, bps, wpb);
    return launch_batch<32, false>(clouds, n_clouds, n_items, counter, a, s, num_sms, bps, wpb);
}

int queries_per_warp(int64_t count, int num_sms, bool foreign) {
    // Few queries: fewer per warp, down to one, until there are ten warps per
    // SM. 32 queries of one warp mostly wait for one another (the union of
    // their nodes, the longest of their lists), and a small call lasts as long
    // as one warp: 2k points, k = 8, 74 us with 32 queries per warp and 39 us
    // with one; 10k points, k = 16, 162 and 115 us (eight per warp). With 20
    // warps per SM as the aim the wider spread costs more than it shortens
    // (10k points 141 us, 40k points 230 against 197 us).
    // Foreign queries in order share less: 40 warps per SM (near a 2M-point
    // scene, k = 8, 4 / 8 / 16 / 32 to a warp: 30k of them 281, 341, 536, 790 us;
    // 60k 429, 413, 554, 852; 100k 548, 472, 466, 1068; 250k 859, 763, 702, 656).
    int per = 32;
    while (per > 1 && (count + per - 1) / per < (int64_t)(foreign ? 40 : 10) * num_sms) per /= 2;
    return per;
}

bool list_points(int64_t count, int k, int num_sms) {
    // At four and fewer per warp there is little to cut; many rounds of warps hide
    // their slowest, and the parts' work adds up, the more so the longer the lists
    // (normals of precision mixes, of the time without the list, k = 4, 8, 16, 32:
    // 130k points 0.76, 0.76, 0.76, 0.79; 220k 0.78, 0.83, 0.91, 1.00; 300k 0.93, 1.00,
    // 1.05, 1.12; scenes 300k 0.88, 0.87, 0.89, 0.94; a scene of 207k, k = 31: 1.09).
    const int most = k <= 8 ? 2600 : (k <= 16 ? 1500 : 750);
    return queries_per_warp(count, num_sms, false) >= 8 && count <= (int64_t)most * num_sms;
}

bool order_foreign(int64_t count, int64_t u, int k, int num_sms) {
    // The order takes about 60 us. Queries near a 2M-point scene, one to a warp as
    // given and in order, k = 1, 8, 16, 32: 20k of them 145, 220, 320, 694 us and
    // 200, 240, 317, 541 us; 30k 196, 294, 447, 978 and 211, 281, 377, 627; 40k
    // 249, 383, 580, 1297 and 233, 322, 441, 775.
    return u > kTinyTree && count >= (int64_t)(k <= 16 ? 180 : 120) * num_sms;
}

cudaError_t enqueue_query(const BuildBufs& b, const QueryParams& q, cudaStream_t s, int num_sms) {
    if (q.count <= 0) return cudaSuccess;
    if (q.k < 1 || q.k > 32) return cudaErrorInvalidValue;
    if (q.compat) return enqueue_query_compat(b, q, s, num_sms);
    QArgs a;
    a.k = q.k;
    a.start = q.start;
    a.count = q.count;
    a.u = q.u;
    a.out_idx = q.out_idx;
    a.out_d2 = q.out_d2;
    a.out_normals = q.out_normals;
    a.vx = q.vx;
    a.vy = q.vy;
    a.vz = q.vz;
    a.gap = q.eigengap_fp64;
    a.code_bits = q.code_bits;
    a.seed_halo = q.seed_halo;
    a.learned_skip_seed = q.learned_skip_seed;
    a.device_count = q.device_count;
    a.step_limit = q.step_limit;
    if (q.ext_queries) {
        a.ext = q.ext_queries;
        a.order = q.order;
        a.order_shift = q.order_shift;
        a.items = q.items;
        // queries as given: close ones gain once there are more than warps fit;
        // a box of the tree's point spacing, were the points spread over its cube
        a.close = q.count > 20 * num_sms && q.u > kTinyTree ? 1.0f / cbrtf((float)q.u) : 0.0f;
    } else {
        a.parts = nullptr;
        a.learned_r2 = q.learned_r2;
        a.cell_lut = q.learned_r2 ? q.cell_lut : nullptr;
        a.lut_shift = q.lut_shift;
        a.cell_pmax = q.cell_pmax;
        a.cell_span = q.cell_span < 2 ? 2 : (q.cell_span > 4 ? 4 : q.cell_span);
    }
    if (a.seed_halo > kMaxHalo) a.seed_halo = kMaxHalo;
    if (a.seed_halo < 0) a.seed_halo = 0;
    const bool foreign = q.ext_queries && q.u > kTinyTree;
    a.warp_queries = foreign && !q.order ? 1 : queries_per_warp(q.count, num_sms, foreign);
    const bool ext = q.ext_queries != nullptr;
    if (!ext && !a.cell_lut && !q.device_count && list_points(q.count, q.k, num_sms)) {
        uint64_t* items = reinterpret_cast<uint64_t*>(b.scratch);  // the build is done with it
        const int64_t room = q.count * kItemBytes / (int64_t)sizeof(uint64_t);
        k_point_items<<<(unsigned)((q.count + 255) / 256), 256, 0, s>>>(
            b.pts4, q.start, q.count, a.warp_queries, q.count <= (int64_t)750 * num_sms ? 8.0f : 10.0f, items, room,
            b.st);
        a.parts = items;
        a.parts_end = items + room;
    }
    const bool nrm = q.out_normals != nullptr && !ext;
    switch (q.k) {
        case 8: return launch_k<8, true>(b, a, ext, nrm, s, num_sms);
        case 10: return launch_k<10, true>(b, a, ext, nrm, s, num_sms);
        case 16: return launch_k<16, true>(b, a, ext, nrm, s, num_sms);
        case 32: return launch_k<32, true>(b, a, ext, nrm, s, num_sms);
        default: break;
    }
    if (q.k <= 4) return launch_k<4, false>(b, a, ext, nrm, s, num_sms);
    if (q.k <= 8) return launch_k<8, false>(b, a, ext, nrm, s, num_sms);
    if (q.k <= 12) return launch_k<12, false>(b, a, ext, nrm, s, num_sms);
    if (q.k <= 16) return launch_k<16, false>(b, a, ext, nrm, s, num_sms);
    if (q.k <= 24) return launch_k<24, false>(b, a, ext, nrm, s, num_sms);
    return launch_k<32, false>(b, a, ext, nrm, s, num_sms);
}

}  // namespace shapex
