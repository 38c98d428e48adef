// Build stages of the normal-estimation path on sm_100a:
//   bbox -> Morton encode (+ digit histograms) -> onesweep LSD radix sort ->
//   dedup + decode -> Karras radix tree -> search boxes -> octree.
// Each kernel cites the reference stage it replaces (paths relative to the
// reference project root).

#include <cfloat>
#include <cstdint>

#include "pipeline.cuh"

namespace shapex {

namespace {

constexpr uint32_t LB_AGG = 1u << 30;
constexpr uint32_t LB_PRE = 2u << 30;
constexpr uint32_t LB_VAL = (1u << 30) - 1;
constexpr unsigned long long LB64_AGG = 1ull << 62;
constexpr unsigned long long LB64_PRE = 2ull << 62;
constexpr unsigned long long LB64_VAL = (1ull << 62) - 1;

__device__ __forceinline__ float warp_min(float v) {
    for (int o = 16; o; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v) {
    const int lane = threadIdx.x & 31;
    for (int o = 1; o < 32; o <<= 1) {
        T t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    return v;
}

// Block-wide exclusive scan (blockDim.x = NT, multiple of 32). Returns the
// thread's exclusive prefix; *total receives the block sum.
template <int NT, typename T>
__device__ __forceinline__ T block_excl_scan(T v, T* smem_warp, T* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T inc = warp_incl_scan(v);
    if (lane == 31) smem_warp[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        T w = (lane < NT / 32) ? smem_warp[lane] : T(0);
        T wi = warp_incl_scan(w);
        if (lane < NT / 32) smem_warp[lane] = wi - w;
        if (lane == NT / 32 - 1) smem_warp[NT / 32] = wi;
    }
    __syncthreads();
    T r = inc - v + smem_warp[warp];
    *total = smem_warp[NT / 32];
    __syncthreads();
    return r;
}

// ---------------------------------------------------------------------------
// bbox: replaces 3x DeviceReduce::Max + 3x DeviceReduce::Min and the host
// min/max of src/RadixTree.cu:218-241 with one pass over x, y, z producing a
// single isotropic [min, max]. Also rejects NaN/Inf.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_bbox(const float* __restrict__ x, const float* __restrict__ y,
                                              const float* __restrict__ z, int64_t n, DevState* st) {
    float lo = FLT_MAX, hi = -FLT_MAX;
    bool bad = false;
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    auto take = [&](float v) {
        bad |= !isfinite(v);
        lo = fminf(lo, v);
        hi = fmaxf(hi, v);
    };
    const bool vec = (((uintptr_t)x | (uintptr_t)y | (uintptr_t)z) & 15) == 0;
    int64_t done = 0;
    if (vec) {
        const int64_t n4 = n >> 2;
        const float4* x4 = reinterpret_cast<const float4*>(x);
        const float4* y4 = reinterpret_cast<const float4*>(y);
        const float4* z4 = reinterpret_cast<const float4*>(z);
        for (int64_t i = tid; i < n4; i += stride) {
            const float4 a = __ldcs(x4 + i), b = __ldcs(y4 + i), c = __ldcs(z4 + i);
            take(a.x); take(a.y); take(a.z); take(a.w);
            take(b.x); take(b.y); take(b.z); take(b.w);
            take(c.x); take(c.y); take(c.z); take(c.w);
        }
        done = n4 << 2;
    }
    for (int64_t i = done + tid; i < n; i += stride) {
        take(x[i]); take(y[i]); take(z[i]);
    }
    lo = warp_min(lo);
    hi = warp_max(hi);
    __shared__ float s_lo[8], s_hi[8];
    __shared__ int s_bad;
    if (threadIdx.x == 0) s_bad = 0;
    __syncthreads();
    if (bad) s_bad = 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { s_lo[warp] = lo; s_hi[warp] = hi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) { lo = fminf(lo, s_lo[w]); hi = fmaxf(hi, s_hi[w]); }
        // min is kept inverted so that both words start at 0 and use atomicMax
        atomicMax(&st->min_ord, ~f2ord(lo));
        atomicMax(&st->max_ord, f2ord(hi));
        if (s_bad) set_err(&st->err, ERRBIT_NONFINITE);
    }
}

__device__ __forceinline__ void load_bbox(const DevState* st, float& mn, float& range) {
    mn = ord2f(~st->min_ord);
    const float mx = ord2f(st->max_ord);
    range = __fsub_rn(mx, mn);  // float tree_range = max - min, src/RadixTree.cu:246
}

// Digit offsets, trivial-pass detection and ping-pong parity, by one block of
// NT threads (kSortBins / NT adjacent digits each). With first < last only
// passes [first, last) run, all of them, or none where the keys are in order
// and `last` - `first` is even (the result is in the same buffer then);
// otherwise those of the first `passes` whose digits are not all equal.
template <int NT>
__device__ __forceinline__ void sort_prep(int64_t n, int passes, DevState* st, int first, int last) {
    constexpr int kPer = kSortBins / NT;
    __shared__ uint32_t s_w[NT / 32 + 1];
    __shared__ int s_triv[kSortPasses];
    for (int p = first; p < (first < last ? last : passes); ++p) {
        uint32_t h[kPer], sum = 0, tot;
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            h[i] = __ldcg(&st->hist[p][kPer * threadIdx.x + i]);
            sum += h[i];
        }
        uint32_t ex = block_excl_scan<NT, uint32_t>(sum, s_w, &tot);
        if (threadIdx.x == 0) s_triv[p] = 0;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            st->digit_off[p][kPer * threadIdx.x + i] = ex;
            ex += h[i];
            if ((int64_t)h[i] == n) s_triv[p] = 1;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        int act = 0;
        const bool sorted = !st->disorder && (last - first) % 2 == 0;
        for (int p = 0; p < kSortPasses; ++p) {
            const bool run = first < last ? p >= first && p < last && !sorted : p < passes && !s_triv[p];
            st->pass_active[p] = run;
            st->pass_parity[p] = act & 1;
            act += run;
        }
        st->n_active = act;
    }
}
__global__ void __launch_bounds__(kSortBins) k_sort_prep(int64_t n, DevState* st, int first = 0, int last = 0) {
    sort_prep<kSortBins>(n, kSortPasses, st, first, last);
}

// ---------------------------------------------------------------------------
// encode: replaces makeCodes (src/RadixTree.cu:21-39, 244-248); also builds
// the digit histograms of the onesweep sort's passes in the same pass, and its
// last block to finish prepares the passes.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_encode(const float* __restrict__ x, const float* __restrict__ y,
                                                const float* __restrict__ z, int64_t n, int code_bits, int passes,
                                                uint64_t* __restrict__ keys, DevState* st) {
    __shared__ uint32_t s_h[kCodePasses][kSortBins];
    __shared__ bool s_last;
    for (int i = threadIdx.x; i < passes * kSortBins; i += blockDim.x) (&s_h[0][0])[i] = 0;
    __syncthreads();
    float mn, range;
    load_bbox(st, mn, range);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->min_coord = mn;
        st->max_coord = ord2f(st->max_ord);
        st->range = range;
    }
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint64_t c = point_to_code(__ldcs(x + i), __ldcs(y + i), __ldcs(z + i), mn, range, code_bits);
        keys[i] = c;
#pragma unroll
        for (int p = 0; p < kCodePasses; ++p)
            if (p < passes) atomicAdd(&s_h[p][(c >> (kSortBits * p)) & (kSortBins - 1)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < passes * kSortBins; i += blockDim.x) {
        const uint32_t v = (&s_h[0][0])[i];
        if (v) atomicAdd(&(&st->hist[0][0])[i], v);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&st->tile_counter[kSortPasses + 3], 1u) + 1 == gridDim.x;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    sort_prep<256>(n, passes, st, 0, 0);
}

// ---------------------------------------------------------------------------
// Onesweep LSD radix sort pass over 64-bit keys (Adinets & Merrill,
// "Onesweep: A Faster Least Significant Digit Radix Sort for GPUs", 2022):
// warp-level multi-split ranking with ballot peer masks, decoupled look-back
// over per-tile digit counts, scatter through shared memory. Replaces
// DeviceRadixSort::SortKeys (src/RadixTree.cu:316-337). Stable.
//
// 9-bit digits (512 bins, one per thread), so a 63-bit Morton code takes 7
// passes instead of 8. A tile publishes its digit counts as soon as it has
// ranked its keys, scatters them into shared memory, and only then reads its
// predecessors' counts. Three blocks per SM (the whole shared-memory
// carveout).
// ---------------------------------------------------------------------------
constexpr int kSortWarps = kSortThreads / 32;
static_assert(kSortThreads == kSortBins, "one digit per thread");

// Launches of at most this many tiles (they are resident together) look back
// eight tiles per step: a pass over 25 tiles (100k keys) 12.7 -> 11.3 us.
constexpr unsigned kFewTiles = 148;

struct SortSmem {
    uint32_t hist[kSortWarps][kSortBins];  // per-warp digit counts, then per-warp offsets
    uint64_t keys[kSortTile];
    uint32_t local_start[kSortBins];  // first slot of each digit in the tile
    int32_t goff[kSortBins];          // global position of the digit's run minus local_start
    uint32_t scan_w[kSortWarps + 1];
    uint32_t tile_id;
};

__global__ void __launch_bounds__(kSortThreads, 3) k_onesweep(uint64_t* buf0, uint64_t* buf1, int64_t n, int pass,
                                                           uint32_t* __restrict__ lookback, DevState* st,
                                                           int spin_limit, int stall_first_tile) {
    // a look-back of this build gave up: its key order is lost, write nothing
    if (!st->pass_active[pass] || (st->err & ERRBIT_LOOKBACK)) return;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SortSmem& S = *reinterpret_cast<SortSmem*>(smem_raw);
    const int parity = st->pass_parity[pass];
    const bool few_tiles = gridDim.x <= kFewTiles;
    const uint64_t* __restrict__ in = parity ? buf1 : buf0;
    uint64_t* __restrict__ out = parity ? buf0 : buf1;
    const int shift = kSortBits * pass;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    for (int i = tid; i < kSortWarps * kSortBins; i += kSortThreads) (&S.hist[0][0])[i] = 0;
    if (tid == 0) S.tile_id = atomicAdd(&st->tile_counter[pass], 1u);
    __syncthreads();
    const uint32_t tile = S.tile_id;
    const int64_t base = (int64_t)tile * kSortTile;

    uint64_t key[kSortIpt];
    uint32_t rank[kSortIpt];
    const int64_t wbase = base + (int64_t)warp * 32 * kSortIpt;
#pragma unroll
    for (int i = 0; i < kSortIpt; ++i) {
        const int64_t idx = wbase + i * 32 + lane;
        key[i] = idx < n ? in[idx] : 0ull;
    }
#pragma unroll
    for (int i = 0; i < kSortIpt; ++i) {
        const int64_t idx = wbase + i * 32 + lane;
        const bool valid = idx < n;
        const uint32_t d = (uint32_t)(key[i] >> shift) & (kSortBins - 1);
        // lanes holding the same digit: one ballot for validity, one per digit
        // bit (measured slightly faster than __match_any_sync)
        uint32_t peers = __ballot_sync(0xffffffffu, valid);
        if (!valid) peers = ~peers;
#pragma unroll
        for (int bb = 0; bb < kSortBits; ++bb) {
            const uint32_t v = __ballot_sync(0xffffffffu, (d >> bb) & 1u);
            peers &= ((d >> bb) & 1u) ? v : ~v;
        }
        uint32_t b = 0;
        if (valid) b = S.hist[warp][d];
        __syncwarp();
        if (valid && lane == 31 - __clz(peers)) S.hist[warp][d] = b + __popc(peers);
        __syncwarp();
        rank[i] = b + __popc(peers & lanemask_lt());
    }
    __syncthreads();

    // digit `tid`: exclusive prefix over warps and the tile's count, published
    // at once so that successors' look-backs find it early
    const int dg = tid;
    uint32_t cnt = 0;
    for (int w = 0; w < kSortWarps; ++w) {
        const uint32_t c = S.hist[w][dg];
        S.hist[w][dg] = cnt;
        cnt += c;
    }
    if (tile == 0) {
        if (!stall_first_tile) st_relaxed(lookback + dg, LB_PRE | cnt);
    } else {
        st_relaxed(lookback + (size_t)tile * kSortBins + dg, LB_AGG | cnt);
    }
    {
        uint32_t tot;
        S.local_start[dg] = block_excl_scan<kSortThreads, uint32_t>(cnt, S.scan_w, &tot);
    }
    __syncthreads();
    // keys into shared memory in digit order
#pragma unroll
    for (int i = 0; i < kSortIpt; ++i) {
        const int64_t idx = wbase + i * 32 + lane;
        if (idx < n) {
            const uint32_t d = (uint32_t)(key[i] >> shift) & (kSortBins - 1);
            S.keys[S.local_start[d] + S.hist[warp][d] + rank[i]] = key[i];
        }
    }
    // decoupled look-back on digit `dg`, after the scatter: by then most
    // predecessors have published (reading them earlier, or several at a time,
    // measured slower: the polls compete with the tiles still ranking)
    uint32_t excl = 0;
    if (tile > 0) {
        int64_t p = (int64_t)tile - 1;
        int spins = 0;
        // Few tiles run all at once, and the last would walk over most of them
        // one L2 latency at a time: they read eight predecessors per step. (With
        // more tiles than fit, eight polls at a time disturb the tiles still
        // ranking: see the comment above.)
        bool wait = few_tiles;
        while (wait && p >= 0) {
            uint32_t v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = p >= j ? ld_relaxed(lookback + (size_t)(p - j) * kSortBins + dg) : LB_PRE;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t f = v[j] >> 30;
                if (f == 0) {
                    if (++spins > spin_limit) {
                        set_err(&st->err, ERRBIT_LOOKBACK);
                        wait = false;
                    }
                    break;
                }
                excl += v[j] & LB_VAL;
                if (f == 2) {
                    wait = false;
                    break;
                }
                --p;
            }
        }
        if (few_tiles) p = -1;
        while (p >= 0) {
            const uint32_t v = ld_relaxed(lookback + (size_t)p * kSortBins + dg);
            const uint32_t f = v >> 30;
            if (f == 0) {
                if (++spins > spin_limit) {
                    set_err(&st->err, ERRBIT_LOOKBACK);
                    break;
                }
                continue;
            }
            excl += v & LB_VAL;
            if (f == 2) break;
            --p;
        }
        st_relaxed(lookback + (size_t)tile * kSortBins + dg, LB_PRE | (excl + cnt));
    }
    S.goff[dg] = (int32_t)(st->digit_off[pass][dg] + excl) - (int32_t)S.local_start[dg];
    __syncthreads();
    const int tile_n = (int)min64(kSortTile, n - base);
    for (int j = tid; j < tile_n; j += kSortThreads) {
        const uint64_t k = S.keys[j];
        const uint32_t d = (uint32_t)(k >> shift) & (kSortBins - 1);
        const int64_t pos = (int64_t)S.goff[d] + j;
        if (pos >= 0 && pos < n) out[pos] = k;
        else set_err(&st->err, ERRBIT_BOUNDS);
    }
}

// ---------------------------------------------------------------------------
// dedup + decode: replaces findDups + InclusiveSum + moveDups
// (src/RadixTree.cu:71-97, 258-303) and decodePoints (src/Octree.cu:14-24,
// 305-315) with one pass: flag, block scan, decoupled look-back, compact, and
// decode of each surviving code.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kDedupThreads) k_dedup(const uint64_t* buf0, const uint64_t* buf1, int64_t n,
                                                         int code_bits, uint64_t* __restrict__ codes_out,
                                                         float4* __restrict__ pts4, float* __restrict__ pts3,
                                                         uint32_t* __restrict__ lookback, DevState* st,
                                                         int spin_limit) {
    // a sort look-back gave up: no order to dedup; u stays 0 and later stages do nothing
    if (st->err & ERRBIT_LOOKBACK) return;
    constexpr int kWarps = kDedupThreads / 32;
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ uint32_t s_wcnt[kWarps];
    __shared__ uint32_t s_tile, s_excl;
    const uint64_t* __restrict__ keys = (st->n_active & 1) ? buf1 : buf0;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(&st->tile_counter[kSortPasses], 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    // Warp-striped: a warp's 32 * kDedupIpt keys are contiguous and element i
    // of lane l is key wbase + 32 i + l, so loads and the compacted stores of
    // each step are coalesced. Flags are kept as one ballot per step.
    const int64_t wbase = (int64_t)tile * kDedupTile + (int64_t)warp * 32 * kDedupIpt;
    uint64_t k[kDedupIpt];
    uint32_t m[kDedupIpt];
    uint64_t last = (wbase > 0 && wbase - 1 < n) ? keys[wbase - 1] : 0ull;  // the key before this step's
    uint32_t wcnt = 0;
#pragma unroll
    for (int i = 0; i < kDedupIpt; ++i) {
        const int64_t j = wbase + 32 * i + lane;
        k[i] = j < n ? keys[j] : 0ull;
        uint64_t prev = __shfl_up_sync(kFull, k[i], 1);
        if (lane == 0) prev = last;
        last = __shfl_sync(kFull, k[i], 31);
        m[i] = __ballot_sync(kFull, j < n && (j == 0 || k[i] != prev));
        wcnt += __popc(m[i]);
    }
    if (lane == 0) s_wcnt[warp] = wcnt;
    __syncthreads();
    uint32_t woff = 0, tot = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const uint32_t c = s_wcnt[w];
        woff += w < warp ? c : 0u;
        tot += c;
    }
    // Decoupled look-back by warp 0, 32 predecessors per step: lane i reads
    // tile p - i. The walk ends at the nearest tile with an inclusive prefix
    // (tile 0 always publishes one); it needs every tile up to that one ready.
    if (warp == 0) {
        uint32_t excl = 0;
        if (tile == 0) {
            if (lane == 0) st_relaxed(lookback, LB_PRE | tot);
        } else {
            if (lane == 0) st_relaxed(lookback + tile, LB_AGG | tot);
            int64_t p = (int64_t)tile - 1;
            int spins = 0;
            for (;;) {
                const int64_t q = p - lane;
                const uint32_t v = q >= 0 ? ld_relaxed(lookback + q) : LB_PRE;
                const uint32_t f = v >> 30;
                const uint32_t pre = __ballot_sync(kFull, f == 2);
                const uint32_t need = pre ? (((pre & (0u - pre)) << 1) - 1u) : kFull;  // lanes up to the first prefix
                if (__ballot_sync(kFull, f == 0) & need) {
                    if (++spins > spin_limit) {
                        if (lane == 0) set_err(&st->err, ERRBIT_LOOKBACK);
                        break;
                    }
                    continue;
                }
                excl += __reduce_add_sync(kFull, ((need >> lane) & 1u) ? (v & LB_VAL) : 0u);
                if (pre) break;
                p -= 32;
            }
            if (lane == 0) st_relaxed(lookback + tile, LB_PRE | (excl + tot));
        }
        if (lane == 0) {
            s_excl = excl;
            if ((int64_t)(tile + 1) * kDedupTile >= n) st->u = (unsigned long long)(excl + tot);
        }
    }
    __syncthreads();
    const float mn = st->min_coord, range = st->range;
    uint32_t base = s_excl + woff;
#pragma unroll
    for (int i = 0; i < kDedupIpt; ++i) {
        if ((m[i] >> lane) & 1u) {
            const uint32_t pos = base + __popc(m[i] & lanemask_lt());
            if ((int64_t)pos >= n) {
                set_err(&st->err, ERRBIT_BOUNDS);
            } else {
                codes_out[pos] = k[i];
                const float3 p = code_to_point(k[i], mn, range, code_bits);
                pts4[pos] = make_float4(p.x, p.y, p.z, 0.0f);
                pts3[3 * (size_t)pos + 0] = p.x;
                pts3[3 * (size_t)pos + 1] = p.y;
                pts3[3 * (size_t)pos + 2] = p.z;
            }
        }
        base += __popc(m[i]);
    }
}

// ---------------------------------------------------------------------------
// Front of the build for small clouds: bbox, encode, sort, dedup and decode (as
// the kernels above) in one block, keys in shared memory. A small build is a
// chain of launches whose kernels have little to do; this one replaces eleven
// of them and three memsets (it clears the state and scratch itself). Up to 8192
// points, what 1024 threads hold at 8 keys each: these stages took 126 us on
// 2011 points and take 33 us (whole build 199 and 84 us); at 8192 points the
// whole build takes 136 us, with the separate kernels 180 us.
// IPT keys per thread; element order is warp by warp, so ranking by warps is
// stable. Slots past n hold all ones and stay last.
// ---------------------------------------------------------------------------
constexpr int kFrontThreads = 1024;
constexpr int kFrontWarps = kFrontThreads / 32;
static_assert(kFrontMax == 8 * kFrontThreads, "8 keys per thread");

template <int IPT>
struct FrontSmem {
    uint64_t keys[IPT * kFrontThreads];
    uint32_t hist[kFrontWarps][kSortBins];
    uint32_t start[kSortBins];
    uint32_t scan_w[kFrontWarps + 1];
    float lo[kFrontWarps], hi[kFrontWarps];
    uint32_t diff_lo[kFrontWarps], diff_hi[kFrontWarps];
    uint32_t cnt[kFrontWarps];
    int bad;
};

template <int IPT>
__global__ void __launch_bounds__(kFrontThreads) k_front(const float* __restrict__ x, const float* __restrict__ y,
                                                         const float* __restrict__ z, int n, int code_bits,
                                                         uint64_t* __restrict__ codes_out, float4* __restrict__ pts4,
                                                         float* __restrict__ pts3, uint32_t* __restrict__ scratch,
                                                         int scratch_words, DevState* st) {
    constexpr unsigned kFull = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    FrontSmem<IPT>& S = *reinterpret_cast<FrontSmem<IPT>*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < scratch_words; i += kFrontThreads) scratch[i] = 0;
    // the state up to the sort's histograms, which nothing reads here
    for (int i = tid; i < (int)(offsetof(DevState, hist) / 4); i += kFrontThreads) reinterpret_cast<uint32_t*>(st)[i] = 0;
    if (tid == 0) S.bad = 0;
    const int base = warp * 32 * IPT + lane;
    float px[IPT], py[IPT], pz[IPT];
    float lo = FLT_MAX, hi = -FLT_MAX;
    bool bad = false;
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
        const int e = base + 32 * i;
        if (e < n) {
            px[i] = x[e];
            py[i] = y[e];
            pz[i] = z[e];
            lo = fminf(lo, fminf(px[i], fminf(py[i], pz[i])));
            hi = fmaxf(hi, fmaxf(px[i], fmaxf(py[i], pz[i])));
            bad |= !(isfinite(px[i]) && isfinite(py[i]) && isfinite(pz[i]));
        }
    }
    lo = warp_min(lo);
    hi = warp_max(hi);
    if (lane == 0) {
        S.lo[warp] = lo;
        S.hi[warp] = hi;
    }
    __syncthreads();  // S.bad is clear, the state is clear
    if (bad) S.bad = 1;
    lo = warp_min(S.lo[lane]);
    hi = warp_max(S.hi[lane]);
    const float mn = lo, range = __fsub_rn(hi, lo);
    uint64_t key[IPT];
    uint64_t diff = 0;
    const uint64_t key0 = point_to_code(x[0], y[0], z[0], mn, range, code_bits);
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
        key[i] = ~0ull;
        if (base + 32 * i < n) {
            key[i] = point_to_code(px[i], py[i], pz[i], mn, range, code_bits);
            diff |= key[i] ^ key0;
        }
        S.keys[base + 32 * i] = key[i];
    }
    // digits in which no two keys differ need no pass
    const uint32_t dl = __reduce_or_sync(kFull, (uint32_t)diff), dh = __reduce_or_sync(kFull, (uint32_t)(diff >> 32));
    if (lane == 0) {
        S.diff_lo[warp] = dl;
        S.diff_hi[warp] = dh;
    }
    __syncthreads();
    diff = ((uint64_t)__reduce_or_sync(kFull, S.diff_hi[lane]) << 32) | __reduce_or_sync(kFull, S.diff_lo[lane]);
    for (int shift = 0; shift < code_bits; shift += kSortBits) {
        if (!((diff >> shift) & (kSortBins - 1))) continue;
        for (int i = tid; i < kFrontWarps * kSortBins; i += kFrontThreads) (&S.hist[0][0])[i] = 0;
        __syncthreads();
        uint32_t rank[IPT];
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const uint32_t d = (uint32_t)(key[i] >> shift) & (kSortBins - 1);
            uint32_t peers = kFull;
#pragma unroll
            for (int bb = 0; bb < kSortBits; ++bb) {
                const uint32_t v = __ballot_sync(kFull, (d >> bb) & 1u);
                peers &= ((d >> bb) & 1u) ? v : ~v;
            }
            const uint32_t b = S.hist[warp][d];
            __syncwarp();
            if (lane == 31 - __clz(peers)) S.hist[warp][d] = b + __popc(peers);
            __syncwarp();
            rank[i] = b + __popc(peers & lanemask_lt());
        }
        __syncthreads();
        uint32_t cnt = 0;
        if (tid < kSortBins)
            for (int w = 0; w < kFrontWarps; ++w) {
                const uint32_t c = S.hist[w][tid];
                S.hist[w][tid] = cnt;
                cnt += c;
            }
        uint32_t tot;
        const uint32_t at = block_excl_scan<kFrontThreads, uint32_t>(cnt, S.scan_w, &tot);
        if (tid < kSortBins) S.start[tid] = at;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < IPT; ++i) {
            const uint32_t d = (uint32_t)(key[i] >> shift) & (kSortBins - 1);
            S.keys[S.start[d] + S.hist[warp][d] + rank[i]] = key[i];
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < IPT; ++i) key[i] = S.keys[base + 32 * i];
        __syncthreads();
    }
    // dedup and decode
    uint32_t m[IPT], wcnt = 0;
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
        const int e = base + 32 * i;
        m[i] = __ballot_sync(kFull, e < n && (e == 0 || S.keys[e - 1] != key[i]));
        wcnt += __popc(m[i]);
    }
    if (lane == 0) S.cnt[warp] = wcnt;
    __syncthreads();
    const uint32_t c = S.cnt[lane];
    const uint32_t inc = warp_incl_scan(c);
    uint32_t pos = __shfl_sync(kFull, inc - c, warp);
    if (tid == 0) {
        st->min_coord = mn;
        st->max_coord = hi;
        st->range = range;
        if (S.bad) st->err = ERRBIT_NONFINITE;
    }
    if (tid == 31) st->u = inc;
#pragma unroll
    for (int i = 0; i < IPT; ++i) {
        if ((m[i] >> lane) & 1u) {
            const uint32_t o = pos + __popc(m[i] & lanemask_lt());
            const float3 p = code_to_point(key[i], mn, range, code_bits);
            codes_out[o] = key[i];
            pts4[o] = make_float4(p.x, p.y, p.z, 0.0f);
            pts3[3 * o + 0] = p.x;
            pts3[3 * o + 1] = p.y;
            pts3[3 * o + 2] = p.z;
        }
        pos += __popc(m[i]);
    }
}

// ---------------------------------------------------------------------------
// Karras radix tree: replaces constructTree (src/RadixTree.cu:99-194,
// launched at :351-364). One thread per internal node, same search steps and
// integer semantics as the reference, so topology is bit-exact. Node 0 is
// computed twice: with the reference's root range l = N-1 (:128-130) for the
// exported arrays when root_compat is set, and with the full range for the
// features of the learned radius. Also records each leaf's parent and each
// node's range end for them.
// ---------------------------------------------------------------------------
struct KNode {
    int64_t j;
    int64_t gamma;
    int dnode;
    bool hl, hr;
};

__device__ __forceinline__ KNode karras_node(const uint64_t* __restrict__ codes, int64_t i, int64_t N, int cb,
                                             bool compat_root) {
    const uint64_t ci = codes[i];
    int d;
    if (i == 0) {
        d = 1;
    } else {
        const int dd = delta_codes(ci, codes[i + 1], cb) - delta_codes(ci, codes[i - 1], cb);
        d = (dd > 0) - (dd < 0);
    }
    int64_t l = 0;
    if (i == 0) {
        l = compat_root ? N - 1 : N;
    } else {
        const int dmin = delta_codes(ci, codes[i - d], cb);
        int64_t lmax = 2;
        while (i + lmax * d >= 0 && i + lmax * d <= N && delta_codes(ci, codes[i + lmax * d], cb) > dmin) lmax *= 2;
        const int64_t lcut = (d == -1) ? i : N - i;
        // t = lmax / 2, lmax / 4, ... (powers-of-two divisions as shifts: 64-bit
        // divisions made the radix stage 22% slower on 13M codes)
        for (int sh = 1; (lmax >> sh) >= 1; ++sh) {
            const int64_t t = lmax >> sh;
            if (l + t <= lcut && delta_codes(ci, codes[i + (l + t) * d], cb) > dmin) l += t;
        }
    }
    KNode r;
    r.j = i + l * d;
    r.dnode = delta_codes(codes[i], codes[r.j], cb);
    int64_t s = 0;
    if (l >= 1) {
        const int nlow = 63 - __clzll((long long)l);
        const int lc = nlow + ((uint64_t)l > (uint64_t)one_shl(nlow));  // ceil(log2 l)
        const int64_t scut = (d == -1) ? i - 1 : N - i - 1;
        // t = ceil(l / 2), ceil(l / 4), ... up to 2^lc (shifts, not divisions)
        for (int sh = 1; sh <= lc; ++sh) {
            const int64_t t = (l + ((int64_t)1 << sh) - 1) >> sh;
            if (s + t <= scut && delta_codes(ci, codes[i + (s + t) * d], cb) > r.dnode) s += t;
        }
    }
    r.gamma = i + s * d + min(d, 0);
    r.hl = min(i, r.j) == r.gamma;
    r.hr = max(i, r.j) == r.gamma + 1;
    return r;
}

__global__ void __launch_bounds__(256) k_karras(const uint64_t* __restrict__ codes, int code_bits, int root_compat,
                                                int32_t* __restrict__ left_child, int32_t* __restrict__ parent,
                                                uint8_t* __restrict__ prefix_n, uint8_t* __restrict__ hll,
                                                uint8_t* __restrict__ hlr, int32_t* __restrict__ sparent,
                                                int32_t* __restrict__ leaf_parent, int32_t* __restrict__ range_end,
                                                DevState* st) {
    const int64_t u = (int64_t)st->u;
    const int64_t N = u - 1;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    // entries of `parent` that no node claims are 0: those of the root, of the
    // last leaf's number, and, with the compat root, of the full root's children
    if (i == N) parent[i] = 0;
    if (i >= N) return;
    const KNode f = karras_node(codes, i, N, code_bits, false);
    // full root range
    range_end[i] = (int32_t)f.j;
    if (f.hl) leaf_parent[f.gamma] = (int32_t)i; else sparent[f.gamma] = (int32_t)i;
    if (f.hr) leaf_parent[f.gamma + 1] = (int32_t)i; else sparent[f.gamma + 1] = (int32_t)i;
    KNode e = f;
    if (i == 0 && root_compat) e = karras_node(codes, 0, N, code_bits, true);
    left_child[i] = (int32_t)e.gamma;
    prefix_n[i] = (uint8_t)e.dnode;
    hll[i] = e.hl;
    hlr[i] = e.hr;
    // The compat root's parent claims are written after this kernel (by k_leaves)
    // so that, in a tree the compat root breaks, they win deterministically.
    if (!f.hl) parent[f.gamma] = (int32_t)i;
    if (!f.hr) parent[f.gamma + 1] = (int32_t)i;
    if (i == 0) parent[0] = 0;
}

__device__ __forceinline__ void root_parent(const int32_t* __restrict__ left_child, int32_t* __restrict__ parent,
                                            const uint8_t* __restrict__ hll, const uint8_t* __restrict__ hlr,
                                            int64_t u, DevState* st) {
    if (u < 2) return;
    const int32_t g = left_child[0];
    if (g < 0 || g + 1 >= u) {
        set_err(&st->err, ERRBIT_BOUNDS);
        return;
    }
    if (!hll[0]) parent[g] = 0;
    if (!hlr[0]) parent[g + 1] = 0;
}

// ---------------------------------------------------------------------------
// Search hierarchy. Its leaves are the maximal Morton subtrees of at most M
// points, in Morton order; 32 consecutive nodes form a node of the next
// level, up to a top level of at most 32 nodes.
//
// k_leaves finds the leaves from the sorted codes alone. Point i starts a leaf
// when the subtree that joins it to point i - 1 holds more than M points: when
// some run of M + 1 points [a, a + M] across the gap shares at least the
// prefix that codes i - 1 and i share. So with w(a) = the common prefix of
// codes a and a + M, point i starts a leaf when the largest w(a) over a in
// [i - M, i - 1] is at least the common prefix of codes i - 1 and i: a sliding
// maximum, one ballot per 32 codes, and a decoupled look-back over the tiles'
// leaf counts. For M = 32 the maximum takes shuffles alone; smaller M (a small
// leaf_bucket) takes doubling windows in shared memory. On 13M codes (20M
// precision mix) this and k_boxes take 0.220 ms (0.288 ms with the shared-memory
// windows and 1024-code tiles; 4096-code tiles 0.200 ms, but 2 us more on a 2k
// cloud), where merging the boxes of a binary tree bottom-up took 0.530 ms; it
// reads no radix tree, so batched
// builds make none. M is at most 32, one point per lane of the scan: of the
// layouts simulated on 400k-point clouds (fixed runs of 16, 32 and 64 points,
// runs cut at the best prefix, subtrees of at most 32 and 96) subtrees of at
// most 32 let a warp scan the fewest points, 420 on a scene (96: 770; fixed
// runs of 32: 920).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kLeafThreads) k_leaves(const uint64_t* __restrict__ codes, int M,
                                                         int32_t* __restrict__ leaf_start,
                                                         uint32_t* __restrict__ lookback, int root_compat,
                                                         const int32_t* __restrict__ left_child,
                                                         int32_t* __restrict__ parent,
                                                         const uint8_t* __restrict__ hll,
                                                         const uint8_t* __restrict__ hlr, DevState* st,
                                                         int spin_limit) {
    constexpr int kHalo = kLeafMax, kSpan = kLeafTile + 2 * kHalo;
    constexpr int kCells = kLeafIpt * kLeafThreads / 32;  // 32-code steps of a tile
    constexpr int kPerLane = kCells / 32;  // counts of steps per lane of the scanning warp
    static_assert(kCells % 32 == 0, "one warp scans the steps' counts");
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ uint64_t s_code[kSpan];   // codes [t0 - kHalo, t0 + kLeafTile + kHalo)
    __shared__ int8_t s_w[2][kSpan];     // window maxima of w, ping-pong
    __shared__ uint32_t s_cnt[kCells];
    __shared__ uint32_t s_tile;
    const int64_t u = (int64_t)st->u;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_tile = atomicAdd(&st->tile_counter[kSortPasses + 2], 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t t0 = (int64_t)tile * kLeafTile;
    if (root_compat && tile == 0 && tid == 0) root_parent(left_child, parent, hll, hlr, u, st);
    if (t0 >= u) return;
    // warp by warp, 32 codes a step: step r of the warp starts at this code
    const int64_t at = t0 + (int64_t)warp * 32 * kLeafIpt;
    uint32_t flags[kLeafIpt];
    if (M == kHalo) {
        // w of a step's codes needs the next step's code on the same lane only,
        // and the window [i - 32, i - 1] is the end of the step before and the
        // start of this one: a suffix and a prefix maximum by shuffles
        uint64_t c = at + lane >= 32 && at + lane - 32 < u ? codes[at + lane - 32] : 0ull;
        uint64_t next = at + lane < u ? codes[at + lane] : 0ull;
        int before = -1;     // the suffix maximum of the step before
        uint64_t last = 0;   // its last code
#pragma unroll
        for (int r = -1; r < kLeafIpt; ++r) {
            const int64_t i = at + 32 * r + lane;
            int w = i >= 0 && i + 32 < u ? __clzll((long long)(c ^ next)) : -1;
            int pre = __shfl_up_sync(kFull, w, 1);
            if (lane == 0) pre = -1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(kFull, pre, o);
                pre = lane >= o ? max(pre, v) : pre;
                const int x = __shfl_down_sync(kFull, w, o);
                w = lane + o < 32 ? max(w, x) : w;
            }
            uint64_t prev = __shfl_up_sync(kFull, c, 1);
            if (lane == 0) prev = last;
            last = __shfl_sync(kFull, c, 31);
            if (r >= 0) {
                const int d = __clzll((long long)(prev ^ c));
                const bool f = i < u && (i == 0 || max(before, pre) >= d);
                flags[r] = __ballot_sync(kFull, f);
                if (lane == 0) s_cnt[warp * kLeafIpt + r] = __popc(flags[r]);
            }
            before = w;
            c = next;
            const int64_t n2 = i + 64;
            next = r + 1 < kLeafIpt && n2 < u ? codes[n2] : 0ull;
        }
    } else {
        for (int j = tid; j < kSpan; j += kLeafThreads) {
            const int64_t i = t0 - kHalo + j;
            s_code[j] = i >= 0 && i < u ? codes[i] : 0ull;
        }
        __syncthreads();
        for (int j = tid; j < kSpan; j += kLeafThreads) {
            const int64_t a = t0 - kHalo + j;
            s_w[0][j] =
                a >= 0 && j + M < kSpan && a + M < u ? (int8_t)__clzll((long long)(s_code[j] ^ s_code[j + M])) : -1;
        }
        __syncthreads();
        int p = 1, cur = 0;  // s_w[cur][j] = the largest w over [j, j + p)
        for (; 2 * p <= M; p *= 2, cur ^= 1) {
            for (int j = tid; j < kSpan; j += kLeafThreads)
                s_w[cur ^ 1][j] = j + p < kSpan ? max(s_w[cur][j], s_w[cur][j + p]) : s_w[cur][j];
            __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < kLeafIpt; ++r) {
            const int64_t i = at + 32 * r + lane;
            const int j = kHalo + (int)(i - t0);
            bool f = i < u;
            if (f && i > 0) {
                const int d = __clzll((long long)(s_code[j - 1] ^ s_code[j]));
                f = max(s_w[cur][j - M], s_w[cur][j - p]) >= d;
            }
            flags[r] = __ballot_sync(kFull, f);
            if (lane == 0) s_cnt[warp * kLeafIpt + r] = __popc(flags[r]);
        }
    }
    __syncthreads();
    if (warp == 0) {
        uint32_t c = 0;
#pragma unroll
        for (int e = 0; e < kPerLane; ++e) c += s_cnt[kPerLane * lane + e];
        const uint32_t inc = warp_incl_scan(c);
        const uint32_t tot = __shfl_sync(kFull, inc, 31);
        // look-back, 32 predecessors per step (as k_dedup)
        uint32_t excl = 0;
        if (tile == 0) {
            if (lane == 0) st_relaxed(lookback, LB_PRE | tot);
        } else {
            if (lane == 0) st_relaxed(lookback + tile, LB_AGG | tot);
            int64_t q0 = (int64_t)tile - 1;
            int spins = 0;
            for (;;) {
                const int64_t q = q0 - lane;
                const uint32_t v = q >= 0 ? ld_relaxed(lookback + q) : LB_PRE;
                const uint32_t fl = v >> 30;
                const uint32_t pre = __ballot_sync(kFull, fl == 2);
                const uint32_t need = pre ? (((pre & (0u - pre)) << 1) - 1u) : kFull;
                if (__ballot_sync(kFull, fl == 0) & need) {
                    if (++spins > spin_limit) {
                        if (lane == 0) set_err(&st->err, ERRBIT_LOOKBACK);
                        break;
                    }
                    continue;
                }
                excl += __reduce_add_sync(kFull, ((need >> lane) & 1u) ? (v & LB_VAL) : 0u);
                if (pre) break;
                q0 -= 32;
            }
            if (lane == 0) st_relaxed(lookback + tile, LB_PRE | (excl + tot));
        }
        uint32_t first = excl + inc - c;
#pragma unroll
        for (int e = 0; e < kPerLane; ++e) {
            const uint32_t mine = s_cnt[kPerLane * lane + e];
            s_cnt[kPerLane * lane + e] = first;
            first += mine;
        }
        if (lane == 0 && t0 + kLeafTile >= u) {
            uint32_t n = excl + tot, off = 0;
            int l = 0;
            for (;; ++l) {
                st->level_off[l] = off;
                st->level_count[l] = n;
                if (n <= kFan || l == kMaxLevels - 1) break;
                off += n;
                n = (n + kFan - 1) / kFan;
            }
            st->top_level = l;
        }
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kLeafIpt; ++r) {
        if (!((flags[r] >> lane) & 1u)) continue;
        const uint32_t pos = s_cnt[warp * kLeafIpt + r] + __popc(flags[r] & lanemask_lt());
        const int64_t i = at + 32 * r + lane;
        if ((int64_t)pos < u) leaf_start[pos] = (int32_t)i;
        else set_err(&st->err, ERRBIT_BOUNDS);
    }
}

__device__ __forceinline__ float warp_min_f(float v) {
    float r;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float warp_max_f(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// Boxes of the hierarchy, bottom up: a warp takes 32 consecutive leaves (one
// per lane, whose points follow one another, so the lanes' 16-byte loads share
// cache lines) and reduces their boxes to the level-1 node's; the warp whose
// node completes a group of 32 siblings (an arrival counter per parent) goes
// on with the parent.
__global__ void __launch_bounds__(128) k_boxes(const float4* __restrict__ pts, const int32_t* __restrict__ leaf_start,
                                               uint32_t* __restrict__ arrivals, SNode* __restrict__ snodes,
                                               DevState* st) {
    constexpr unsigned kFull = 0xffffffffu;
    const int64_t u = (int64_t)st->u;
    const uint32_t nl = u > 0 && !(st->err & ERRBIT_LOOKBACK) ? st->level_count[0] : 0u;
    const int lane = threadIdx.x & 31;
    const int top = st->top_level;
    const uint32_t groups = (nl + 31) / 32;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    for (uint32_t g = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); g < groups; g += warps) {
        const uint32_t leaf = g * 32 + lane;
        float4 lo = make_float4(INFINITY, INFINITY, INFINITY, 0.f), hi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
        if (leaf < nl) {
            const int32_t f = leaf_start[leaf], e = leaf + 1 < nl ? leaf_start[leaf + 1] : (int32_t)u;
            const int32_t cnt = e - f;
            if (f < 0 || cnt < 1 || cnt > kLeafMax || e > u) {
                set_err(&st->err, ERRBIT_BOUNDS);
            } else {
#pragma unroll 4
                for (int32_t q = f; q < e; ++q) {
                    const float4 v = __ldg(pts + q);
                    lo.x = fminf(lo.x, v.x); lo.y = fminf(lo.y, v.y); lo.z = fminf(lo.z, v.z);
                    hi.x = fmaxf(hi.x, v.x); hi.y = fmaxf(hi.y, v.y); hi.z = fmaxf(hi.z, v.z);
                }
                lo.w = __int_as_float(f);
                hi.w = __int_as_float(cnt);
                snodes[leaf].lo = lo;
                snodes[leaf].hi = hi;
            }
        }
        uint32_t node = g;
        for (int l = 1; l <= top; ++l) {
            lo = make_float4(warp_min_f(lo.x), warp_min_f(lo.y), warp_min_f(lo.z), 0.f);
            hi = make_float4(warp_max_f(hi.x), warp_max_f(hi.y), warp_max_f(hi.z), 0.f);
            SNode* mine = snodes + st->level_off[l] + node;
            if (lane == 0) {
                mine->lo = lo;
                mine->hi = hi;
            }
            if (l == top) break;
            // the parent's other children may be other warps': the last to arrive reduces them all
            const uint32_t parent = node / kFan, first = parent * kFan;
            const uint32_t kids = min((uint32_t)kFan, st->level_count[l] - first);
            uint32_t seen = 0;
            __threadfence();
            if (lane == 0) seen = atomicAdd(arrivals + (st->level_off[l + 1] - st->level_off[2]) + parent, 1u);
            seen = __shfl_sync(kFull, seen, 0);
            if (seen + 1 != kids) break;
            __threadfence();
            lo = make_float4(INFINITY, INFINITY, INFINITY, 0.f);
            hi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.f);
            if (lane < kids) {
                lo = __ldcg(&snodes[st->level_off[l] + first + lane].lo);
                hi = __ldcg(&snodes[st->level_off[l] + first + lane].hi);
            }
            node = parent;
        }
    }
}

// ---------------------------------------------------------------------------
// Octree: replaces calcEdgeCounts + InclusiveSum (src/Octree.cu:38-50,
// 215-247) with one counting + decoupled look-back scan kernel writing the
// exclusive offsets and the node total, and zeroing the nodes.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kScanThreads) k_oct_scan(const uint8_t* __restrict__ prefix_n,
                                                           const int32_t* __restrict__ parent,
                                                           int32_t* __restrict__ counts,
                                                           int32_t* __restrict__ offsets,
                                                           unsigned long long* __restrict__ lookback,
                                                           OtNode* __restrict__ nodes, int64_t cap,
                                                           DevState* st, int spin_limit) {
    __shared__ long long s_w[kScanThreads / 32 + 1];
    __shared__ uint32_t s_tile;
    __shared__ long long s_excl;
    const int64_t N = (int64_t)st->u - 1;
    const int tid = threadIdx.x;
    if (tid == 0) s_tile = atomicAdd(&st->tile_counter[kSortPasses + 1], 1u);
    __syncthreads();
    const uint32_t tile = s_tile;
    const int64_t first = (int64_t)tile * kScanTile + (int64_t)tid * kScanIpt;
    int32_t c[kScanIpt];
    long long sum = 0;
    const int root_level = N > 0 ? prefix_n[0] / 3 : 0;
#pragma unroll
    for (int i = 0; i < kScanIpt; ++i) {
        const int64_t j = first + i;
        int32_t v = 0;
        if (j == 0) {
            v = 1;  // the root (src/Octree.cu:217-218)
        } else if (j < N) {
            const int32_t pp = parent[j];
            v = prefix_n[j] / 3 - ((pp >= 0 && pp < N) ? prefix_n[pp] / 3 : root_level);
        }
        c[i] = v;
        if (j < N) counts[j] = v;
        sum += v;
    }
    // Counts can be negative only in a tree broken by the compat root; values
    // travel through the look-back as 62-bit two's complement.
    auto sx62 = [](unsigned long long v) { return (long long)(v << 2) >> 2; };
    long long tot;
    const long long toff = block_excl_scan<kScanThreads, long long>(sum, s_w, &tot);
    if (tid < 32) {
        // look-back, 32 predecessors per step (as k_dedup)
        constexpr unsigned kFull = 0xffffffffu;
        unsigned long long* mine = lookback + tile;
        long long excl = 0;
        if (tile == 0) {
            if (tid == 0) st_relaxed64(mine, LB64_PRE | ((unsigned long long)tot & LB64_VAL));
        } else {
            if (tid == 0) st_relaxed64(mine, LB64_AGG | ((unsigned long long)tot & LB64_VAL));
            int64_t p = (int64_t)tile - 1;
            int spins = 0;
            for (;;) {
                const int64_t q = p - tid;
                const unsigned long long v = q >= 0 ? ld_relaxed64(lookback + q) : LB64_PRE;
                const uint32_t f = (uint32_t)(v >> 62);
                const uint32_t pre = __ballot_sync(kFull, f == 2);
                const uint32_t need = pre ? (((pre & (0u - pre)) << 1) - 1u) : kFull;  // lanes up to the first prefix
                if (__ballot_sync(kFull, f == 0) & need) {
                    if (++spins > spin_limit) {
                        if (tid == 0) set_err(&st->err, ERRBIT_LOOKBACK);
                        break;
                    }
                    continue;
                }
                long long part = ((need >> tid) & 1u) ? sx62(v & LB64_VAL) : 0ll;
#pragma unroll
                for (int o = 16; o >= 1; o >>= 1) part += __shfl_xor_sync(kFull, part, o);
                excl += part;
                if (pre) break;
                p -= 32;
            }
            if (tid == 0) st_relaxed64(mine, LB64_PRE | ((unsigned long long)(excl + tot) & LB64_VAL));
        }
        if (tid == 0) {
            s_excl = excl;
            if ((int64_t)(tile + 1) * kScanTile >= N) {
                const long long total = excl + tot;
                st->n_oct = (N > 0 && total > 0) ? (unsigned long long)total : 0ull;
                st->root_level = root_level;
            }
        }
    }
    __syncthreads();
    long long run = s_excl + toff;
#pragma unroll
    for (int i = 0; i < kScanIpt; ++i) {
        const int64_t j = first + i;
        if (j <= N) offsets[j] = (int32_t)run;
        run += c[i];
    }
    // zero the tile's own nodes (src/Octree.cu:250-253); the root's corner and
    // size are written by k_oct_make (src/Octree.cu:257-261)
    const long long z0 = s_excl < 0 ? 0 : s_excl, z1 = s_excl + tot < cap ? s_excl + tot : (long long)cap;
    if (tid == 0 && s_excl + tot > cap) set_err(&st->err, ERRBIT_OCT_CAPACITY);
    uint2* words = reinterpret_cast<uint2*>(nodes);  // 56 B = 7 x 8 B per node
    for (long long w = 7 * z0 + tid; w < 7 * z1; w += kScanThreads) words[w] = make_uint2(0u, 0u);
}

__device__ __forceinline__ int64_t oct_walk_up(int64_t r, const int32_t* __restrict__ counts,
                                               const int32_t* __restrict__ parent, int64_t N, DevState* st) {
    for (int it = 0; it < 130; ++it) {
        if (r < 0 || r >= N) { set_err(&st->err, ERRBIT_BOUNDS); return -1; }
        if (counts[r] != 0) return r;
        r = parent[r];
    }
    set_err(&st->err, ERRBIT_BOUNDS);
    return -1;
}

// makeNodes, src/Octree.cu:114-161: each radix node emits its chain of
// counts[i] octree nodes (deepest first) and links the chain's top under the
// bottom node of its nearest contributing ancestor.
__device__ __forceinline__ void make_chain(int64_t i, int64_t m, int64_t N, OtNode* __restrict__ nodes,
                                           const int32_t* __restrict__ offsets, const int32_t* __restrict__ counts,
                                           const uint64_t* __restrict__ codes, const uint8_t* __restrict__ prefix_n,
                                           const int32_t* __restrict__ parent, int code_bits, DevState* st) {
    const float mn = st->min_coord, range = st->range;
    const int CL = code_bits;
    const int root_level = st->root_level;
    auto cell = [&](int level) { return __fdiv_rn(range, (float)one_shl(level - root_level)); };
    auto put_corner = [&](int64_t o, uint64_t pre, int level) {
        const float3 c = code_to_point(shl_clamp(pre, CL - 3 * level), mn, range, CL);
        nodes[o].corner[0] = c.x;
        nodes[o].corner[1] = c.y;
        nodes[o].corner[2] = c.z;
        nodes[o].cell_size = cell(level);
    };
    if (i == 0) {
        const uint64_t rp = shr_clamp(codes[0], CL - 3 * root_level);
        const float3 c = code_to_point(shl_clamp(rp, CL - 3 * root_level), mn, range, CL);
        nodes[0].corner[0] = c.x;
        nodes[0].corner[1] = c.y;
        nodes[0].corner[2] = c.z;
        nodes[0].cell_size = range;
        return;
    }
    int64_t oct = offsets[i];
    const int nn = counts[i];
    const int lvl_i = prefix_n[i] / 3;
    const uint64_t ci = codes[i];
    for (int j = 0; j < nn - 1; ++j) {
        const int level = lvl_i - j;
        const uint64_t pre = shr_clamp(ci, CL - 3 * level);
        const int64_t par = oct + 1;
        if (par >= 0 && par < m && oct >= 0 && oct < m) {
            nodes[par].children[pre & 7] = (int32_t)oct;
            atomicOr(&nodes[par].child_node_mask, 1 << (pre & 7));
            put_corner(oct, pre, level);
        } else {
            set_err(&st->err, ERRBIT_BOUNDS);
        }
        oct = par;
    }
    if (nn > 0) {
        const int64_t rp = oct_walk_up(parent[i], counts, parent, N, st);
        if (rp < 0) return;
        const int64_t op = offsets[rp];
        const int top = lvl_i - nn + 1;
        const uint64_t pre = shr_clamp(ci, CL - 3 * top);
        if (op >= 0 && op < m && oct >= 0 && oct < m) {
            nodes[op].children[pre & 7] = (int32_t)oct;
            atomicOr(&nodes[op].child_node_mask, 1 << (pre & 7));
            put_corner(oct, pre, top);
        } else {
            set_err(&st->err, ERRBIT_BOUNDS);
        }
    }
}

// linkLeafNodes, src/Octree.cu:65-112: each leaf child of a radix node goes
// into the bottom octree node of the nearest contributing ancestor.
__device__ __forceinline__ void link_leaves(int64_t i, int64_t m, int64_t u, OtNode* __restrict__ nodes,
                                            const int32_t* __restrict__ offsets, const int32_t* __restrict__ counts,
                                            const uint64_t* __restrict__ codes, const uint8_t* __restrict__ hll,
                                            const uint8_t* __restrict__ hlr, const uint8_t* __restrict__ prefix_n,
                                            const int32_t* __restrict__ parent,
                                            const int32_t* __restrict__ left_child, int code_bits, DevState* st) {
    const bool sides[2] = {hll[i] != 0, hlr[i] != 0};
    if (!sides[0] && !sides[1]) return;
    const int lvl = prefix_n[i] / 3 + 1;
    const int64_t rn = oct_walk_up(i, counts, parent, u - 1, st);
    if (rn < 0) return;
    const int64_t node = offsets[rn];
#pragma unroll
    for (int side = 0; side < 2; ++side) {
        if (!sides[side]) continue;
        const int64_t leaf = (int64_t)left_child[i] + side;
        if (leaf < 0 || leaf >= u || node < 0 || node >= m) { set_err(&st->err, ERRBIT_BOUNDS); continue; }
        const uint64_t pre = shr_clamp(codes[leaf], code_bits - 3 * lvl);
        nodes[node].children[pre & 7] = (int32_t)leaf;
        atomicOr(&nodes[node].child_leaf_mask, 1 << (pre & 7));
    }
}

// Both for radix node i: they write different children and masks.
__global__ void __launch_bounds__(256) k_oct_make(OtNode* __restrict__ nodes, int64_t cap,
                                                  const int32_t* __restrict__ offsets,
                                                  const int32_t* __restrict__ counts,
                                                  const uint64_t* __restrict__ codes,
                                                  const uint8_t* __restrict__ hll, const uint8_t* __restrict__ hlr,
                                                  const uint8_t* __restrict__ prefix_n,
                                                  const int32_t* __restrict__ parent,
                                                  const int32_t* __restrict__ left_child, int code_bits,
                                                  DevState* st) {
    const int64_t m = (int64_t)st->n_oct;
    if (m > cap) return;
    const int64_t u = (int64_t)st->u;
    const int64_t N = u - 1;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= N) return;
    if (m >= 1) make_chain(i, m, N, nodes, offsets, counts, codes, prefix_n, parent, code_bits, st);
    link_leaves(i, m, u, nodes, offsets, counts, codes, hll, hlr, prefix_n, parent, left_child, code_bits, st);
}

// Digit histograms of given keys (the histogram half of k_encode), for
// sorting keys that were not produced by k_encode.
__global__ void __launch_bounds__(256) k_hist_keys(const uint64_t* __restrict__ keys, int64_t n, DevState* st) {
    __shared__ uint32_t s_h[kSortPasses][kSortBins];
    for (int i = threadIdx.x; i < kSortPasses * kSortBins; i += blockDim.x) (&s_h[0][0])[i] = 0;
    __syncthreads();
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
        const uint64_t c = keys[i];
#pragma unroll
        for (int p = 0; p < kSortPasses; ++p) atomicAdd(&s_h[p][(c >> (kSortBits * p)) & (kSortBins - 1)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kSortPasses * kSortBins; i += blockDim.x) {
        const uint32_t v = (&s_h[0][0])[i];
        if (v) atomicAdd(&(&st->hist[0][0])[i], v);
    }
}

// After the sort passes the result sits in buf1 when an odd number of passes
// ran; copy it back into buf0.
__global__ void __launch_bounds__(256) k_copy_if_odd(const uint64_t* __restrict__ src, uint64_t* __restrict__ dst,
                                                     int64_t n, const DevState* st) {
    if (!(st->n_active & 1)) return;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) dst[i] = src[i];
}

// Order keys of foreign queries (their places by binary search over the
// tree's codes), the digit histograms of the passes that sort them, and whether
// they come out of order at all.
__global__ void __launch_bounds__(256) k_query_keys(const float* __restrict__ q, int64_t n,
                                                    const uint64_t* __restrict__ codes, int64_t u, int code_bits,
                                                    int shift, int first, uint64_t* __restrict__ keys,
                                                    const DevState* tree, DevState* st) {
    __shared__ uint32_t s_h[kSortPasses][kSortBins];
    for (int i = threadIdx.x; i < kSortPasses * kSortBins; i += blockDim.x) (&s_h[0][0])[i] = 0;
    __syncthreads();
    const float mn = tree->min_coord, range = tree->range;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    auto place = [&](int64_t i) {
        const uint64_t code = query_to_code(q[3 * i], q[3 * i + 1], q[3 * i + 2], mn, range, code_bits);
        return (uint64_t)code_position(codes, u, code) << (shift + kOrderShift);
    };
    for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += stride) {
        const int lane = threadIdx.x & 31;
        const int64_t i = i0 + lane;
        const uint64_t at = i < n ? place(i) : ~0ull;
        if (i < n) {
            const uint64_t k = at | (uint64_t)i;
            keys[i] = k;
            for (int p = first; p < kSortPasses - 1; ++p)
                atomicAdd(&s_h[p][(k >> (kSortBits * p)) & (kSortBins - 1)], 1u);
        }
        // in order by the digits that are sorted; the step from the query before
        // the warp's first costs another search, made where all others are up
        uint64_t before = __shfl_up_sync(0xffffffffu, at, 1);
        if (lane == 0) before = 0;
        bool down = before >> (kSortBits * first) > at >> (kSortBits * first);
        if (!__any_sync(0xffffffffu, down) && lane == 0 && i0 > 0)
            down = place(i0 - 1) >> (kSortBits * first) > at >> (kSortBits * first);
        if (down) st->disorder = 1;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kSortPasses * kSortBins; i += blockDim.x) {
        const uint32_t v = (&s_h[0][0])[i];
        if (v) atomicAdd(&(&st->hist[0][0])[i], v);
    }
}

// Work items of sorted foreign queries, one thread per query: an aligned group
// of `group` queries that spans kTogetherSpan places, else its aligned parts of
// `per` queries that span kWindowSpan, else single ones. Queries far apart share
// nothing, and one warp that took several of them ended last: 250k queries that
// are tree points moved by 1e-5, a few of them far from the rest in the tree's
// order, took 736 us in parts of 16, without the few 312 us.
__global__ void __launch_bounds__(256) k_query_items(const uint64_t* __restrict__ keys, int64_t n, int shift, int per,
                                                     int group, uint64_t* __restrict__ items, DevState* tree) {
    constexpr unsigned kFull = 0xffffffffu;
    __shared__ uint32_t s_at[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    int lo = (int)(keys[min64(i, n - 1)] >> shift), hi = lo, size = 1;
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
        lo = min(lo, __shfl_xor_sync(kFull, lo, o));
        hi = max(hi, __shfl_xor_sync(kFull, hi, o));
        if (2 * o == per && hi - lo <= kWindowSpan) size = per;
        if (2 * o == group && hi - lo <= kTogetherSpan) size = group;
    }
    const uint32_t firsts = __ballot_sync(kFull, i < n && (lane & (size - 1)) == 0);
    if (lane == 0) s_at[warp] = __popc(firsts);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t total = 0;
        for (int w = 0; w < 8; ++w) {
            const uint32_t c = s_at[w];
            s_at[w] = total;
            total += c;
        }
        const uint32_t base = atomicAdd(&tree->items, total);
        for (int w = 0; w < 8; ++w) s_at[w] += base;
    }
    __syncthreads();
    if ((firsts >> lane) & 1u)
        items[s_at[warp] + __popc(firsts & lanemask_lt())] = ((uint64_t)min64(size, n - i) << 32) | (uint64_t)i;
}

inline unsigned grid_for(int64_t work, int threads, int64_t cap_blocks) {
    int64_t b = (work + threads - 1) / threads;
    if (b < 1) b = 1;
    if (cap_blocks > 0 && b > cap_blocks) b = cap_blocks;
    return (unsigned)b;
}

}  // namespace

// Onesweep's shared memory (68 KB per block) with the whole carveout for
// shared memory, so that the 3 blocks its registers allow fit on an SM.
static cudaError_t set_onesweep_attributes() {
    cudaError_t e = cudaFuncSetAttribute(k_onesweep, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)sizeof(SortSmem));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_onesweep, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
    return e;
}

cudaError_t enqueue_sort_keys(uint64_t* keys, uint64_t* tmp, int64_t n, uint32_t* lookback, DevState* st,
                              cudaStream_t s, int num_sms) {
    cudaError_t e = set_onesweep_attributes();
    if (e != cudaSuccess) return e;
    cudaMemsetAsync(st, 0, sizeof(DevState), s);
    if (n <= 0) return cudaGetLastError();
    k_hist_keys<<<grid_for(n, 256, num_sms * 4), 256, 0, s>>>(keys, n, st);
    k_sort_prep<<<1, kSortBins, 0, s>>>(n, st);
    const int64_t sort_tiles = (n + kSortTile - 1) / kSortTile;
    for (int pass = 0; pass < kSortPasses; ++pass) {
        cudaMemsetAsync(lookback, 0, sizeof(uint32_t) * kSortBins * sort_tiles, s);
        k_onesweep<<<(unsigned)sort_tiles, kSortThreads, sizeof(SortSmem), s>>>(keys, tmp, n, pass, lookback, st,
                                                                                 kSpinLimit, 0);
    }
    k_copy_if_odd<<<grid_for(n, 256, num_sms * 4), 256, 0, s>>>(tmp, keys, n, st);
    return cudaGetLastError();
}

cudaError_t enqueue_query_order(const BuildBufs& b, const QueryOrder& o, const float* queries, int64_t n, int64_t u,
                                int code_bits, const uint64_t** order, const uint64_t** items, int* shift,
                                cudaStream_t s, int num_sms, int* launches) {
    cudaError_t e = set_onesweep_attributes();
    if (e != cudaSuccess) return e;
    int bits = 1;  // places are in [0, u]
    while (((int64_t)1 << bits) <= u) ++bits;
    *shift = bits < 30 ? 30 - bits : 0;
    // A warp takes 32 queries, so a place need only be right to a few queries:
    // the top 18 bits up to 2M queries, 27 above (bits 45..62, 36..62).
    const int passes = n <= ((int64_t)1 << 21) ? 2 : 3;
    const int first = kSortPasses - 1 - passes;
    cudaMemsetAsync(o.st, 0, sizeof(DevState), s);
    k_query_keys<<<grid_for(n, 256, num_sms * 4), 256, 0, s>>>(queries, n, b.codes, u, code_bits, *shift, first, o.keys0,
                                                               b.st, o.st);
    k_sort_prep<<<1, kSortBins, 0, s>>>(n, o.st, first, kSortPasses - 1);
    const int64_t tiles = (n + kSortTile - 1) / kSortTile;
    cudaMemsetAsync(o.lookback, 0, sizeof(uint32_t) * kSortBins * tiles * passes, s);
    for (int pass = first; pass < kSortPasses - 1; ++pass)
        k_onesweep<<<(unsigned)tiles, kSortThreads, sizeof(SortSmem), s>>>(
            o.keys0, o.keys1, n, pass, o.lookback + kSortBins * tiles * (pass - first), o.st, kSpinLimit, 0);
    *order = passes & 1 ? o.keys1 : o.keys0;
    uint64_t* list = passes & 1 ? o.keys0 : o.keys1;
    k_query_items<<<grid_for(n, 256, 0), 256, 0, s>>>(*order, n, *shift + kOrderShift, queries_per_warp(n, num_sms, true),
                                                      queries_per_warp(n, num_sms, false), list, b.st);
    *items = list;
    *launches += 3 + passes;
    return cudaGetLastError();
}

template <int IPT>
static cudaError_t launch_front_n(const BuildBufs& b, int64_t n, int code_bits, const ScratchLayout& scratch,
                                  cudaStream_t s) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_front<IPT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FrontSmem<IPT>));
    if (e != cudaSuccess) return e;
    k_front<IPT><<<1, kFrontThreads, sizeof(FrontSmem<IPT>), s>>>(b.x, b.y, b.z, (int)n, code_bits, b.codes, b.pts4,
                                                                  b.pts3, b.scratch, (int)scratch.sort, b.st);
    return cudaGetLastError();
}
static cudaError_t launch_front(const BuildBufs& b, int64_t n, int code_bits, const ScratchLayout& scratch,
                                cudaStream_t s) {
    if (n <= kFrontThreads) return launch_front_n<1>(b, n, code_bits, scratch, s);
    if (n <= 2 * kFrontThreads) return launch_front_n<2>(b, n, code_bits, scratch, s);
    if (n <= 4 * kFrontThreads) return launch_front_n<4>(b, n, code_bits, scratch, s);
    return launch_front_n<8>(b, n, code_bits, scratch, s);
}

// With `again` the scan's scratch is cleared first (a build starts with it clear).
static cudaError_t launch_octree(const BuildBufs& b, const BuildParams& p, cudaStream_t s, bool again, int* launches) {
    const int64_t n = p.n;
    const int64_t scan_tiles = (n + kScanTile - 1) / kScanTile;
    unsigned long long* lookback = reinterpret_cast<unsigned long long*>(b.scratch + ScratchLayout(n).oct);
    if (again) {
        cudaMemsetAsync(lookback, 0, sizeof(unsigned long long) * scan_tiles, s);
        cudaMemsetAsync(&b.st->tile_counter[kSortPasses + 1], 0, sizeof(uint32_t), s);
    }
    OtNode* nodes = static_cast<OtNode*>(b.oct_nodes);
    k_oct_scan<<<(unsigned)scan_tiles, kScanThreads, 0, s>>>(b.prefix_n, b.parent, b.oct_counts, b.oct_offsets, lookback,
                                                             nodes, b.oct_cap, b.st, p.spin_limit);
    k_oct_make<<<grid_for(n, 256, 0), 256, 0, s>>>(nodes, b.oct_cap, b.oct_offsets, b.oct_counts, b.codes,
                                                   b.has_leaf_left, b.has_leaf_right, b.prefix_n, b.parent, b.left_child,
                                                   p.code_bits, b.st);
    if (launches) *launches += 2;
    return cudaGetLastError();
}

cudaError_t enqueue_octree(const BuildBufs& b, const BuildParams& p, cudaStream_t s, int* launches) {
    return launch_octree(b, p, s, true, launches);
}

cudaError_t enqueue_build(const BuildBufs& b, const BuildParams& p, cudaStream_t s, int num_sms, cudaEvent_t* ev,
                          int* launches) {
    int nl = 0;
    // stage i runs between events i and i+1; each stage is also an NVTX range
    static const char* const kStageNames[kBuildEvents - 1] = {
        "shapex.build.bbox", "shapex.build.encode", "shapex.build.sort", "shapex.build.dedup",
        "shapex.build.radix_tree", "shapex.build.search_boxes", "shapex.build.octree"};
    auto mark = [&](int i) {
        if (ev) cudaEventRecord(ev[i], s);
        if (i > 0) nvtxRangePop();
        if (i < kBuildEvents - 1) nvtxRangePushA(kStageNames[i]);
    };
    {
        // per device and cheap: set on every build
        cudaError_t e = set_onesweep_attributes();
        if (e != cudaSuccess) return e;
    }
    const int64_t n = p.n;
    const int passes = sort_passes(p.code_bits);
    const ScratchLayout scratch(n);
    bool front = false;
    mark(0);
    if (n <= 0) {
        cudaMemsetAsync(b.st, 0, sizeof(DevState), s);
        for (int i = 1; i < kBuildEvents; ++i) mark(i);
        if (launches) *launches = 0;
        return cudaGetLastError();
    }
    if (n <= kFrontMax && !p.stall_first_tile) {
        // one block from coordinates to unique decoded points; it also clears
        // the state and the scratch of what follows
        const cudaError_t e = launch_front(b, n, p.code_bits, scratch, s);
        if (e != cudaSuccess) {
            nvtxRangePop();
            return e;
        }
        ++nl;
        // the stages in one: stage 0 takes their time (an event between two
        // kernels costs 2.7 us, as much as a small kernel)
        if (ev) cudaEventRecord(ev[1], s);
        front = true;
    } else {
        cudaMemsetAsync(b.st, 0, sizeof(DevState), s);
        cudaMemsetAsync(b.scratch, 0, sizeof(uint32_t) * scratch.words(passes), s);
        k_bbox<<<grid_for((n + 3) / 4, 256, num_sms * 4), 256, 0, s>>>(b.x, b.y, b.z, n, b.st);
        mark(1);
        k_encode<<<grid_for(n, 256, num_sms * 4), 256, 0, s>>>(b.x, b.y, b.z, n, p.code_bits, passes, b.keys0, b.st);
        mark(2);
        nl += 2;
        const int64_t sort_tiles = (n + kSortTile - 1) / kSortTile;
        for (int pass = 0; pass < passes; ++pass) {
            k_onesweep<<<(unsigned)sort_tiles, kSortThreads, sizeof(SortSmem), s>>>(
                b.keys0, b.keys1, n, pass, b.scratch + scratch.sort + pass * scratch.sort_pass, b.st, p.spin_limit,
                p.stall_first_tile);
            ++nl;
        }
        mark(3);
        const int64_t dd_tiles = (n + kDedupTile - 1) / kDedupTile;
        k_dedup<<<(unsigned)dd_tiles, kDedupThreads, 0, s>>>(b.keys0, b.keys1, n, p.code_bits, b.codes, b.pts4, b.pts3,
                                                             b.scratch + scratch.dedup, b.st, p.spin_limit);
        ++nl;
    }
    if (!front) mark(4);
    if (p.build_radix) {
        k_karras<<<grid_for(n, 256, 0), 256, 0, s>>>(b.codes, p.code_bits, p.root_compat, b.left_child, b.parent,
                                                     b.prefix_n, b.has_leaf_left, b.has_leaf_right, b.sparent,
                                                     b.leaf_parent, b.range_end, b.st);
        ++nl;
    }
    mark(5);
    const int64_t leaf_tiles = (n + kLeafTile - 1) / kLeafTile;
    k_leaves<<<(unsigned)leaf_tiles, kLeafThreads, 0, s>>>(
        b.codes, p.bucket < kLeafMax ? p.bucket : kLeafMax, b.leaf_start, b.scratch + scratch.leaves,
        p.build_radix && p.root_compat, b.left_child, b.parent, b.has_leaf_left, b.has_leaf_right, b.st, p.spin_limit);
    // 32 leaves per warp, about 20 points each: a grid for four warps per 1024
    // points (per 4096 the warps took several groups in turn: 100k points 32 us for
    // leaves and boxes, now 26; 2M 62 and 50 us)
    k_boxes<<<grid_for(n, 1024, num_sms * 8), 128, 0, s>>>(b.pts4, b.leaf_start, b.scratch + scratch.arrivals,
                                                               b.snodes, b.st);
    nl += 2;
    mark(6);
    if (p.build_octree) {
        cudaError_t e = launch_octree(b, p, s, false, &nl);
        if (e != cudaSuccess) {
            nvtxRangePop();  // the octree stage's range
            return e;
        }
    }
    mark(7);
    if (launches) *launches = nl;
    return cudaGetLastError();
}

}  // namespace shapex
