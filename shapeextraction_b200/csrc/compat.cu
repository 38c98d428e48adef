// Reference-compatible kNN search and normals.
//
// Reproduces the reference's approximate search bit-exactly on the GPU:
// knnSearchKernel<k> (src/Octree.hpp:136-193) walks the OTNode array best
// first with a bounded search heap of 32 node slots (SEARCH_Q_SIZE,
// src/Octree.hpp:17) and a result heap of k point slots, both the bounded
// min-max heap of src/dequeue.hpp:55-289 (a full heap drops its largest
// priority when the new one is not larger, src/dequeue.hpp:60-67). Node
// priority is nodeBoxDistance (src/Octree.cu:326-352): 0 inside the cube,
// else the smallest distance to one of its six face planes. Point priority is
// Point::distance2 (src/PointCloud.hpp:30-35) as nvcc contracts it,
// fma(dz, dz, fma(dx, dx, dy*dy)). The search runs until the node heap is
// empty (the early stop of src/Octree.hpp:152-155 never fires because its
// bound is never updated). Results leave the result heap in remove-min order;
// a query with fewer than k results repeats its first one
// (src/Octree.hpp:181-191).
//
// The normals of this mode follow estimateNormals (src/NormalEstimation.hpp:
// 96-192): centroid as a plain FP32 sum divided by k, covariance as FP32 fmas
// of the centred points divided by k-1, in the neighbours' output order; the
// 3x3 eigensolve, done by a closed library in the reference, is the FP64
// Jacobi of the exact mode on that FP32 matrix; orientation towards the
// viewpoint.
//
// Layout: one thread per query. Both heaps live in shared memory as
// [slot][thread] arrays, so the threads of a warp touch 32 distinct banks
// whatever slots they address. Queries are the tree's Morton-ordered points
// (or caller queries), so neighbouring threads walk similar paths.
//
// Bound by divergence and the latency of dependent node loads: every thread's
// heaps take their own paths, and walks differ in length (488 pops on average,
// 1305 for the longest of 32, on a 200k-point scene). So threads are persistent
// and take a new query as soon as theirs ends (waiting until 4, 8 or 16 of a
// warp have ended, to write results together: 19.7, 20.7, 22.3 ms against 18.9);
// each step a thread pops if it has dealt with its node, and inserts one thing,
// its next point that the results take or its next child node, through one copy
// of the code; an item on its way through a heap is carried in registers and
// written once; one loop climbs minimum and maximum levels alike. 200k points,
// k = 16: 53.2 ms with one query per thread in lockstep over the eight child
// numbers, 31.7 ms with the carried items and each thread's own next child,
// 18.9 ms now (of 100k points: 3.6 G warp instructions, 8 of 32 threads in each).

#include <cstdint>

#include "eig3.cuh"
#include "pipeline.cuh"

namespace shapex {

namespace {

constexpr int kCompatThreads = 64;
constexpr int kSearchSlots = 32;  // SEARCH_Q_SIZE, src/Octree.hpp:17

// Bounded min-max heap over one thread's column of [slot][thread] arrays.
// Even levels are min levels, odd levels max levels (src/dequeue.hpp:55-289).
struct ColumnHeap {
    float* pri;     // pri[slot * kCompatThreads]
    int32_t* item;  // item[slot * kCompatThreads]
    int size;
    int cap;

    __device__ __forceinline__ float P(int i) const { return pri[i * kCompatThreads]; }
    __device__ __forceinline__ int32_t I(int i) const { return item[i * kCompatThreads]; }
    __device__ __forceinline__ void put(int i, float p, int32_t it) {
        pri[i * kCompatThreads] = p;
        item[i * kCompatThreads] = it;
    }
    static __device__ __forceinline__ int par(int i) { return (i - 1) / 2; }
    static __device__ __forceinline__ int lc(int i) { return 2 * i + 1; }
    static __device__ __forceinline__ int rc(int i) { return 2 * i + 2; }
    static __device__ __forceinline__ bool min_level(int i) { return ((31 - __clz(i + 1)) & 1) == 0; }

    __device__ __forceinline__ int largest() const {
        if (size >= 3) return P(1) > P(2) ? 1 : 2;
        return size - 1;  // 1 of two, 0 of one
    }
    // smallest (MIN) or largest (!MIN) of i's children and grandchildren,
    // first in the order lc, rc, lc(lc), rc(lc), lc(rc), rc(rc) on ties
    template <bool MIN>
    __device__ __forceinline__ int pick(int i, float& pm) const {
        int m = lc(i);
        pm = P(m);
        const int desc[5] = {rc(i), lc(lc(i)), rc(lc(i)), lc(rc(i)), rc(rc(i))};
#pragma unroll
        for (int d = 0; d < 5; ++d) {
            if (desc[d] < size) {
                const float pd = P(desc[d]);
                if (MIN ? pd < pm : pd > pm) {
                    m = desc[d];
                    pm = pd;
                }
            }
        }
        return m;
    }
    // Place item (w, it) at slot i or below it (percolate of src/dequeue.hpp),
    // i on a minimum level (MIN) or a maximum level (!MIN).
    template <bool MIN>
    __device__ __forceinline__ void down(int i, float w, int32_t it) {
        while (lc(i) < size) {
            float pm;
            const int m = pick<MIN>(i, pm);
            if (!(MIN ? pm < w : pm > w)) break;
            put(i, pm, I(m));
            const bool grandchild = m > rc(i);
            i = m;
            if (!grandchild) break;
            const int q = par(m);
            const float pp = P(q);
            if (MIN ? w > pp : w < pp) {  // the carried item stays at the parent, the parent's goes on
                const int32_t pit = I(q);
                put(q, w, it);
                w = pp;
                it = pit;
            }
        }
        put(i, w, it);
    }
    __device__ __forceinline__ void remove_min(float& p, int32_t& it) {
        p = P(0);
        it = I(0);
        --size;
        down<true>(0, P(size), I(size));
    }
    // Insert; the caller has checked that a full heap's largest is not below w.
    __device__ __forceinline__ void insert(int32_t it, float w) {
        if (size == cap) {  // drop the largest
            const int l = largest();
            --size;
            if (l > 0) down<false>(l, P(size), I(size));
        }
        int i = size++;
        bool lvl = min_level(i);
        if (i > 0) {
            const int q = par(i);
            const float pq = P(q);
            if (lvl ? w > pq : w < pq) {
                put(i, pq, I(q));
                i = q;
                lvl = !lvl;
            }
        }
        while (i >= 3) {
            const int g = par(par(i));
            const float pg = P(g);
            if (!(lvl ? w < pg : w > pg)) break;
            put(i, pg, I(g));
            i = g;
        }
        put(i, w, it);
    }
    // Whether insert() would keep an item of priority w (src/dequeue.hpp:60-67).
    __device__ __forceinline__ bool takes(float w) const { return size < cap || P(largest()) >= w; }
};

// nodeBoxDistance, src/Octree.cu:326-352
__device__ __forceinline__ float face_distance(float qx, float qy, float qz, const OtNode& n) {
    const float x1 = n.corner[0], x2 = __fadd_rn(n.corner[0], n.cell_size);
    const float y1 = n.corner[1], y2 = __fadd_rn(n.corner[1], n.cell_size);
    const float z1 = n.corner[2], z2 = __fadd_rn(n.corner[2], n.cell_size);
    if (qx > x1 && qx < x2 && qy > y1 && qy < y2 && qz > z1 && qz < z2) return 0.0f;
    float m = fabsf(__fsub_rn(qx, x1));
    m = fminf(m, fabsf(__fsub_rn(qx, x2)));
    m = fminf(m, fabsf(__fsub_rn(qy, y1)));
    m = fminf(m, fabsf(__fsub_rn(qy, y2)));
    m = fminf(m, fabsf(__fsub_rn(qz, z1)));
    m = fminf(m, fabsf(__fsub_rn(qz, z2)));
    return m;
}

// Point::distance2 as the reference build contracts it
__device__ __forceinline__ float ref_distance2(float qx, float qy, float qz, float4 p) {
    const float dx = __fsub_rn(qx, p.x), dy = __fsub_rn(qy, p.y), dz = __fsub_rn(qz, p.z);
    return __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
}

struct CompatArgs {
    int k;
    int64_t start, count, u, m;
    const float* ext;
    int32_t* out_idx;
    float* out_d2;
    float* out_normals;
    float vx, vy, vz;
};

// One thread's finished query: its results in remove-min order and, with
// NORMALS, its normal. The order goes into the (empty) node heap's column so
// that the covariance reads the neighbours in it.
template <bool NORMALS>
__device__ __forceinline__ void write_results(ColumnHeap& rq, int32_t* order, float* order_d2, float qx, float qy,
                                              float qz, int64_t qi, const float4* __restrict__ pts,
                                              const CompatArgs& a) {
    int32_t first = -1;
    float first_d2 = __int_as_float(0x7f800000);
    for (int c = 0; c < a.k; ++c) {
        int32_t it;
        float p;
        if (rq.size == 0) {
            it = first;
            p = first_d2;
        } else {
            rq.remove_min(p, it);
        }
        if (c == 0) {
            first = it;
            first_d2 = p;
        }
        order[c * kCompatThreads] = it;
        order_d2[c * kCompatThreads] = p;
    }
    if (a.out_idx) {
        for (int c = 0; c < a.k; ++c) a.out_idx[qi * a.k + c] = order[c * kCompatThreads];
        if (a.out_d2)
            for (int c = 0; c < a.k; ++c) a.out_d2[qi * a.k + c] = order_d2[c * kCompatThreads];
    }
    if (NORMALS) {
        float* out = a.out_normals + 3 * qi;
        if (first < 0) {
            out[0] = out[1] = out[2] = __int_as_float(0x7fc00000);
        } else {
            // calculateCovariance<k>, src/NormalEstimation.hpp:96-120
            float cx = 0.0f, cy = 0.0f, cz = 0.0f;
            for (int c = 0; c < a.k; ++c) {
                const float4 p = __ldg(pts + order[c * kCompatThreads]);
                cx = __fadd_rn(cx, p.x);
                cy = __fadd_rn(cy, p.y);
                cz = __fadd_rn(cz, p.z);
            }
            const float fk = (float)a.k;
            cx = __fdiv_rn(cx, fk);
            cy = __fdiv_rn(cy, fk);
            cz = __fdiv_rn(cz, fk);
            float cv[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
            for (int c = 0; c < a.k; ++c) {
                const float4 p = __ldg(pts + order[c * kCompatThreads]);
                const float m0 = __fsub_rn(p.x, cx), m1 = __fsub_rn(p.y, cy), m2 = __fsub_rn(p.z, cz);
                cv[0] = __fmaf_rn(m0, m0, cv[0]);
                cv[1] = __fmaf_rn(m0, m1, cv[1]);
                cv[2] = __fmaf_rn(m0, m2, cv[2]);
                cv[3] = __fmaf_rn(m1, m1, cv[3]);
                cv[4] = __fmaf_rn(m1, m2, cv[4]);
                cv[5] = __fmaf_rn(m2, m2, cv[5]);
            }
            const float den = (float)(a.k - 1);
            double C[6];
#pragma unroll
            for (int e = 0; e < 6; ++e) C[e] = (double)__fdiv_rn(cv[e], den);
            double w[3], nv[3];
            eig3<double>(C, w, nv);
            float nx = (float)nv[0], ny = (float)nv[1], nz = (float)nv[2];
            // normalsFromEigenVectors, src/NormalEstimation.hpp:158-192
            const float dot = (a.vx - qx) * nx + (a.vy - qy) * ny + (a.vz - qz) * nz;
            if (dot < 0.0f) {
                nx = -nx;
                ny = -ny;
                nz = -nz;
            }
            out[0] = nx;
            out[1] = ny;
            out[2] = nz;
        }
    }
}

template <bool EXT, bool NORMALS>
__global__ void __launch_bounds__(kCompatThreads)
    k_knn_compat(const OtNode* __restrict__ nodes, const float4* __restrict__ pts, CompatArgs a, DevState* st) {
    constexpr unsigned kFull = 0xffffffffu;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31;
    float* s_pri = reinterpret_cast<float*>(smem_raw) + tid;
    int32_t* s_item = reinterpret_cast<int32_t*>(s_pri + kSearchSlots * kCompatThreads);
    float* r_pri = reinterpret_cast<float*>(s_item + kSearchSlots * kCompatThreads);
    int32_t* r_item = reinterpret_cast<int32_t*>(r_pri + a.k * kCompatThreads);
    ColumnHeap sq{s_pri, s_item, 0, kSearchSlots};
    ColumnHeap rq{r_pri, r_item, 0, a.k};
    uint32_t err = 0;
    float qx = 0.0f, qy = 0.0f, qz = 0.0f;
    uint32_t qi = 0;
    bool live = false;       // the thread has a query
    bool more = true;        // the counter still had queries (the same for the whole warp)
    // the popped node's points and child nodes not dealt with yet
    uint32_t leaf_mask = 0, node_mask = 0;
    const int32_t* child = nullptr;
    // every node enters the heap at most once (children of a popped node), so
    // a walk of more than m pops means a malformed octree
    int32_t pops = 0;
    for (;;) {
        // A thread whose walk has ended writes its results and takes a new query.
        const bool ended = live && sq.size == 0 && !(leaf_mask | node_mask);
        const uint32_t idle = __ballot_sync(kFull, ended || !live);
        if (idle == kFull || (more && idle)) {
            if (ended) {
                write_results<NORMALS>(rq, s_item, s_pri, qx, qy, qz, qi, pts, a);
                live = false;
            }
            __syncwarp();
            if (!more) break;
            const uint32_t want = __ballot_sync(kFull, !live);
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&st->work, (uint32_t)__popc(want));
            base = __shfl_sync(kFull, base, 0);
            more = (int64_t)base + __popc(want) < a.count;
            qi = live ? qi : base + __popc(want & lanemask_lt());
            if (!live && qi < a.count) {
                if (EXT) {
                    qx = a.ext[3 * (int64_t)qi];
                    qy = a.ext[3 * (int64_t)qi + 1];
                    qz = a.ext[3 * (int64_t)qi + 2];
                } else {
                    const float4 q = pts[a.start + qi];
                    qx = q.x;
                    qy = q.y;
                    qz = q.z;
                }
                live = true;
                rq.size = 0;
                pops = 0;
                sq.size = 1;
                sq.put(0, 0.0f, 0);  // the root
            }
            __syncwarp();
        }
        // threads that have dealt with their node pop the next
        if (!(leaf_mask | node_mask) && sq.size > 0) {
            float pr;
            int32_t ni;
            sq.remove_min(pr, ni);
            child = nodes[ni].children;
            node_mask = (uint32_t)nodes[ni].child_node_mask & 0xffu;
            leaf_mask = (uint32_t)nodes[ni].child_leaf_mask & 0xffu;
            if (++pops > a.m) {
                err |= ERRBIT_SEARCH_LIMIT;
                sq.size = 0;
                leaf_mask = node_mask = 0;
            }
        }
        __syncwarp();
        // one insertion per thread: its next point that the results take, or
        // else its next child node (the two heaps are independent)
        bool take = false, leaf = false;
        int32_t it = 0;
        float w = 0.0f;
        while (leaf_mask && !take) {
            const int c = __ffs(leaf_mask) - 1;
            leaf_mask &= leaf_mask - 1;
            it = child[c];
            if (it < 0 || it >= a.u) {
                err |= ERRBIT_BOUNDS;
                continue;
            }
            w = ref_distance2(qx, qy, qz, __ldg(pts + it));
            take = leaf = rq.takes(w);
        }
        __syncwarp();
        if (!take && node_mask) {
            const int c = __ffs(node_mask) - 1;
            node_mask &= node_mask - 1;
            it = child[c];
            if (it < 0 || it >= a.m) {
                err |= ERRBIT_BOUNDS;
            } else {
                w = face_distance(qx, qy, qz, nodes[it]);
                take = sq.takes(w);
            }
        }
        __syncwarp();
        if (take) {
            ColumnHeap h{leaf ? r_pri : s_pri, leaf ? r_item : s_item, leaf ? rq.size : sq.size,
                         leaf ? a.k : kSearchSlots};
            h.insert(it, w);
            if (leaf) rq.size = h.size;
            else sq.size = h.size;
        }
        __syncwarp();
    }
    if (err) atomicOr(&st->err, err);
}

template <bool EXT, bool NORMALS>
cudaError_t launch_compat(const BuildBufs& b, const CompatArgs& a, cudaStream_t s, int num_sms) {
    const int smem = (kSearchSlots + a.k) * kCompatThreads * 8;
    cudaError_t e = cudaFuncSetAttribute(k_knn_compat<EXT, NORMALS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_knn_compat<EXT, NORMALS>, kCompatThreads, smem);
    if (e != cudaSuccess) return e;
    const int64_t want = (a.count + kCompatThreads - 1) / kCompatThreads;
    const int64_t resident = (int64_t)(per_sm > 0 ? per_sm : 1) * num_sms;
    const unsigned blocks = (unsigned)(want < resident ? want : resident);
    k_knn_compat<EXT, NORMALS><<<blocks, kCompatThreads, smem, s>>>(static_cast<const OtNode*>(b.oct_nodes), b.pts4,
                                                                    a, b.st);
    return cudaGetLastError();
}

}  // namespace

cudaError_t enqueue_query_compat(const BuildBufs& b, const QueryParams& q, cudaStream_t s, int num_sms) {
    if (q.count <= 0) return cudaSuccess;
    if (q.k < 1 || q.k > 32 || q.n_octree < 1 || !b.oct_nodes) return cudaErrorInvalidValue;
    CompatArgs a;
    a.k = q.k;
    a.start = q.start;
    a.count = q.count;
    a.u = q.u;
    a.m = q.n_octree;
    a.ext = q.ext_queries;
    a.out_idx = q.out_idx;
    a.out_d2 = q.out_d2;
    a.out_normals = q.out_normals;
    a.vx = q.vx;
    a.vy = q.vy;
    a.vz = q.vz;
    if (a.ext) return launch_compat<true, false>(b, a, s, num_sms);
    if (a.out_normals) return launch_compat<false, true>(b, a, s, num_sms);
    return launch_compat<false, false>(b, a, s, num_sms);
}

}  // namespace shapex
