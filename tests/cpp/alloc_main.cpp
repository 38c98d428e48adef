// Allocation failures inside the C ABI, on the CPU. The host code of the entry
// points (capi.cu, capi_mlp.cu, capi_batch.cu: no kernels) is linked against
// stand-ins for the CUDA runtime (alloc_runtime.cpp) and the kernel launchers
// (below). Device memory is host memory, every launcher checks that each buffer it is handed is
// alive and large enough and fills its outputs, and the runtime fails one
// allocation of a call on request.
//
// A scenario is a small, a middle and a large call on one context. For every
// allocation of the small call on a new context, and of the large call after
// the small one: that allocation fails, the call says so (or, where it copes,
// works all the same), and the three calls then work.
#include <cstdio>
#include <functional>
#include <set>
#include <string>
#include <utility>
#include <vector>

#include "alloc_runtime.hpp"
#include "pipeline.cuh"
#include "shapex.h"

using namespace shapex;
using fake::complain;
using fake::live;

// ---- the kernel launchers ----------------------------------------------------
static std::set<std::pair<int, int>> g_shapes;  // leaf sizes of the builds, blocks per SM of the shared launches
static int g_batches = 0;                       // batched calls

namespace shapex {
static void fill(float* p, int64_t n) {
    for (int64_t i = 0; i < n; ++i) p[i] = 7.0f;
}
cudaError_t enqueue_build(const BuildBufs& b, const BuildParams& p, cudaStream_t, int, cudaEvent_t*, int* launches) {
    const int64_t n = p.n;
    if (launches) *launches = 1;
    g_shapes.insert({p.bucket < kLeafMax ? p.bucket : kLeafMax, -1});
    if (!live(b.st, sizeof(DevState), "build: st")) return cudaErrorInvalidValue;
    *b.st = DevState{};
    if (n == 0) return cudaSuccess;
    bool ok = live(b.x, 4 * n, "build: x") && live(b.y, 4 * n, "build: y") && live(b.z, 4 * n, "build: z") &&
              live(b.keys0, 8 * n, "build: keys0") && live(b.keys1, 8 * n, "build: keys1") &&
              live(b.scratch, 4 * ScratchLayout(n).words(kCodePasses), "build: scratch") &&
              live(b.codes, 8 * n, "build: codes") && live(b.pts4, 16 * n, "build: pts4") &&
              live(b.pts3, 12 * n, "build: pts3") && live(b.leaf_start, 4 * n, "build: leaf_start") &&
              live(b.snodes, sizeof(SNode) * hierarchy_nodes(n), "build: snodes");
    if (ok && p.build_radix)
        ok = live(b.left_child, 4 * n, "build: left_child") && live(b.parent, 4 * n, "build: parent") &&
             live(b.prefix_n, n, "build: prefix_n") && live(b.has_leaf_left, n, "build: has_leaf_left") &&
             live(b.has_leaf_right, n, "build: has_leaf_right") && live(b.sparent, 4 * n, "build: sparent") &&
             live(b.leaf_parent, 4 * n, "build: leaf_parent") && live(b.range_end, 4 * n, "build: range_end");
    if (ok && p.build_octree)
        ok = live(b.oct_counts, 4 * n, "build: oct_counts") && live(b.oct_offsets, 4 * n + 4, "build: oct_offsets") &&
             live(b.oct_nodes, sizeof(OtNode) * b.oct_cap, "build: oct_nodes");
    if (!ok) return cudaErrorInvalidValue;
    b.st->u = (unsigned long long)n;
    b.st->n_oct = 1;
    return cudaSuccess;
}
cudaError_t enqueue_octree(const BuildBufs&, const BuildParams&, cudaStream_t, int*) { return cudaSuccess; }
bool order_foreign(int64_t count, int64_t, int, int) { return count > 5000; }
bool list_points(int64_t, int, int) { return false; }
cudaError_t enqueue_query_order(const BuildBufs&, const QueryOrder& o, const float* q, int64_t n, int64_t, int,
                                const uint64_t** order, const uint64_t** items, int* shift, cudaStream_t, int,
                                int* launches) {
    const int64_t tiles = (n + kSortTile - 1) / kSortTile;
    if (!(live(q, 12 * n, "order: queries") && live(o.keys0, 8 * n, "order: keys0") &&
          live(o.keys1, 8 * n, "order: keys1") && live(o.lookback, 3 * 4 * tiles * kSortBins, "order: lookback") &&
          live(o.st, sizeof(DevState), "order: st")))
        return cudaErrorInvalidValue;
    *order = o.keys0;
    *items = o.keys1;
    *shift = 0;
    ++*launches;
    return cudaSuccess;
}
cudaError_t enqueue_query(const BuildBufs& b, const QueryParams& q, cudaStream_t, int) {
    bool ok = live(b.st, sizeof(DevState), "query: st") && live(b.pts4, 16 * q.u, "query: pts4") &&
              live(b.snodes, sizeof(SNode), "query: snodes");
    if (q.ext_queries) ok = live(q.ext_queries, 12 * q.count, "query: queries") && ok;
    if (q.order) ok = live(q.order, 8 * q.count, "query: order") && ok;
    if (q.learned_r2) ok = live(q.learned_r2, 4 * q.count, "query: learned_r2") && ok;
    if (q.cell_lut) ok = live(q.cell_lut, 4, "query: cell_lut") && ok;
    if (q.out_idx) ok = live(q.out_idx, 4 * q.k * q.count, "query: out_idx") && ok;
    if (q.out_d2) ok = live(q.out_d2, 4 * q.k * q.count, "query: out_d2") && ok;
    if (q.out_normals) ok = live(q.out_normals, 12 * q.count, "query: out_normals") && ok;
    if (!ok) return cudaErrorInvalidValue;
    for (int64_t i = 0; q.out_idx && i < q.k * q.count; ++i) q.out_idx[i] = 7;
    if (q.out_d2) fill(q.out_d2, q.k * q.count);
    if (q.out_normals) fill(q.out_normals, 3 * q.count);
    return cudaSuccess;
}
cudaError_t enqueue_query_batch(const BatchCloud* clouds, int n_clouds, int64_t, unsigned long long* counter,
                                const QueryParams& q, cudaStream_t, int) {
    g_shapes.insert({-1, q.batch_blocks_per_sm});
    if (!(live(clouds, sizeof(BatchCloud) * n_clouds, "batch: descriptors") && live(counter, 8, "batch: counter")))
        return cudaErrorInvalidValue;
    for (int i = 0; i < n_clouds; ++i) {
        const BatchCloud& d = clouds[i];
        if (!(live(d.st, sizeof(DevState), "batch: st") && live(d.pts, 16 * d.st->u, "batch: pts") &&
              live(d.snodes, sizeof(SNode), "batch: snodes") && live(d.out_normals, 12 * d.st->u, "batch: out")))
            return cudaErrorInvalidValue;
        fill(d.out_normals, 3 * (int64_t)d.st->u);
    }
    return cudaSuccess;
}
cudaError_t enqueue_batch_collect(const DevState* st, int n, unsigned long long* u, uint32_t* err, cudaStream_t) {
    ++g_batches;
    for (int i = 0; i < n; ++i) {
        u[i] = st[i].u;
        err[i] = st[i].err;
    }
    return cudaSuccess;
}
cudaError_t enqueue_cell_lut(const BuildBufs&, int, int level, uint32_t* lut, cudaStream_t, int) {
    return live(lut, 4 * (((int64_t)1 << (3 * level)) + 1), "cell table") ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t enqueue_features(const BuildBufs&, int64_t, int, int64_t, int64_t count, float* out, cudaStream_t) {
    if (!live(out, 4 * kMlpF * count, "features")) return cudaErrorInvalidValue;
    fill(out, kMlpF * count);
    return cudaSuccess;
}
cudaError_t enqueue_predict_radius(const BuildBufs&, const float* params, float, int64_t, int, int64_t, int64_t count,
                                   float* r2, float* yhat, cudaStream_t) {
    if (!live(params, 4 * kMlpParams, "predict: params")) return cudaErrorInvalidValue;
    if (r2 && !live(r2, 4 * count, "predict: r2")) return cudaErrorInvalidValue;
    if (yhat && !live(yhat, 4 * count, "predict: yhat")) return cudaErrorInvalidValue;
    if (r2) fill(r2, count);
    if (yhat) fill(yhat, count);
    return cudaSuccess;
}
cudaError_t enqueue_mlp_forward(const float* params, const float* X, int64_t n, float* yhat, float*, float*,
                                cudaStream_t) {
    if (!(live(params, 4 * kMlpParams, "forward: params") && live(X, 4 * kMlpF * n, "forward: X") &&
          live(yhat, 4 * n, "forward: yhat")))
        return cudaErrorInvalidValue;
    fill(yhat, n);
    return cudaSuccess;
}
cudaError_t enqueue_mlp_grad(const float* params, const float* X, const float* y, int64_t n, float, float* grads,
                             float* loss, cudaStream_t, int) {
    if (!(live(params, 4 * kMlpParams, "grad: params") && live(X, 4 * kMlpF * n, "grad: X") && live(y, 4 * n, "grad: y") &&
          live(grads, 4 * kMlpParams, "grad: grads") && live(loss, 4, "grad: loss")))
        return cudaErrorInvalidValue;
    *loss += 7.0f;
    return cudaSuccess;
}
cudaError_t enqueue_adam(float* params, float* grads, float* m, float* v, float, int, cudaStream_t) {
    const bool ok = live(params, 4 * kMlpParams, "adam: params") && live(grads, 4 * kMlpParams, "adam: grads") &&
                    live(m, 4 * kMlpParams, "adam: m") && live(v, 4 * kMlpParams, "adam: v");
    return ok ? cudaSuccess : cudaErrorInvalidValue;
}
}  // namespace shapex

// ---- scenarios ---------------------------------------------------------------
// A call of size s (0 small, 1 middle, 2 large) on the context: its status, or
// -1 when it succeeded with outputs missing.
using Call = std::function<int(se_ctx*, int)>;

template <typename T>
static int written(int status, const std::vector<T>& out) {
    if (status != SE_OK) return status;
    for (const T& v : out)
        if (v != T(7)) return -1;
    return SE_OK;
}

static int train(se_ctx* c, int s) {
    const int steps = s == 0 ? 3 : (s == 1 ? 5 : 9);
    std::vector<float> X(kMlpF * 64), y(64), losses(steps);
    if (int rc = se_mlp_init(c, 1)) return rc;
    return written(se_mlp_train(c, X.data(), y.data(), 64, steps, 16, 1e-3f, losses.data(), SE_MEM_HOST), losses);
}

// Host arrays; `points` scales the clouds, the larger calls have more of them.
static int batch(se_ctx* c, int s, int points) {
    std::vector<int64_t> off{0}, u;
    std::vector<int32_t> ks;
    for (int i = 0; i < 2 + s; ++i) {
        off.push_back(off.back() + points * (2 * s + 1) - 7 * i);
        ks.push_back(i % 2 ? 8 : 16);
    }
    u.resize(ks.size());
    const int64_t n = off.back();
    std::vector<float> x(n), out(3 * n);
    return written(se_normals_batch(c, x.data(), x.data(), x.data(), off.data(), (int)ks.size(), ks.data(), out.data(),
                                    u.data(), SE_MEM_HOST),
                   out);
}

static int build(se_ctx* c, int n) {
    std::vector<float> x(n);
    return se_build(c, x.data(), x.data(), x.data(), n, SE_MEM_HOST);
}

// Host arrays: foreign queries, lists, normals (with a learned radius when the
// context has one).
static int queries(se_ctx* c, int s) {
    const int n = 700 * (s + 1), k = 5;
    if (int rc = se_mlp_init(c, 1)) return rc;
    if (int rc = build(c, n)) return rc;
    std::vector<float> q(3 * n), d2(k * n), normals(3 * n);
    std::vector<int32_t> idx(k * n), mine(k * n);
    if (int rc = written(se_knn(c, k, q.data(), n, idx.data(), nullptr, SE_MEM_HOST), idx)) return rc;
    if (int rc = written(se_knn_self(c, k, 0, n, mine.data(), d2.data(), SE_MEM_HOST), mine)) return rc;
    if (int rc = written(SE_OK, d2)) return rc;
    return written(se_normals(c, k, 0, n, normals.data(), SE_MEM_HOST), normals);
}

// Foreign queries on device arrays, enough of them to be ordered: the order's
// buffers are all that the call allocates.
static int foreign(se_ctx* c, int s) {
    const int n = 6000 * (s + 1), k = 5;
    std::vector<float> q(3 * n);
    std::vector<int32_t> idx(k * n);
    fake::Device dq(q.data(), 4 * q.size()), di(idx.data(), 4 * idx.size());
    return written(se_knn(c, k, (float*)q.data(), n, idx.data(), nullptr, SE_MEM_DEVICE), idx);
}

// The radius model's entry points on host arrays.
static int model(se_ctx* c, int s) {
    const int n = 40 * (s + 1);
    if (int rc = se_mlp_init(c, 1)) return rc;
    if (int rc = build(c, n)) return rc;
    std::vector<float> X(kMlpF * n), y(n), r2(n), out(n), grads(kMlpParams);
    float loss = 0.0f;
    if (int rc = written(se_mlp_predict(c, 0, n, y.data(), r2.data(), SE_MEM_HOST), y)) return rc;
    if (int rc = written(SE_OK, r2)) return rc;
    if (int rc = written(se_mlp_forward(c, X.data(), n, out.data(), SE_MEM_HOST), out)) return rc;
    if (int rc = se_mlp_grad(c, X.data(), y.data(), n, grads.data(), &loss, SE_MEM_HOST)) return rc;
    if (loss != 7.0f) return -1;
    return written(se_features(c, 0, n, X.data(), SE_MEM_HOST), X);
}

static int check(const char* name, const se_options& opt, const Call& call, bool copes = false,
                 int (*prepare)(se_ctx*) = nullptr) {
    int allocs = 0;
    for (const bool fresh : {true, false}) {  // the first call's allocations, those of a larger call
        const std::string title = std::string(name) + (fresh ? ", first call" : ", larger call");
        const int size = fresh ? 0 : 2;
        int n = 1;
        for (int i = 0; i <= n; ++i) {  // i = 0: none fails, which counts them
            fake::where = title + ", allocation " + std::to_string(i) + " of " + std::to_string(n);
            se_ctx* c = nullptr;
            se_create(&c, &opt);
            if (prepare) prepare(c);
            if (!fresh && call(c, 0) != SE_OK) complain("the small call failed");
            const int before = fake::allocs;
            if (i > 0) fake::fail_at = before + i;
            const int rc = call(c, size);
            fake::fail_at = 0;
            if (i == 0) n = fake::allocs - before;
            if (rc != (i == 0 || copes ? SE_OK : SE_ERR_OOM))
                complain(copes ? "the call failed or left outputs out" : "its failure is not reported");
            if (call(c, 0) != SE_OK) complain("the small call after it failed or left outputs out");
            if (call(c, 1) != SE_OK) complain("the middle call after it failed or left outputs out");
            if (call(c, 2) != SE_OK) complain("the large call after it failed or left outputs out");
            se_destroy(c);
        }
        allocs += n;
    }
    if (fake::blocks() > 0) complain("memory left after se_destroy");
    std::printf("%s: %d allocations\n", name, allocs);
    return allocs;
}

// The batch tuner times no schedule twice: no leaf sizes (all those it tried
// were the same), no limits of the blocks per SM, no cut-offs with the same
// clouds above them.
static int tuner(const se_options& opt) {
    fake::where = "tuner";
    se_ctx* c = nullptr;
    se_create(&c, &opt);
    for (const int big : {1000, 40000}) {
        const std::vector<int64_t> off{0, 500, 500 + big, 500 + 2 * big, 500 + 3 * big};
        const std::vector<int32_t> ks{8, 8, 8, 16};
        std::vector<float> x(off.back());
        g_shapes.clear();
        g_batches = 0;
        se_batch_tuning best;
        float ms = 0.0f;
        if (se_tune_batch(c, x.data(), x.data(), x.data(), off.data(), 4, ks.data(), SE_MEM_HOST, 1, &best, &ms) != SE_OK)
            complain("failed");
        if (g_shapes.size() != 2) complain("tried leaf sizes or blocks per SM");
        // two calls each: the present setting; per round 3 halos, the other block shape and,
        // where clouds lie above 32768 points, that cut-off (4 clouds take 4 lanes at most)
        if (g_batches != 2 * (1 + 2 * (3 + 1 + (big > 32768)))) complain("other schedules than expected");
        std::printf("tuner: %d batches\n", g_batches);
    }
    se_destroy(c);
    return fake::bad;
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    se_options opt;
    se_options_init(&opt);
    opt.batch_graph = 0;
    int allocs = 0;
    if (what == "tuner") return tuner(opt) ? 1 : 0;
    if (what == "train") allocs = check("train", opt, train);
    if (what == "batch slices") {
        opt.batch_lanes = 1;  // one lane, never regrown: it holds 1024 points at least
        allocs = check("batch slices", opt, [](se_ctx* c, int s) { return batch(c, s, 50); });
    }
    if (what == "queries") allocs = check("queries", opt, queries);
    if (what == "learned") {
        opt.learned = opt.learned_skip_seed = opt.learned_cell_scan = 1;
        allocs = check("learned", opt, queries);
    }
    if (what == "foreign") allocs = check("foreign", opt, foreign, true, [](se_ctx* c) { return build(c, 100); });
    if (what == "model") allocs = check("model", opt, model);
    if (what == "batch lanes") allocs = check("batch lanes", opt, [](se_ctx* c, int s) { return batch(c, s, 2000); });
    if (allocs == 0) complain("no such scenario, or nothing allocated in it");
    return fake::bad ? 1 : 0;
}
