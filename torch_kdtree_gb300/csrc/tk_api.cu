// C ABI of the engine (include/tk_knn.h): error reporting, tree life cycle,
// and the KD query pipeline (query binning + KD kernel launch).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <tuple>
#include <vector>

#include "kd_filter.cuh"
#include "kd_query.cuh"
#include "kd_wide.cuh"
#include "sort.cuh"
#include "tk_internal.h"

namespace tk {

namespace {
thread_local std::string g_err;

struct DeviceGuard {
    int prev = -1;
    bool changed = false;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) == cudaSuccess && prev != dev) {
            changed = cudaSetDevice(dev) == cudaSuccess;
        }
    }
    ~DeviceGuard() {
        if (changed) cudaSetDevice(prev);
    }
};

int sm_count(int dev) {
    static std::mutex mu;
    static std::vector<int> cache;
    std::lock_guard<std::mutex> lock(mu);
    if (dev < 0) dev = 0;
    if ((int)cache.size() <= dev) cache.resize(dev + 1, 0);
    if (cache[dev] == 0) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 1;
        cache[dev] = v;
    }
    return cache[dev];
}

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }
}  // namespace

int fail(int status, const std::string& msg) {
    g_err = msg;
    return status;
}
void clear_error() { g_err.clear(); }

// ------------------------------------------------------------ binning --

// Queries in cell order; with `classes`, each one's cost class (bits 16-23
// of bin_of, see k_bin_count) goes to the same position.
__global__ void k_bin_scatter(int nq, const int* bin_of, const int* pos_of, const int* offsets, int* order,
                              uint32_t* classes) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nq) return;
    const int b = bin_of[i];
    const int dst = offsets[b & 0xFFFF] + pos_of[i];
    order[dst] = i;
    if (classes) classes[dst] = uint32_t(b) >> 16;
}

// ------------------------------------------------------------ planning --

namespace {

int bin_levels(int L, int64_t nq) {
    int lg = 0;
    while ((int64_t(1) << (lg + 1)) <= nq) ++lg;
    return std::max(1, std::min({L, kMaxBinLevels, lg - 4}));
}

// Query workspace: work counter, cell counts, per query its cell, rank,
// place in cell order and cost class, then the scratch of the cell-count
// scan or (used after it) of the cost-class pass.  After the cell scatter
// bin_of and pos_of are free again and receive the class pass's output.
struct WsLayout {
    size_t counter = 0, counts = 0, bin_of = 0, pos_of = 0, order = 0, classes = 0, scan = 0, total = 0;
};

WsLayout ws_layout(int L, int64_t nq) {
    WsLayout w;
    const int B = bin_levels(L, nq);
    size_t o = 0;
    w.counter = o;
    o += 256;
    w.counts = o;
    o += align_up(sizeof(int) * (size_t(1) << B), 256);
    w.bin_of = o;
    o += align_up(sizeof(int) * size_t(nq), 256);
    w.pos_of = o;
    o += align_up(sizeof(int) * size_t(nq), 256);
    w.order = o;
    o += align_up(sizeof(int) * size_t(nq), 256);
    w.classes = o;
    o += align_up(sizeof(uint32_t) * size_t(nq), 256);
    w.scan = o;
    o += std::max(scan_workspace_bytes(int64_t(1) << B), sort_pass8_workspace_bytes(nq));
    w.total = o;
    return w;
}

bool gr_available(int dtype, int dims, int G, int R) {
    const bool full = dtype == TK_F32 && dims == 3;
    if (!full && !(G == 1 || G == 4 || G == 32)) return false;
    if (R < 1 || R > 16 || (R & (R - 1))) return false;
    if (G * R > 128) return false;
    if (G == 16 && R > 8) return false;
    if (G == 32 && R > 4) return false;
    return true;
}

// Points per leaf for one lane per query, see query_levels.  Small clouds get
// 8 to 16, at the depth of the default layout (8 sqrt 2 = 11.31): a level more
// for those just short of a power of two costs 1M queries 10%, in their cells'
// counts (2,000 points, d = 3, k = 4 0.51 -> 0.56 ms).
double one_lane_leaf(int64_t n) { return n <= 65536 ? 11.31 : 22; }

// round(log2(v)), at least 0
int log2_round(double v) { return v <= 1.0 ? 0 : int(std::lround(std::log2(v))); }

// Lanes per query when the caller leaves it to the library: one lane or a
// whole warp (2 to 16 lanes were never the fastest shape; a warp's walk tests
// a path's siblings side by side, see kd_warp.cuh).  One lane's list holds
// k <= 16.  A lane takes far fewer instructions per query but its search is
// one long chain of dependent steps, longer in larger clouds, so calls need
// enough queries to hide it: the crossing was measured, at depths of 22 and
// ~100 points per leaf, near 50,000 queries for 10,000 points, 110,000 for
// 100,000, 200,000 for 1M and 260,000 for 4M (d = 3, k = 5 and 8; ms on one
// lane against a warp: 1M points, 65,536 queries, k=8 0.32 / 0.19; 1,048,576
// queries 0.97 / 2.1; 200,000 points, 131,072 queries, k=4 0.19 / 0.24), lower
// for k = 1, higher for k = 16, and lower in fewer dimensions, where a search
// is shorter (131,072 queries in 200,000 points, k=4: d=2 0.10 / 0.16, d=1
// 0.05 / 0.13).  Small clouds fall slower than the large ones' slope (1,000
// points, d = 3: 20,000 queries, k=4 0.054 / 0.040, k=1 0.043 / 0.036, 40,000
// 0.056 / 0.061 and 0.043 / 0.049; k=16 40,000 0.115 / 0.077, 131,072 0.195 /
// 0.203; 5,000 points, d = 2, k=16 40,000 0.083 / 0.068).  At a depth the
// caller asked for both search the same leaves, and the crossing moves with
// them: small ones leave most of a warp's lanes without a point, large ones are
// a long scan for one lane (a warp's time over one lane's, d = 3, k=16: 100,000
// points in leaves of 12, 130,000 queries 1.44, of 49 0.7; 10,000 in leaves of
// 10, 80,000 queries 1.4; 1M in leaves of 15, k=8, 80,000 0.95, 110,000 1.13);
// more than 192 points always take a warp.  Trees of 4-8 dimensions (1M refs x
// 262k queries N(0,1), depth 12-13): one lane only for k = 1 up to 6 dimensions
// from half a wave of queries on (d=4: 0.40 vs 0.70 ms), a warp otherwise (d=8,
// k=16: 21.4 vs 38.3).
int auto_lanes(const tk_tree* t, int64_t nq, int k) {
    if (k > 16) return 32;
    const double sms = sm_count(t->device);
    if (t->dims > 3) return k == 1 && t->dims <= 6 && double(nq) >= sms * 512 ? 1 : 32;
    if (t->d_filter[0]) {
        // float64: the filtered search takes a warp per query; one lane without
        // the filter wins where a search is short and there are many (ms, one
        // lane / filtered, k=8: d=1 20,000 points, 65,536 queries 0.104 /
        // 0.109, 1M queries 0.42 / 1.63; d=2 200,000 points 65,536 0.39 / 0.19,
        // 1M 1.99 / 2.48, 1M points 4.3 / 2.6; d=3 2,000 points 4.5 / 4.0, k=1
        // 2.7 / 2.9, 200,000 points 7.2 / 4.4; d=2, k=1, 262,144 queries, 1,000
        // points 0.35 / 0.57, 20,000 0.41 / 0.54)
        const double from = t->dims == 1 ? 256 : (t->dims == 2 && t->n <= 50000 ? (t->n <= 5000 ? 700 : 1300) : 2048);
        const bool short_search = t->dims == 1 || (t->dims == 2 ? t->n <= 500000 : t->n <= 5000 && k <= 4);
        return short_search && double(nq) >= sms * from ? 1 : 32;
    }
    const double avg_leaf = double(t->n) / double(int64_t(1) << t->search_levels);
    if (!t->auto_depth && avg_leaf > 192) return 32;
    const double lg = std::log2(double(t->n));
    double crossing = sms * 120.0 * std::max({1.0, lg - 10.3, t->dims > 1 ? 0.3 * lg - 1.05 : 0.0});
    const double by_k = k == 1 ? 0.6 : (k > 8 ? 1.4 : 0.9), by_dims = t->dims == 1 ? 0.4 : (t->dims == 2 ? 0.65 : 1.0);
    crossing *= by_k;
    if (k > 8 && t->dims > 1) crossing = std::max(crossing, sms * 660.0);
    if (!t->auto_depth) {
        if (k == 1) crossing = sms * (165.0 + 28.0 * std::max(0.0, lg - 10.0)) * std::pow(std::max(1.0, avg_leaf / 16), 0.45);
        else crossing *= std::pow(avg_leaf / 32, 0.75);
        if (t->dims == 1) crossing = std::min(crossing, sms * 1000.0);  // by_dims makes it 400
    }
    return double(nq) >= crossing * by_dims ? 1 : 32;
}

int pow2_ceil(int v) {
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

// Blocks of `kfn` that fit an SM.  A property of the code and the launch, asked
// of the driver once per kernel (0.8 us a call).
int blocks_per_sm(const void* kfn, int block, size_t smem) {
    static std::mutex mu;
    static std::map<std::tuple<int, const void*, int, size_t>, int> known;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    int& v = known[std::make_tuple(dev, kfn, block, smem)];
    if (v == 0 && (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kfn, block, smem) != cudaSuccess || v <= 0)) v = 1;
    return v;
}

// Whether a call's queries are ordered by cell and cost class.
// Automatic binning from one wave of queries (SMs x 1024) on: below that each
// thread takes about one query, the cell order gains little leaf sharing, and
// grouping a region's expensive queries into the same warps lengthens the
// slowest warp, which then sets the launch time (131,072 queries: 1.33 ms
// binned vs 1.17 ms in input order; 1,048,576: 3.53 vs 5.84 ms on the
// cube-and-sphere workload).  A warp per query gains by the cost order already
// where a search is long (4-8 dims, or long lists), from ten queries per
// resident warp on: 65,536 queries of 1M points, ms in input order / binned:
// 6 dims k=16 1.93 / 1.78, 8 dims 8.0 / 7.0, 3 dims k=100 0.66 / 0.60; but 3
// dims k=16 0.24 / 0.25, and 10,000 queries lose wherever they are.  So does
// every call on a small cloud, whose searches are alike (80,000 queries, k=50,
// unbinned over binned: 3 dims 1,000 points 0.84, 30,000 0.96, 100,000 1.00,
// 300,000 1.12; 2 dims 100,000 0.93, 300,000 1.03; 6 dims, k=16, 1,000 0.89,
// 10,000 1.00, 100,000 1.02).
bool binned(const tk_tree* t, int L, int G, int64_t nq, int k, const tk_query_opts& o) {
    if (o.bin_queries >= 0) return o.bin_queries == 1;
    const int64_t sms = sm_count(t->device);
    const bool long_search = G == 32 && nq >= sms * 320 &&
                             (t->dims > 3 ? k > 4 && t->n >= 10000
                                          : k > 48 && t->n >= (t->dims == 3 ? int64_t(1) << 16 : int64_t(1) << 18));
    return L >= 2 && (nq >= sms * 1024 || long_search);
}

// Queries that one round of any kernel's grid holds (a warp each, one block
// per SM): no counter, and too few to be binned, so no workspace.
int64_t scratch_free(const tk_tree* t) { return int64_t(sm_count(t->device)) * (kKdBlock / 32); }

// Zero the work counter and, when binning is on, order the queries by the
// tree cell at depth B they fall into (count, exclusive scan, scatter).
// `count(B, counts, bin_of, pos_of)` launches the counting kernel.  With
// `classes` (the counting kernel wrote cost classes), one stable radix pass
// then puts the costliest class first, cell order kept within a class: the
// persistent search takes its work in that order, so the expensive queries
// do not end up in the last chunks (the launch's tail), and a warp's 32
// queries have similar costs (a warp runs as long as its slowest lane).
template <typename CountFn>
int prepare_order(const tk_tree* t, int L, int G, int nq, int k, const tk_query_opts& o, char* ws, cudaStream_t s, int** counter,
                  const int32_t** order, bool classes, CountFn count) {
    const WsLayout w = ws_layout(t->search_levels, nq);
    *order = nullptr;
    const bool bin = binned(t, L, G, nq, k, o);
    cudaError_t e;
    if (bin) {
        const int B = bin_levels(L, nq);
        const int nbins = 1 << B;
        int* counts = reinterpret_cast<int*>(ws + w.counts);
        int* bin_of = reinterpret_cast<int*>(ws + w.bin_of);
        int* pos_of = reinterpret_cast<int*>(ws + w.pos_of);
        int* ord = reinterpret_cast<int*>(ws + w.order);
        e = cudaMemsetAsync(counts, 0, sizeof(int) * nbins, s);
        if (e == cudaSuccess) e = cudaMemsetAsync(*counter, 0, sizeof(int), s);
        if (e != cudaSuccess) return fail(TK_ECUDA, std::string("memset: ") + cudaGetErrorString(e));
        count(B, counts, bin_of, pos_of);
        e = exclusive_scan(counts, nbins, ws + w.scan, s);
        if (e != cudaSuccess) return fail(TK_ECUDA, std::string("bin scan: ") + cudaGetErrorString(e));
        uint32_t* cls = classes ? reinterpret_cast<uint32_t*>(ws + w.classes) : nullptr;
        k_bin_scatter<<<(nq + 255) / 256, 256, 0, s>>>(nq, bin_of, pos_of, counts, ord, cls);
        e = cudaGetLastError();
        if (e != cudaSuccess) return fail(TK_ECUDA, std::string("binning launch: ") + cudaGetErrorString(e));
        *order = ord;
        if (classes) {
            uint32_t* final_order = reinterpret_cast<uint32_t*>(pos_of);
            e = sort_pass8(cls, reinterpret_cast<const uint32_t*>(ord), reinterpret_cast<uint32_t*>(bin_of),
                           final_order, nq, ws + w.scan, w.total - w.scan, s);
            if (e != cudaSuccess) return fail(TK_ECUDA, std::string("cost-class pass: ") + cudaGetErrorString(e));
            *order = reinterpret_cast<const int32_t*>(final_order);
        }
    } else if (*counter) {
        e = cudaMemsetAsync(*counter, 0, sizeof(int), s);
        if (e != cudaSuccess) return fail(TK_ECUDA, std::string("memset: ") + cudaGetErrorString(e));
    }
    return TK_OK;
}

}  // namespace

// Points per leaf a search works best with: one lane follows its own path and
// wants small leaves; a warp scans 32 points at a time and, with a longer
// list, has more to gain from scanning on than from another descent.  Best
// depths measured (k; points per leaf at 10,000 / 100,000 / 1M / 4M points):
// one lane 10 / 24 / 30 / 16 (5,000 points: 10; 100,000 points of 5 and 6 dims
// 12); a warp k=1 39 / 49 / 61 / 64, k=8 156 / 98 / 61 /
// 128, k=16 156 / 98 / 122 / 128, k=100 156 / 195 / 244 / 128; 4-8 dims 61 to
// 122.  float64 without the float filter pays more for a point than for a
// descent.  Of the shapes between, which only callers ask for, two lanes want
// one lane's leaves, four a little more, eight and sixteen 20 to 40 points
// (10,000 points, d = 3, 1M queries, k=1 / 8, 10 and 20 points over 40: 2 lanes
// 0.61, 0.72 / 0.65, 0.76; 4 0.77, 0.81 / 0.85, 0.84; 8 0.92, 0.91 / 1.07, 0.96;
// 16 0.92, 0.94 / 1.09, 0.99).
int query_levels(const tk_tree* t, int lanes, int k) {
    if (!t->auto_depth) return t->search_levels;
    double leaf = one_lane_leaf(t->n);
    if (t->dims > 3) leaf = lanes == 1 ? (t->dims > 4 ? std::min(leaf, 12.0) : leaf) : 90;
    else if (lanes == 32) leaf = t->dtype == TK_F64 && !t->d_filter[0] ? 50 : (k <= 2 ? 50 : (k <= 48 ? 110 : 180));
    else if (lanes >= 8) leaf = k == 1 || (lanes == 8 && k <= 16) ? 25 : 40;
    else if (lanes == 4 && t->dims == 3 && k > 1) leaf *= 1.5;
    else if (lanes > 1) leaf = std::min(leaf, 12.0);
    return std::max(1, std::min(t->search_levels, log2_round(double(t->n) / leaf)));
}

namespace {

template <typename T, int D>
int run_query(const tk_tree* t, const T* q, int nq, int k, T* dists, int32_t* idx, const tk_query_opts& o,
              char* ws, cudaStream_t s) {
    if (o.traversal < 0 || o.traversal > 2) return fail(TK_EINVAL, "traversal must be 0, 1 or 2");
    // warp packets: one lane per query, the warp walks the tree together
    const bool packet = o.traversal == 2 && k <= 16 && t->d_boxes != nullptr;
    // lanes per query and registers per lane
    int G = 1, R = pow2_ceil(k);
    if (!packet) {
        G = o.threads_per_query > 0 ? o.threads_per_query : auto_lanes(t, nq, k);
        if (G != 1 && G != 2 && G != 4 && G != 8 && G != 16 && G != 32)
            return fail(TK_EINVAL, "threads_per_query must be 1, 2, 4, 8, 16 or 32");
        G = std::max(G, pow2_ceil((k + 15) / 16));
        R = pow2_ceil((k + G - 1) / G);
        while (!gr_available(t->dtype, D, G, R) && G < 32) {
            G <<= 1;
            R = pow2_ceil((k + G - 1) / G);
        }
        if (!gr_available(t->dtype, D, G, R)) return fail(TK_EUNSUPPORTED, "no kernel shape for this k");
        if (G == 32 && k == 1) R = 0;  // WarpList<T, 0>
    }

    const int L = packet ? t->search_levels : query_levels(t, G, k);
    // 10 levels (4 KiB for float): deeper staging measured no faster, and at
    // 12 levels (16 KiB) only 3 of the 4 blocks the registers allow stayed
    // resident per SM on the one-lane shape.
    int S = o.smem_levels >= 0 ? o.smem_levels : 10;
    S = std::max(0, std::min({S, L, sizeof(T) == 4 ? 15 : 14}));  // <= 128 KiB of shared memory
    if (!packet && G == 32) S = 0;  // a warp per query reads split values five levels at a time instead
    const int block = kKdBlock;
    const size_t smem = kd_smem_bytes<T>(S);
    const bool filtered = sizeof(T) == 8 && !packet && G == 32 && t->d_filter[0];
    const void* kfn = packet ? kd_packet_kernel<T, D>(R) : (filtered ? kd_filtered_kernel(D, R) : kd_query_kernel<T, D>(G, R));
    if (!kfn) return fail(TK_EUNSUPPORTED, "KD query kernel shape not compiled");
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return fail(TK_ECUDA, std::string("smem attribute: ") + cudaGetErrorString(e));
    }
    int per_sm = blocks_per_sm(kfn, block, smem);
    if (o.blocks_per_sm > 0) per_sm = std::min(per_sm, int(o.blocks_per_sm));
    const int groups_per_block = block / G;
    const int need = (nq + groups_per_block - 1) / groups_per_block;
    const int sms = sm_count(t->device);
    int grid = std::max(1, std::min(need, per_sm * sms));
    // A few blocks left over after as many on every SM would have the last word
    // with long lists on one lane; the counter (grid < need) deals out what they
    // would do (2 dims, 10,000 points, k=16, 80,000 queries, 313 blocks -> 304:
    // 0.119 -> 0.108 ms).
    if (grid == need && G == 1 && k > 8 && grid > sms && grid % sms <= sms / 8) grid -= grid % sms;

    // a grid that holds all queries at once needs no counter
    int* counter = grid < need || binned(t, L, G, nq, k, o) ? reinterpret_cast<int*>(ws + ws_layout(t->search_levels, nq).counter) : nullptr;
    const int32_t* order = nullptr;
    const PointRec<T>* boxes = static_cast<const PointRec<T>*>(t->d_boxes);
    int rc0 = prepare_order(t, L, G, nq, k, o, ws, s, &counter, &order, true, [&](int B, int* counts, int* bin_of, int* pos_of) {
        bin_count_launch<T, D>(q, nq, static_cast<const T*>(t->d_medians), B, L, boxes, counts, bin_of, pos_of, s);
    });
    if (rc0 != TK_OK) return rc0;

    KdArgs<T> a;
    a.pts = static_cast<const PointRec<T>*>(t->d_pts);
    a.medians = static_cast<const T*>(t->d_medians);
    a.leaf_off = t->d_leaf_off;
    a.boxes = static_cast<const PointRec<T>*>(t->d_boxes);  // the 1-3-D searches always prune with node boxes
    a.levels = L;
    a.smem_levels = S;
    a.q = q;
    a.nq = nq;
    a.k = k;
    a.order = order;
    a.out_d = dists;
    a.out_i = idx;
    a.work = counter;
    a.nan_empty = t->nan_empty;
    KdLaunch l{G, R, block, grid, smem};
    if (o.kernel_start_event) cudaEventRecord(static_cast<cudaEvent_t>(o.kernel_start_event), s);
    int rc;
    if constexpr (sizeof(T) == 8) {
        if (filtered) {
            FilterArgs f;
            f.f.pts = static_cast<const PointRec<float>*>(t->d_filter[0]);
            f.f.boxes = static_cast<const PointRec<float>*>(t->d_filter[1]);
            f.f.medians = static_cast<const float*>(t->d_filter[2]);
            f.f.frame = static_cast<const Frame*>(t->d_filter[3]);
            f.pts = a.pts;
            f.levels = L;
            f.q = q;
            f.nq = nq;
            f.k = k;
            f.order = order;
            f.out_d = dists;
            f.out_i = idx;
            f.work = counter;
            rc = kd_filtered_launch(f, D, R, grid, s);
        } else {
            rc = packet ? kd_packet_launch<T, D>(a, l, s) : kd_query_launch<T, D>(a, l, s);
        }
    } else {
        rc = packet ? kd_packet_launch<T, D>(a, l, s) : kd_query_launch<T, D>(a, l, s);
    }
    if (rc == TK_OK && o.kernel_stop_event) cudaEventRecord(static_cast<cudaEvent_t>(o.kernel_stop_event), s);
    return rc;
}

// KD query of a tree of 4-8 dimensions (kd_wide.cuh): one lane per query
// for k <= 16 when the automatic / requested shape is one lane, else a
// 32-lane group per query; binning and options as run_query (warp packets do
// not apply: traversal 2 runs as 1).
template <typename T>
int run_query_wide(const tk_tree* t, const T* q, int nq, int k, T* dists, int32_t* idx, const tk_query_opts& o,
                   char* ws, cudaStream_t s) {
    if (o.traversal < 0 || o.traversal > 2) return fail(TK_EINVAL, "traversal must be 0, 1 or 2");
    int G = o.threads_per_query > 0 ? o.threads_per_query : auto_lanes(t, nq, k);
    if (G != 1 && G != 2 && G != 4 && G != 8 && G != 16 && G != 32)
        return fail(TK_EINVAL, "threads_per_query must be 1, 2, 4, 8, 16 or 32");
    if (G != 1 || k > 16) G = 32;  // kernels of wide trees: 1 (k <= 16) or 32 lanes per query
    const int R = G == 32 && k == 1 ? 0 : pow2_ceil((k + G - 1) / G);  // 0: WarpList<T, 0>
    const int W = record_width(t->dims);
    const int L = query_levels(t, G, k);
    int S = o.smem_levels >= 0 ? o.smem_levels : 10;
    S = std::max(0, std::min({S, L, sizeof(T) == 4 ? 15 : 14}));
    if (G == 32) S = 0;  // a warp per query reads split values five levels at a time instead
    const int block = kKdBlock;
    const size_t smem = kd_smem_bytes<T>(S);
    const void* kfn = kd_wide_kernel<T>(W, G, R);
    if (!kfn) return fail(TK_EUNSUPPORTED, "KD query kernel shape not compiled");
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
        if (e != cudaSuccess) return fail(TK_ECUDA, std::string("smem attribute: ") + cudaGetErrorString(e));
    }
    int per_sm = blocks_per_sm(kfn, block, smem);
    if (o.blocks_per_sm > 0) per_sm = std::min(per_sm, int(o.blocks_per_sm));
    const int groups_per_block = block / G;
    const int need = (nq + groups_per_block - 1) / groups_per_block;
    const int grid = std::max(1, std::min(need, per_sm * sm_count(t->device)));

    // One lane a query, more than a block an SM: uneven loads, which the counter
    // levels (300,000 points of 6 dims, k=1, 80,000 queries 1.44 -> 1.31 ms).
    const bool level = G == 1 && need > sm_count(t->device);
    int* counter = grid < need || level || binned(t, L, G, nq, k, o) ? reinterpret_cast<int*>(ws + ws_layout(t->search_levels, nq).counter) : nullptr;
    const int32_t* order = nullptr;
    const int rc0 = prepare_order(t, L, G, nq, k, o, ws, s, &counter, &order, true, [&](int B, int* counts, int* bin_of, int* pos_of) {
        bin_count_wide_launch<T>(q, nq, t->dims, static_cast<const T*>(t->d_medians), B, L,
                                 static_cast<const T*>(t->d_boxes), W, counts, bin_of, pos_of, s);
    });
    if (rc0 != TK_OK) return rc0;

    KdWideArgs<T> a;
    a.pts = static_cast<const T*>(t->d_pts);
    a.perm = t->d_perm;
    a.medians = static_cast<const T*>(t->d_medians);
    a.leaf_off = t->d_leaf_off;
    // a warp per query prunes with node boxes always: one round trip tests all of a path's siblings
    a.boxes = o.prune_boxes == 0 && G == 1 ? nullptr : static_cast<const T*>(t->d_boxes);
    a.levels = L;
    a.leaf_shift = t->search_levels - L;
    a.smem_levels = S;
    a.dims = t->dims;
    a.q = q;
    a.nq = nq;
    a.k = k;
    a.order = order;
    a.out_d = dists;
    a.out_i = idx;
    a.work = counter;
    if (o.kernel_start_event) cudaEventRecord(static_cast<cudaEvent_t>(o.kernel_start_event), s);
    const int rc = kd_wide_launch<T>(a, W, G, R, grid, block, smem, s);
    if (rc == TK_OK && o.kernel_stop_event) cudaEventRecord(static_cast<cudaEvent_t>(o.kernel_stop_event), s);
    return rc;
}

int run_query_any(const tk_tree* t, const void* q, int n32, int k, void* dists, int32_t* idx, const tk_query_opts& o,
                  char* ws, cudaStream_t s) {
    if (t->dtype == TK_F32) {
        auto* qq = static_cast<const float*>(q);
        auto* dd = static_cast<float*>(dists);
        switch (t->dims) {
            case 1: return run_query<float, 1>(t, qq, n32, k, dd, idx, o, ws, s);
            case 2: return run_query<float, 2>(t, qq, n32, k, dd, idx, o, ws, s);
            case 3: return run_query<float, 3>(t, qq, n32, k, dd, idx, o, ws, s);
            default: return run_query_wide<float>(t, qq, n32, k, dd, idx, o, ws, s);
        }
    } else {
        auto* qq = static_cast<const double*>(q);
        auto* dd = static_cast<double*>(dists);
        switch (t->dims) {
            case 1: return run_query<double, 1>(t, qq, n32, k, dd, idx, o, ws, s);
            case 2: return run_query<double, 2>(t, qq, n32, k, dd, idx, o, ws, s);
            case 3: return run_query<double, 3>(t, qq, n32, k, dd, idx, o, ws, s);
            default: return run_query_wide<double>(t, qq, n32, k, dd, idx, o, ws, s);
        }
    }
}

// The 4th slot of a point record holds an index as raw bits: the original
// index of a point, or the begin / end offset of a leaf in its box records.
template <typename T>
void set_rec_index(PointRec<T>& r, uint32_t v) {
    if (sizeof(T) == 4) {
        std::memcpy(&r.w, &v, 4);
    } else {
        const uint64_t bits = v;
        std::memcpy(&r.w, &bits, 8);
    }
}

// Device image of a tree of 4-8 dimensions: zero-padded coordinate rows of
// record_width(dims), the original indices, and node boxes as lo / hi rows.
template <typename T>
int upload_wide(tk_tree* t, const HostTree<T>& h) {
    const int64_t n = h.n;
    const int W = record_width(h.dims);
    std::vector<T> rows(static_cast<size_t>(n) * W, T(0));
    for (int64_t i = 0; i < n; ++i)
        for (int d = 0; d < h.dims; ++d) rows[size_t(i) * W + d] = h.structured[i * h.dims + d];
    const size_t nnodes = h.box_lo.size() / W;
    std::vector<T> boxes(2 * nnodes * W);
    for (size_t i = 0; i < nnodes; ++i)
        for (int c = 0; c < W; ++c) {
            boxes[(2 * i) * W + c] = h.box_lo[i * W + c];
            boxes[(2 * i + 1) * W + c] = h.box_hi[i * W + c];
        }
    const size_t b_pts = sizeof(T) * rows.size();
    const size_t b_perm = sizeof(int32_t) * size_t(n);
    const size_t b_med = sizeof(T) * h.medians.size();
    const size_t b_off = sizeof(int32_t) * h.leaf_off.size();
    const size_t b_box = sizeof(T) * boxes.size();
    cudaError_t e = cudaMalloc(&t->d_pts, b_pts);
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&t->d_perm), b_perm);
    if (e == cudaSuccess) e = cudaMalloc(&t->d_medians, std::max<size_t>(b_med, sizeof(T)));
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&t->d_leaf_off), b_off);
    if (e == cudaSuccess) e = cudaMalloc(&t->d_boxes, b_box);
    if (e != cudaSuccess) return fail(TK_ENOMEM, std::string("device allocation: ") + cudaGetErrorString(e));
    e = cudaMemcpy(t->d_pts, rows.data(), b_pts, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(t->d_perm, h.perm.data(), b_perm, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && b_med) e = cudaMemcpy(t->d_medians, h.medians.data(), b_med, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(t->d_leaf_off, h.leaf_off.data(), b_off, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(t->d_boxes, boxes.data(), b_box, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return fail(TK_ECUDA, std::string("tree upload: ") + cudaGetErrorString(e));
    t->device_bytes = int64_t(b_pts + b_perm + b_med + b_off + b_box);
    return TK_OK;
}

template <typename T>
int upload_tree(tk_tree* t, const HostTree<T>& h) {
    if (h.dims > 3) return upload_wide(t, h);
    const int64_t n = h.n;
    std::vector<PointRec<T>> recs(static_cast<size_t>(n));
    for (int64_t i = 0; i < n; ++i) {
        T c[3] = {T(0), T(0), T(0)};
        for (int d = 0; d < h.dims; ++d) c[d] = h.structured[i * h.dims + d];
        recs[i].x = c[0];
        recs[i].y = c[1];
        recs[i].z = c[2];
        set_rec_index(recs[i], uint32_t(h.perm[i]));
    }
    const size_t b_pts = sizeof(PointRec<T>) * size_t(n);
    const size_t b_med = sizeof(T) * h.medians.size();
    const size_t b_off = sizeof(int32_t) * h.leaf_off.size();
    const size_t nnodes = h.box_lo.size() / 3;
    std::vector<PointRec<T>> boxes(2 * nnodes);
    const size_t first_leaf = nnodes / 2;  // nnodes = 2^(L+1) - 1
    for (size_t i = 0; i < nnodes; ++i) {
        boxes[2 * i] = PointRec<T>{h.box_lo[3 * i], h.box_lo[3 * i + 1], h.box_lo[3 * i + 2], T(0)};
        boxes[2 * i + 1] = PointRec<T>{h.box_hi[3 * i], h.box_hi[3 * i + 1], h.box_hi[3 * i + 2], T(0)};
        if (i >= first_leaf) {  // a leaf's box also carries its point range [begin, end)
            set_rec_index(boxes[2 * i], uint32_t(h.leaf_off[i - first_leaf]));
            set_rec_index(boxes[2 * i + 1], uint32_t(h.leaf_off[i - first_leaf + 1]));
        }
    }
    const size_t b_box = sizeof(PointRec<T>) * boxes.size();
    cudaError_t e = cudaMalloc(&t->d_pts, b_pts);
    if (e == cudaSuccess) e = cudaMalloc(&t->d_medians, std::max<size_t>(b_med, sizeof(T)));
    if (e == cudaSuccess) e = cudaMalloc(reinterpret_cast<void**>(&t->d_leaf_off), b_off);
    if (e == cudaSuccess) e = cudaMalloc(&t->d_boxes, b_box);
    if (e != cudaSuccess) return fail(TK_ENOMEM, std::string("device allocation: ") + cudaGetErrorString(e));
    e = cudaMemcpy(t->d_pts, recs.data(), b_pts, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && b_med) e = cudaMemcpy(t->d_medians, h.medians.data(), b_med, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(t->d_leaf_off, h.leaf_off.data(), b_off, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(t->d_boxes, boxes.data(), b_box, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return fail(TK_ECUDA, std::string("tree upload: ") + cudaGetErrorString(e));
    t->device_bytes = int64_t(b_pts + b_med + b_off + b_box);
    return TK_OK;
}

void free_tree_device(tk_tree* t) {
    if (t->one_image) {
        if (t->own_image && t->d_pts) cudaFree(t->d_pts);
    } else {
        if (t->d_pts) cudaFree(t->d_pts);
        if (t->d_perm) cudaFree(t->d_perm);
        if (t->d_medians) cudaFree(t->d_medians);
        if (t->d_leaf_off) cudaFree(t->d_leaf_off);
        if (t->d_boxes) cudaFree(t->d_boxes);
    }
    t->d_perm = nullptr;
    t->d_pts = t->d_medians = t->d_boxes = nullptr;
    t->d_leaf_off = nullptr;
}

// Points (T[n*dims]) and / or permutation (int32[n]) of a GPU-built tree in
// the order of its device image.
template <typename T>
int image_layout(const tk_tree* t, T* points, int32_t* perm) {
    DeviceGuard g(t->device);
    if (t->dims > 3) {  // coordinate rows + separate indices
        const int W = record_width(t->dims);
        cudaError_t e = cudaSuccess;
        if (points) {
            std::vector<T> rows(static_cast<size_t>(t->n) * W);
            e = cudaMemcpy(rows.data(), t->d_pts, sizeof(T) * rows.size(), cudaMemcpyDeviceToHost);
            if (e == cudaSuccess)
                for (int64_t i = 0; i < t->n; ++i)
                    for (int d = 0; d < t->dims; ++d) points[i * t->dims + d] = rows[size_t(i) * W + d];
        }
        if (e == cudaSuccess && perm)
            e = cudaMemcpy(perm, t->d_perm, sizeof(int32_t) * size_t(t->n), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) return fail(TK_ECUDA, std::string("layout copy: ") + cudaGetErrorString(e));
        return TK_OK;
    }
    std::vector<PointRec<T>> recs(static_cast<size_t>(t->n));
    const cudaError_t e = cudaMemcpy(recs.data(), t->d_pts, sizeof(PointRec<T>) * recs.size(), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return fail(TK_ECUDA, std::string("layout copy: ") + cudaGetErrorString(e));
    for (int64_t i = 0; i < t->n; ++i) {
        const PointRec<T>& r = recs[size_t(i)];
        if (points) {
            const T c[3] = {r.x, r.y, r.z};
            for (int d = 0; d < t->dims; ++d) points[i * t->dims + d] = c[d];
        }
        if (perm) {
            if (sizeof(T) == 4) {
                uint32_t bits;
                std::memcpy(&bits, &r.w, 4);
                perm[i] = int32_t(bits);
            } else {
                uint64_t bits;
                std::memcpy(&bits, &r.w, 8);
                perm[i] = int32_t(bits);
            }
        }
    }
    return TK_OK;
}

// Runs work(first, last) over [0, count) in pieces, on up to 16 host threads
// (on this one where none can be had).
template <typename F>
void in_threads(size_t count, size_t piece, F work) {
    std::atomic<size_t> next{0};
    auto run = [&] {
        for (size_t i; (i = next.fetch_add(piece)) < count;) work(i, std::min(count, i + piece));
    };
    const size_t want = std::min({size_t(16), size_t(std::max(1u, std::thread::hardware_concurrency())), (count + piece - 1) / piece});
    std::vector<std::thread> pool;
    pool.reserve(want);
    try {
        while (pool.size() + 1 < want) pool.emplace_back(run);
    } catch (...) {  // no more threads than there are
    }
    run();
    for (std::thread& t : pool) t.join();
}

// The same in the layout's order (depth `levels`).  A deeper image holds the
// same points in each range of a leaf of that depth, ordered along the axes
// of its own leaf parents: order each range along the layout's.  On the host,
// in threads (points and permutation of 1M / 4M points: 65 / 325 ms on one
// thread that compared through indices, 5.1 / 23 now; 4.9 / 24 where the image
// has the layout's order and nothing is sorted).
template <typename T>
int ordered_layout(const tk_tree* t, T* points, int32_t* perm) {
    const size_t n = size_t(t->n), dims = size_t(t->dims), ax = size_t(t->levels - 1) % dims;
    const bool wide = dims > 3;
    const size_t row = wide ? size_t(record_width(t->dims)) : 4;  // coordinates from one point to the next
    std::unique_ptr<T[]> rows(new T[n * row]);
    std::unique_ptr<int32_t[]> ids(wide ? new int32_t[n] : nullptr);
    std::vector<int32_t> offs((size_t(1) << t->search_levels) + 1);
    {
        DeviceGuard g(t->device);
        cudaError_t e = cudaMemcpy(rows.get(), t->d_pts, sizeof(T) * n * row, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess && wide) e = cudaMemcpy(ids.get(), t->d_perm, sizeof(int32_t) * n, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess) e = cudaMemcpy(offs.data(), t->d_leaf_off, sizeof(int32_t) * offs.size(), cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) return fail(TK_ECUDA, std::string("layout copy: ") + cudaGetErrorString(e));
    }
    struct Entry {
        T x;
        int32_t id, at;
    };
    const size_t leaves = size_t(1) << t->levels;
    const int shift = t->search_levels - t->levels;
    size_t most = 0;
    for (size_t l = 0; l < leaves; ++l) most = std::max(most, size_t(offs[(l + 1) << shift] - offs[l << shift]));
    std::atomic<bool> short_of_memory{false};
    in_threads(leaves, std::max<size_t>(1, leaves / 256), [&](size_t first, size_t last) {
        std::unique_ptr<Entry[]> v(new (std::nothrow) Entry[std::max<size_t>(1, most)]);
        if (!v) {
            short_of_memory = true;
            return;
        }
        for (size_t l = first; l < last; ++l) {
            const int32_t beg = offs[l << shift], end = offs[(l + 1) << shift];
            for (int32_t i = beg; i < end; ++i) {
                int32_t id;
                if (wide) id = ids[i];
                else std::memcpy(&id, &rows[size_t(i) * row + 3], sizeof id);  // raw bits, the low word of a double
                v[i - beg] = Entry{rows[size_t(i) * row + ax], id, i};
            }
            std::sort(v.get(), v.get() + (end - beg), [](const Entry& a, const Entry& b) {
                return a.x < b.x || (!(b.x < a.x) && a.id < b.id);
            });
            for (int32_t i = beg; i < end; ++i) {
                const Entry& e = v[i - beg];
                if (points) std::memcpy(points + size_t(i) * dims, &rows[size_t(e.at) * row], sizeof(T) * dims);
                if (perm) perm[i] = e.id;
            }
        }
    });
    if (short_of_memory) return fail(TK_ENOMEM, "host allocation failed");
    return TK_OK;
}

template <typename T>
int device_layout(const tk_tree* t, T* points, int32_t* perm) {
    if (t->search_levels == t->levels) return image_layout<T>(t, points, perm);
    try {
        return ordered_layout<T>(t, points, perm);
    } catch (const std::bad_alloc&) {
        return fail(TK_ENOMEM, "host allocation failed");
    }
}

// Argument checks of the GPU builds.
int check_device_build(const void* dev_points, int64_t n, int dims, int dtype, int levels, int device) {
    if (dtype != TK_F32 && dtype != TK_F64) return fail(TK_EINVAL, "dtype must be TK_F32 or TK_F64");
    if (!dev_points) return fail(TK_EINVAL, "points pointer is null");
    if (dims < 1 || dims > kMaxDims)
        return fail(TK_EINVAL, "KD-tree supports dims 1 to " + std::to_string(kMaxDims) + " (got " +
                                   std::to_string(dims) + ")");
    if (n < 1) return fail(TK_EINVAL, "the reference point cloud is empty");
    if (n >= (int64_t(1) << 31)) return fail(TK_EINVAL, "only 32 bit signed indexing implemented (n < 2^31)");
    if (levels < 1 || levels > kMaxLevels)
        return fail(TK_EINVAL, "levels must be in [1, " + std::to_string(kMaxLevels) + "]");
    // node sizes at depth t are floor / ceil of n / 2^t: a leaf parent gets no
    // point exactly when n < 2^(levels-1)
    if (n < (int64_t(1) << (levels - 1)))
        return fail(TK_EINVAL,
                    "Ran out of points while building KD-Tree. Either you required too many levels, "
                    "or you used a lot of coplanar points");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        cudaGetLastError();
        return fail(TK_EINVAL, "CUDA device " + std::to_string(device) + " is not available");
    }
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, dev_points) != cudaSuccess ||
        (attr.type != cudaMemoryTypeDevice && attr.type != cudaMemoryTypeManaged) || attr.device != device) {
        cudaGetLastError();
        return fail(TK_EINVAL, "points must be device memory on CUDA device " + std::to_string(device));
    }
    return TK_OK;
}

// The parts of a tree's image (tree_image) at `image`.
void set_image(tk_tree* t, void* image) {
    const TreeImage im = tree_image(t->n, t->dims, t->dtype, t->search_levels);
    char* p = static_cast<char*>(image);
    t->d_pts = p + im.pts;
    t->d_boxes = p + im.boxes;
    t->d_medians = p + im.medians;
    t->d_leaf_off = reinterpret_cast<int32_t*>(p + im.leaf_off);
    if (t->dims > 3) t->d_perm = reinterpret_cast<int32_t*>(p + im.perm);
    if (im.f_pts) {
        t->d_filter[0] = p + im.f_pts;
        t->d_filter[1] = p + im.f_boxes;
        t->d_filter[2] = p + im.f_medians;
        t->d_filter[3] = p + im.f_frame;
    }
    t->device_bytes = int64_t(im.total);
}

// GPU build of checked arguments into `image` (not owned by the tree).
int device_build(const void* dev_points, int64_t n, int dims, int dtype, int levels, int search_levels, int device,
                 void* image, void* workspace, void* stream, tk_tree** out) {
    tk_tree* t = new (std::nothrow) tk_tree();
    if (!t) return fail(TK_ENOMEM, "host allocation failed");
    t->dtype = dtype;
    t->dims = dims;
    t->levels = levels;
    t->search_levels = search_levels;
    t->device = device;
    t->n = n;
    t->host_layout = false;
    t->one_image = true;
    t->own_image = false;
    set_image(t, image);
    const int rc = dtype == TK_F32
                       ? build_device_tree<float>(static_cast<const float*>(dev_points), n, dims, stream, t, workspace)
                       : build_device_tree<double>(static_cast<const double*>(dev_points), n, dims, stream, t, workspace);
    if (rc != TK_OK) {
        cudaStreamSynchronize(static_cast<cudaStream_t>(stream));  // nothing of it still writes the buffers
        delete t;
        return rc;
    }
    *out = t;
    return TK_OK;
}

}  // namespace
}  // namespace tk

using namespace tk;

extern "C" {

const char* tk_last_error(void) { return g_err.c_str(); }

int tk_version(void) { return 1; }

int tk_cuda_available(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n > 0 ? 1 : 0;
}

int tk_tree_create(const void* host_points, int64_t n, int dims, int dtype, int levels, int device,
                   int n_threads, tk_tree** out) {
    clear_error();
    if (!out) return fail(TK_EINVAL, "out is null");
    *out = nullptr;
    if (dtype != TK_F32 && dtype != TK_F64) return fail(TK_EINVAL, "dtype must be TK_F32 or TK_F64");
    tk_tree* t = new (std::nothrow) tk_tree();
    if (!t) return fail(TK_ENOMEM, "host allocation failed");
    t->dtype = dtype;
    t->dims = dims;
    t->levels = t->search_levels = levels;
    t->device = device;
    t->n = n;
    int rc = dtype == TK_F32
                 ? build_host_tree<float>(static_cast<const float*>(host_points), n, dims, levels, n_threads, t->h32)
                 : build_host_tree<double>(static_cast<const double*>(host_points), n, dims, levels, n_threads,
                                           t->h64);
    if (rc != TK_OK) {
        delete t;
        return rc;
    }
    if (device < 0) {  // host-only tree: layout getters work, queries are refused
        *out = t;
        return TK_OK;
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device >= ndev) {
        cudaGetLastError();
        delete t;
        return fail(TK_EINVAL, "CUDA device " + std::to_string(device) + " is not available");
    }
    {
        DeviceGuard g(device);
        rc = dtype == TK_F32 ? upload_tree<float>(t, t->h32) : upload_tree<double>(t, t->h64);
    }
    if (rc != TK_OK) {
        DeviceGuard g(device);
        free_tree_device(t);
        delete t;
        return rc;
    }
    *out = t;
    return TK_OK;
}

int tk_tree_create_from_layout(const void* structured_points, const int32_t* perm, const void* medians,
                               const int32_t* leaf_offsets, int64_t n, int dims, int dtype, int levels, int device,
                               tk_tree** out) {
    clear_error();
    if (!out) return fail(TK_EINVAL, "out is null");
    *out = nullptr;
    if (dtype != TK_F32 && dtype != TK_F64) return fail(TK_EINVAL, "dtype must be TK_F32 or TK_F64");
    tk_tree* t = new (std::nothrow) tk_tree();
    if (!t) return fail(TK_ENOMEM, "host allocation failed");
    t->dtype = dtype;
    t->dims = dims;
    t->levels = t->search_levels = levels;
    t->device = device;
    t->n = n;
    int rc = dtype == TK_F32
                 ? tree_from_layout<float>(static_cast<const float*>(structured_points), perm,
                                           static_cast<const float*>(medians), leaf_offsets, n, dims, levels, t->h32)
                 : tree_from_layout<double>(static_cast<const double*>(structured_points), perm,
                                            static_cast<const double*>(medians), leaf_offsets, n, dims, levels, t->h64);
    if (rc == TK_OK && device >= 0) {
        int ndev = 0;
        if (cudaGetDeviceCount(&ndev) != cudaSuccess || device >= ndev) {
            cudaGetLastError();
            rc = fail(TK_EINVAL, "CUDA device " + std::to_string(device) + " is not available");
        } else {
            DeviceGuard g(device);
            rc = dtype == TK_F32 ? upload_tree<float>(t, t->h32) : upload_tree<double>(t, t->h64);
            if (rc != TK_OK) free_tree_device(t);
        }
    }
    if (rc != TK_OK) {
        delete t;
        return rc;
    }
    *out = t;
    return TK_OK;
}

int tk_tree_create_device(const void* dev_points, int64_t n, int dims, int dtype, int levels, int device,
                          void* stream, tk_tree** out) {
    clear_error();
    if (!out) return fail(TK_EINVAL, "out is null");
    *out = nullptr;
    int rc = check_device_build(dev_points, n, dims, dtype, levels, device);
    if (rc != TK_OK) return rc;
    DeviceGuard g(device);
    void* image = nullptr;
    void* ws = nullptr;
    const size_t image_bytes = tree_image(n, dims, dtype, levels).total, ws_bytes = build_workspace_bytes(n, dims, dtype);
    cudaError_t e = cudaMalloc(&image, image_bytes);
    if (e == cudaSuccess) e = cudaMalloc(&ws, ws_bytes);
    if (e != cudaSuccess) {
        if (image) cudaFree(image);
        return fail(TK_ENOMEM, std::string("device allocation: ") + cudaGetErrorString(e));
    }
    rc = device_build(dev_points, n, dims, dtype, levels, levels, device, image, ws, stream, out);
    if (rc == TK_OK) (*out)->own_image = true;
    else cudaFree(image);
    cudaFree(ws);
    return rc;
}

size_t tk_tree_image_size(int64_t n, int dims, int dtype, int search_levels) {
    if (n < 1 || dims < 1 || dims > kMaxDims || search_levels < 1 || search_levels > kMaxLevels) return 0;
    return tree_image(n, dims, dtype, search_levels).total;
}

int tk_tree_search_levels(int64_t n, int dims, int dtype, int levels) {
    (void)dtype;
    // the deepest that query_levels asks for
    const int deep = log2_round(double(std::max<int64_t>(n, 1)) / (dims > 3 ? 90.0 : one_lane_leaf(n)));
    return std::min(kMaxLevels, std::max(levels, deep));
}

size_t tk_tree_build_workspace_size(int64_t n, int dims, int dtype) {
    if (n < 1 || dims < 1 || dims > kMaxDims) return 0;
    return build_workspace_bytes(n, dims, dtype);
}

int tk_tree_build_device(const void* dev_points, int64_t n, int dims, int dtype, int levels, int search_levels,
                         int device, void* image, size_t image_bytes, void* workspace, size_t workspace_bytes,
                         void* stream, tk_tree** out) {
    clear_error();
    if (!out) return fail(TK_EINVAL, "out is null");
    *out = nullptr;
    int rc = check_device_build(dev_points, n, dims, dtype, levels, device);
    if (rc != TK_OK) return rc;
    const bool auto_depth = search_levels == 0;
    if (auto_depth) search_levels = tk_tree_search_levels(n, dims, dtype, levels);
    if (search_levels < levels || search_levels > kMaxLevels || n < (int64_t(1) << (search_levels - 1)))
        return fail(TK_EINVAL, "search_levels must be at least levels, and leave a point for every leaf parent");
    if (!image || image_bytes < tree_image(n, dims, dtype, search_levels).total)
        return fail(TK_EWORKSPACE, "tree image buffer too small");
    if (!workspace || workspace_bytes < build_workspace_bytes(n, dims, dtype))
        return fail(TK_EWORKSPACE, "workspace too small");
    if (ws_misaligned(workspace) || ws_misaligned(image))
        return fail(TK_EINVAL, "image and workspace must be 256-byte aligned");
    DeviceGuard g(device);
    rc = device_build(dev_points, n, dims, dtype, levels, search_levels, device, image, workspace, stream, out);
    if (rc == TK_OK) (*out)->auto_depth = auto_depth;
    return rc;
}

int tk_tree_destroy(tk_tree* t) {
    clear_error();
    if (!t) return TK_OK;
    if (t->device >= 0) {
        DeviceGuard g(t->device);
        free_tree_device(t);
        tk::free_host_pipe(t->pipe);
        t->pipe = nullptr;
    }
    delete t;
    return TK_OK;
}

int tk_tree_get_info(const tk_tree* t, tk_tree_info* out) {
    if (!t || !out) return fail(TK_EINVAL, "null argument");
    out->n_points = t->n;
    out->dims = t->dims;
    out->dtype = t->dtype;
    out->levels = t->levels;
    out->device = t->device;
    out->n_leaves = int64_t(1) << t->levels;
    out->device_bytes = t->device_bytes;
    return TK_OK;
}

int tk_tree_get_perm(const tk_tree* t, int32_t* out) {
    if (!t || !out) return fail(TK_EINVAL, "null argument");
    if (!t->host_layout)
        return t->dtype == TK_F32 ? device_layout<float>(t, nullptr, out) : device_layout<double>(t, nullptr, out);
    const auto& p = t->dtype == TK_F32 ? t->h32.perm : t->h64.perm;
    std::memcpy(out, p.data(), sizeof(int32_t) * p.size());
    return TK_OK;
}

int tk_tree_get_points(const tk_tree* t, void* out) {
    if (!t || !out) return fail(TK_EINVAL, "null argument");
    if (!t->host_layout)
        return t->dtype == TK_F32 ? device_layout<float>(t, static_cast<float*>(out), nullptr)
                                  : device_layout<double>(t, static_cast<double*>(out), nullptr);
    if (t->dtype == TK_F32)
        std::memcpy(out, t->h32.structured.data(), sizeof(float) * t->h32.structured.size());
    else
        std::memcpy(out, t->h64.structured.data(), sizeof(double) * t->h64.structured.size());
    return TK_OK;
}

int tk_tree_get_splits(const tk_tree* t, void* medians, int32_t* leaf_offsets) {
    if (!t) return fail(TK_EINVAL, "null argument");
    if (!t->host_layout) {
        DeviceGuard g(t->device);
        const size_t nparts = (size_t(1) << t->levels) - 1;
        cudaError_t e = cudaSuccess;
        if (medians)
            e = cudaMemcpy(medians, t->d_medians, (t->dtype == TK_F32 ? 4 : 8) * nparts, cudaMemcpyDeviceToHost);
        if (e == cudaSuccess && leaf_offsets)  // every 2^(search_levels - levels)-th offset of the image
            e = cudaMemcpy2D(leaf_offsets, sizeof(int32_t), t->d_leaf_off,
                             sizeof(int32_t) << (t->search_levels - t->levels), sizeof(int32_t), nparts + 2,
                             cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) return fail(TK_ECUDA, std::string("split copy: ") + cudaGetErrorString(e));
        return TK_OK;
    }
    if (medians) {
        if (t->dtype == TK_F32)
            std::memcpy(medians, t->h32.medians.data(), sizeof(float) * t->h32.medians.size());
        else
            std::memcpy(medians, t->h64.medians.data(), sizeof(double) * t->h64.medians.size());
    }
    if (leaf_offsets) {
        const auto& o = t->dtype == TK_F32 ? t->h32.leaf_off : t->h64.leaf_off;
        std::memcpy(leaf_offsets, o.data(), sizeof(int32_t) * o.size());
    }
    return TK_OK;
}

int64_t tk_tree_query_scratch_free(const tk_tree* t) { return t && t->device >= 0 ? scratch_free(t) : 0; }

size_t tk_tree_query_workspace_size(const tk_tree* t, int64_t nq) {
    if (!t || nq < 0) return 0;
    return ws_layout(t->search_levels, std::max<int64_t>(nq, 1)).total;
}

int tk_tree_query(const tk_tree* t, const void* q, int64_t nq, int k, void* dists, int32_t* idx,
                  const tk_query_opts* opts, void* workspace, size_t workspace_bytes, void* stream) {
    clear_error();
    if (!t) return fail(TK_EINVAL, "tree is null");
    if (nq < 0 || nq >= (int64_t(1) << 31)) return fail(TK_EINVAL, "number of queries must be in [0, 2^31)");
    if (k < 1) return fail(TK_EINVAL, "k must be >= 1");
    if (k > t->n) return fail(TK_EINVAL, "You requested more nearest neighbors than there are in the KD-Tree");
    if (k > kMaxK) return fail(TK_EINVAL, "k is limited to 128 on the GPU");
    if (t->device < 0 || !t->d_pts) return fail(TK_EINVAL, "tree was built host-only (device < 0); it has no device image");
    if (nq == 0) return TK_OK;
    if (!q || !dists || !idx) return fail(TK_EINVAL, "null query or output pointer");
    tk_query_opts o{0, -1, -1, 0, 0, nullptr, nullptr, -1, 0};
    if (opts) o = *opts;
    const bool free_of_scratch = !workspace && o.bin_queries <= 0 && o.blocks_per_sm <= 0 && nq <= scratch_free(t);
    const size_t need = free_of_scratch ? 0 : ws_layout(t->search_levels, nq).total;
    if (!free_of_scratch && (!workspace || workspace_bytes < need))
        return fail(TK_EWORKSPACE, "workspace too small: need " + std::to_string(need) + " bytes");
    if (ws_misaligned(workspace)) return fail(TK_EINVAL, "workspace must be 256-byte aligned");
    DeviceGuard g(t->device);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char* ws = static_cast<char*>(workspace);
    return run_query_any(t, q, int(nq), k, dists, idx, o, ws, s);
}

}  // extern "C"

// ------------------------------------------------------ transient trees --

namespace tk {
namespace {

// The tree of one call, its depth the one that the call's query wants.
tk_tree transient_tree(int64_t n, int64_t nq, int dims, int k, int dtype) {
    tk_tree t;
    t.dtype = dtype;
    t.dims = dims;
    t.n = n;
    if (cudaGetDevice(&t.device) != cudaSuccess) t.device = 0;
    t.host_layout = false;
    t.one_image = true;
    t.own_image = false;
    t.auto_depth = true;
    t.nan_empty = true;
    t.search_levels = kMaxLevels;
    if (tree_image(n, dims, dtype, 1).f_pts) t.d_filter[0] = &t;  // it will have one: shapes the query (set_image places it)
    t.search_levels = query_levels(&t, auto_lanes(&t, nq, k), k);
    t.levels = t.search_levels;
    return t;
}

struct TransientWs {
    size_t image = 0, build = 0, query = 0, total = 0;
};
TransientWs transient_ws(const tk_tree& t, int64_t nq) {
    TransientWs w;
    size_t o = align_up(tree_image(t.n, t.dims, t.dtype, t.search_levels).total, 256);
    w.build = o;
    o += align_up(build_workspace_bytes(t.n, t.dims, t.dtype), 256);
    w.query = o;
    o += align_up(ws_layout(t.search_levels, nq).total, 256);
    w.total = o;
    return w;
}

}  // namespace

size_t transient_tree_workspace_bytes(int64_t n, int64_t nq, int dims, int k, int dtype) {
    return transient_ws(transient_tree(n, nq, dims, k, dtype), nq).total;
}

int transient_tree_query(const void* ref, int64_t n, const void* q, int64_t nq, int dims, int k, int dtype,
                         void* dists, int32_t* idx, void* workspace, void* stream, const int** odd) {
    tk_tree t = transient_tree(n, nq, dims, k, dtype);
    const TransientWs w = transient_ws(t, nq);
    char* ws = static_cast<char*>(workspace);
    set_image(&t, ws + w.image);
    const int rc = dtype == TK_F32
                       ? enqueue_device_tree<float>(static_cast<const float*>(ref), n, dims, stream, &t, ws + w.build, odd)
                       : enqueue_device_tree<double>(static_cast<const double*>(ref), n, dims, stream, &t, ws + w.build, odd);
    if (rc != TK_OK) return rc;
    const tk_query_opts o{0, -1, -1, 0, 0, nullptr, nullptr, -1, 0};
    return run_query_any(&t, q, int(nq), k, dists, idx, o, ws + w.query, static_cast<cudaStream_t>(stream));
}

}  // namespace tk

// ------------------------------------------------ allocation-free query --
//
// Scratch of tk_tree_query_noalloc: one static device array, sized for
// TK_NOALLOC_MAX_QUERIES queries (counter + 2^16 cell counts + four 32-bit
// arrays of that many queries + the scratch of the cost-class radix pass:
// 256 counts per tile of 2,048 queries and their scan's tile sums, laid out
// as ws_layout() lays out a caller's workspace; the call checks the layout
// against this size before any launch).  Every GPU that loads the library
// holds it until the process exits, and every call on a device shares it.
namespace tk {
namespace {

constexpr size_t kNoAllocScratchBytes = 256 + sizeof(int) * (size_t(1) << kMaxBinLevels) +
                                        4 * sizeof(int) * size_t(TK_NOALLOC_MAX_QUERIES) +
                                        sizeof(int) * 256 * ((size_t(TK_NOALLOC_MAX_QUERIES) + 2047) / 2048) + 1024;
static_assert(TK_NOALLOC_MAX_QUERIES % 64 == 0, "each scratch array must stay 256-byte aligned");

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_noalloc_mu;
void* g_noalloc_ptr[kNoAllocMaxDevices] = {};

// Device address of g_noalloc_scratch on the current device (looked up once
// per device; in host code the symbol itself is only a host-side stand-in).
int noalloc_scratch(int dev, void** out) {
    if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(TK_EINVAL, "device ordinal out of range");
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return fail(TK_ECUDA, std::string("cudaGetSymbolAddress(scratch): ") + cudaGetErrorString(e));
        g_noalloc_ptr[dev] = p;
    }
    *out = g_noalloc_ptr[dev];
    return TK_OK;
}

}  // namespace
}  // namespace tk

extern "C" int tk_tree_query_noalloc(const tk_tree* t, const void* q, int64_t nq, int k, void* dists, int32_t* idx,
                                     const tk_query_opts* opts, void* stream) {
    clear_error();
    if (!t) return fail(TK_EINVAL, "tree is null");
    if (nq < 0 || nq > TK_NOALLOC_MAX_QUERIES)
        return fail(TK_EINVAL, "tk_tree_query_noalloc takes at most " + std::to_string(TK_NOALLOC_MAX_QUERIES) +
                                   " queries per call (got " + std::to_string(nq) + "); split the batch");
    if (k < 1) return fail(TK_EINVAL, "k must be >= 1");
    if (k > t->n) return fail(TK_EINVAL, "You requested more nearest neighbors than there are in the KD-Tree");
    if (k > kMaxK) return fail(TK_EINVAL, "k is limited to 128 on the GPU");
    if (t->device < 0 || !t->d_pts) return fail(TK_EINVAL, "tree was built host-only (device < 0); it has no device image");
    if (nq == 0) return TK_OK;
    if (!q || !dists || !idx) return fail(TK_EINVAL, "null query or output pointer");
    DeviceGuard g(t->device);
    void* scratch = nullptr;
    int rc = noalloc_scratch(t->device, &scratch);
    if (rc != TK_OK) return rc;
    if (ws_layout(t->search_levels, nq).total > kNoAllocScratchBytes)
        return fail(TK_EINVAL, "query needs more scratch than the static array holds");
    tk_query_opts o{0, -1, -1, 0, 0, nullptr, nullptr, -1, 0};
    if (opts) o = *opts;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    char* ws = static_cast<char*>(scratch);
    return run_query_any(t, q, int(nq), k, dists, idx, o, ws, s);
}

// ------------------------------------------------- host-buffer query --
//
// tk_tree_query_host: queries and results in host memory.  The queries are
// uploaded into device staging with one copy (the search reads each query
// more than once; host reads at link latency slowed it down), then:
//  * direct: the result buffers are registered (pinned) memory that the GPU
//    can address, so the query kernel writes the results into host memory
//    itself (over NVLink-C2C on Grace-Blackwell), spread over the search
//    instead of a download after it;
//  * staged: the results go to device staging and are downloaded after the
//    search.
// Device staging and workspace are kept per tree (grown as needed) and freed
// with it; calls on one tree are serialised by its mutex.

namespace tk {

struct HostPipe {
    std::mutex mu;
    char* buf = nullptr;
    size_t cap = 0;
};

void free_host_pipe(HostPipe* p) {
    if (!p) return;
    if (p->buf) cudaFree(p->buf);
    delete p;
}

namespace {

std::mutex g_pipe_create_mu;

HostPipe* host_pipe(const tk_tree* t) {
    std::lock_guard<std::mutex> lk(g_pipe_create_mu);
    if (!t->pipe) t->pipe = new HostPipe();
    return t->pipe;
}

// Device address of registered host memory, or null when the GPU cannot
// address it (pageable memory, or not host memory at all).
void* mapped_host(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return a.type == cudaMemoryTypeHost ? a.devicePointer : nullptr;
}

int pipe_buffer(HostPipe* p, size_t need, char** out) {
    if (p->cap < need) {
        if (p->buf) cudaFree(p->buf);
        p->buf = nullptr;
        p->cap = 0;
        const cudaError_t e = cudaMalloc(&p->buf, need);
        if (e != cudaSuccess) return fail(TK_ECUDA, std::string("host query staging: ") + cudaGetErrorString(e));
        p->cap = need;
    }
    *out = p->buf;
    return TK_OK;
}

}  // namespace
}  // namespace tk

extern "C" int tk_tree_query_host(const tk_tree* t, const void* q, int64_t nq, int k, void* dists, int32_t* idx,
                                  const tk_query_opts* opts, int transfer, void* stream) {
    using namespace tk;
    clear_error();
    if (!t) return fail(TK_EINVAL, "tree is null");
    if (nq < 0 || nq >= (int64_t(1) << 31)) return fail(TK_EINVAL, "number of queries must be in [0, 2^31)");
    if (k < 1) return fail(TK_EINVAL, "k must be >= 1");
    if (k > t->n) return fail(TK_EINVAL, "You requested more nearest neighbors than there are in the KD-Tree");
    if (k > kMaxK) return fail(TK_EINVAL, "k is limited to 128 on the GPU");
    if (t->device < 0 || !t->d_pts) return fail(TK_EINVAL, "tree was built host-only (device < 0); it has no device image");
    if (transfer != TK_HOST_AUTO && transfer != TK_HOST_DIRECT && transfer != TK_HOST_STAGED)
        return fail(TK_EINVAL, "transfer must be TK_HOST_AUTO, TK_HOST_DIRECT or TK_HOST_STAGED");
    if (nq == 0) return TK_OK;
    if (!q || !dists || !idx) return fail(TK_EINVAL, "null query or output pointer");

    DeviceGuard g(t->device);
    void* md = nullptr;
    void* mi = nullptr;
    if (transfer != TK_HOST_STAGED) {
        md = mapped_host(dists);
        mi = mapped_host(idx);
    }
    const bool direct = md && mi;
    if (transfer == TK_HOST_DIRECT && !direct)
        return fail(TK_EINVAL, "direct transfer needs registered (pinned) result buffers the GPU can address");

    HostPipe* p = host_pipe(t);
    std::lock_guard<std::mutex> lk(p->mu);
    const size_t es = t->dtype == TK_F32 ? 4 : 8;
    const size_t qb = es * size_t(t->dims) * size_t(nq), db = es * size_t(k) * size_t(nq),
                 ib = 4 * size_t(k) * size_t(nq);
    const size_t wsb = align_up(ws_layout(t->search_levels, nq).total, 256);
    const size_t need = wsb + align_up(qb, 256) + (direct ? 0 : align_up(db, 256) + align_up(ib, 256));
    char* buf = nullptr;
    int rc = pipe_buffer(p, need, &buf);
    if (rc != TK_OK) return rc;
    tk_query_opts o{0, -1, -1, 0, 0, nullptr, nullptr, -1, 0};
    if (opts) o = *opts;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaSuccess;
    char* dq = buf + wsb;
    e = cudaMemcpyAsync(dq, q, qb, cudaMemcpyDefault, s);  // unified addressing: any kind of buffer
    if (direct) {
        if (e == cudaSuccess) rc = tk_tree_query(t, dq, nq, k, md, static_cast<int32_t*>(mi), &o, buf, wsb, s);
    } else {
        char* dd = dq + align_up(qb, 256);
        char* di = dd + align_up(db, 256);
        if (e == cudaSuccess) rc = tk_tree_query(t, dq, nq, k, dd, reinterpret_cast<int32_t*>(di), &o, buf, wsb, s);
        if (e == cudaSuccess && rc == TK_OK) e = cudaMemcpyAsync(dists, dd, db, cudaMemcpyDefault, s);
        if (e == cudaSuccess && rc == TK_OK) e = cudaMemcpyAsync(idx, di, ib, cudaMemcpyDefault, s);
    }
    const cudaError_t se = cudaStreamSynchronize(s);  // whatever was queued completes, also on failure
    if (rc != TK_OK) return rc;
    if (e == cudaSuccess) e = se;
    if (e != cudaSuccess) return fail(TK_ECUDA, std::string("host query: ") + cudaGetErrorString(e));
    return TK_OK;
}
