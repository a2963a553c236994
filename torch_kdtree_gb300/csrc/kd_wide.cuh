// Exact KD-tree KNN query for trees of 4 to 8 dimensions (sm_103a).
//
// The reference compiles its KD-tree for dims 1-3 and tells users to add
// template instantiations for more (its README); the query is the same
// algorithm at any dimension.  Trees of up to 3 dimensions keep the 16-byte
// point records of kd_query.cuh; here, a tree of `dims` in 4..8 stores
// W = 4 (dims 4), 6 (dims 5-6) or 8 (dims 7-8) zero-padded coordinates per point, its
// original indices in a separate array, and node boxes as lo / hi rows of W.
// Padded coordinates are 0 in both the records and the (padded) query, so
// each adds (0 - 0)^2 = +0 to the distance after the real terms: the sum is
// the reference's ((0 + d0^2) + d1^2) + ... bit for bit.  The split axis
// cycles with the real `dims`.
//
// Queries are binned by cell, warps persistent.  One lane per query (k <= 16)
// searches with exact per-axis plane bounds on a stack of far cells and
// node-box pruning; a warp per query (k <= 128) walks as kd_warp.cuh says.  A
// leaf point is first tested as a float against the list's worst distance;
// only candidates that pass load their original index and build the
// (distance, index) key.
#pragma once

#include <cuda_runtime.h>

#include "kd_warp.cuh"
#include "tk_device.cuh"
#include "tk_internal.h"

namespace tk {

template <typename T>
struct KdWideArgs {
    const T* pts;             // [n][W] coordinates in leaf order, zero padded
    const int32_t* perm;      // [n] original index of each point
    const T* medians;         // [2^L - 1] heap order
    const int32_t* leaf_off;  // [2^(L + leaf_shift) + 1]
    const T* boxes;           // [2 (2^(L+1) - 1)][W]: node i's lo row at 2i, hi row at 2i+1; or null
    int levels, smem_levels, dims;
    int leaf_shift;           // the image's leaves lie this many levels below the searched ones
    const T* q;               // [nq, dims]
    int nq, k;
    const int32_t* order;     // [nq] processing order (binned), or null
    T* out_d;                 // [nq, k]
    int32_t* out_i;           // [nq, k]
    int* work;                // global work counter, zero at launch; null: see next_queries
};

template <typename T, int W>
struct WideEntry {
    int node;
    T e[W];  // per-axis squared distance from the query to the cell's slab
};

// v[ax] for a run-time axis without indexing a register array dynamically
template <typename T, int W>
__device__ __forceinline__ T pick_w(const T (&v)[W], int ax) {
    T r = v[0];
#pragma unroll
    for (int c = 1; c < W; ++c) r = ax == c ? v[c] : r;
    return r;
}

template <typename T, int W>
__device__ __forceinline__ T sum_w(const T (&e)[W]) {
    T b = e[0];
#pragma unroll
    for (int c = 1; c < W; ++c) b = add_rn(b, e[c]);
    return b;
}

// Rows start at multiples of 4 W bytes (f32) or 8 W bytes (f64) from a
// cudaMalloc base: 16-byte loads for W = 4 and 8, 8-byte loads for W = 6 (f32).
template <typename T, int W>
__device__ __forceinline__ void load_row(const T* row, T (&c)[W]) {
    static_assert(W % 2 == 0, "rows of an even number of coordinates");
    if constexpr (sizeof(T) == 4 && W % 4 == 0) {
#pragma unroll
        for (int i = 0; i < W / 4; ++i) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(row) + i);
            c[4 * i] = v.x;
            c[4 * i + 1] = v.y;
            c[4 * i + 2] = v.z;
            c[4 * i + 3] = v.w;
        }
    } else if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int i = 0; i < W / 2; ++i) {
            const float2 v = __ldg(reinterpret_cast<const float2*>(row) + i);
            c[2 * i] = v.x;
            c[2 * i + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < W / 2; ++i) {
            const double2 v = __ldg(reinterpret_cast<const double2*>(row) + i);
            c[2 * i] = v.x;
            c[2 * i + 1] = v.y;
        }
    }
}

// The reference's distance arithmetic over W (zero-padded) coordinates.
template <typename T, int W>
__device__ __forceinline__ T sqdist_w(const T (&q)[W], const T (&p)[W]) {
    const T d0 = sub_rn(q[0], p[0]);
    T acc = mul_rn(d0, d0);
#pragma unroll
    for (int c = 1; c < W; ++c) {
        const T dc = sub_rn(q[c], p[c]);
        acc = add_rn(acc, mul_rn(dc, dc));
    }
    return acc;
}

// Lower bound on the computed distance to any point in node's box (as
// box_bound in kd_query.cuh, over W coordinates).
template <typename T, int W>
__device__ __forceinline__ T box_bound_w(const T* boxes, int node, const T (&q)[W]) {
    T lo[W], hi[W], e[W];
    load_row<T, W>(boxes + size_t(2 * node) * W, lo);
    load_row<T, W>(boxes + size_t(2 * node + 1) * W, hi);
#pragma unroll
    for (int c = 0; c < W; ++c) {
        const T g = q[c] < lo[c] ? sub_rn(q[c], lo[c]) : (q[c] > hi[c] ? sub_rn(q[c], hi[c]) : T(0));
        e[c] = mul_rn(g, g);
    }
    return sum_w<T, W>(e);
}

// One lane per query.
template <typename T, int W, int R>
__device__ __forceinline__ void kd_search_wide(const KdWideArgs<T>& a, const T* s_med, const T (&q)[W], T* out_d,
                                               int32_t* out_i) {
    TopK<T, 1, R> list;
    list.init(a.k, 0);
    Key<T> worst = Key<T>::sentinel();
    T worst_d = worst.dist();
    WideEntry<T, W> stk[kMaxLevels];  // far cells
    int sp = 0;
    int node = 0, depth = 0;
    T e[W];
#pragma unroll
    for (int c = 0; c < W; ++c) e[c] = T(0);
    const int L = a.levels, dims = a.dims;
    const int first_leaf = (1 << L) - 1;

    for (;;) {
        int ax = depth % dims;
        while (depth < L) {
            const T m = depth < a.smem_levels ? s_med[node] : __ldg(a.medians + node);
            const T qa = pick_w<T, W>(q, ax);
            const T diff = sub_rn(qa, m);
            const T plane = mul_rn(diff, diff);
            const bool go_left = qa < m;  // src/kdtree.cpp:30
            WideEntry<T, W> far;
            far.node = 2 * node + (go_left ? 2 : 1);
#pragma unroll
            for (int c = 0; c < W; ++c) far.e[c] = (c == ax) ? plane : e[c];
            if (sum_w<T, W>(far.e) <= worst_d) {
                stk[sp] = far;
                ++sp;
            }
            node = 2 * node + (go_left ? 1 : 2);
            ++depth;
            ax = (ax + 1 == dims) ? 0 : ax + 1;
        }
        if (!a.boxes || box_bound_w<T, W>(a.boxes, node, q) <= worst_d) {
            const int leaf = node - first_leaf;
            const int beg = __ldg(a.leaf_off + (leaf << a.leaf_shift));
            const int end = __ldg(a.leaf_off + ((leaf + 1) << a.leaf_shift));
            for (int j = beg; j < end; ++j) {
                T p[W];
                load_row<T, W>(a.pts + size_t(j) * W, p);
                const T d = sqdist_w<T, W>(q, p);
                if (d <= worst.dist())
                    worst = offer<T, 1, R>(list, Key<T>::make(d, uint32_t(__ldg(a.perm + j))), worst, 0u, 0, 0);
            }
            worst_d = worst.dist();
        }
        bool resumed = false;
        while (sp > 0) {
            --sp;
            const WideEntry<T, W> s = stk[sp];
            if (sum_w<T, W>(s.e) <= worst_d && (!a.boxes || box_bound_w<T, W>(a.boxes, s.node, q) <= worst_d)) {
                node = s.node;
#pragma unroll
                for (int c = 0; c < W; ++c) e[c] = s.e[c];
                depth = 31 - __clz(node + 1);
                resumed = true;
                break;
            }
        }
        if (!resumed) break;
    }
    list.store(a.k, 0, out_d, out_i, 0);
}

// The same search with a whole warp per query (kd_warp.cuh); always prunes
// with node boxes.
template <typename T, int W, int R>
__device__ __forceinline__ void kd_search_wide_warp(const KdWideArgs<T>& a, const T (&q)[W], T* out_d, int32_t* out_i,
                                                    Key<T>* buf, int lane) {
    WarpList<T, R> wl;
    wl.init(a.k, buf, lane);
    const int L = a.levels, dims = a.dims;
    const int first_leaf = (1 << L) - 1;
    bool nan_q = false;  // all distances are NaN and enter no list: the home leaf is enough
#pragma unroll
    for (int c = 0; c < W; ++c) nan_q |= q[c] != q[c];
    auto qa = [&](int ax) { return pick_w<T, W>(q, ax); };

    int leaf = warp_descend(a.medians, 0, 0, L, dims, lane, qa);
    T bound = T(0);  // of this lane's sibling (lane 31: of the leaf)
    bool pending = false;
    int range = 0;  // lanes 29, 30: the leaf's point range
    for (int fresh = 0;;) {  // lanes fresh .. L - 1 have new siblings
        if ((lane >= fresh && lane < L) || lane == 31) {
            bound = box_bound_w<T, W>(a.boxes, lane == 31 ? leaf : path_sibling(leaf, L, lane), q);
            pending = lane != 31 && !nan_q;
        } else if (lane >= 29) {
            range = __ldg(a.leaf_off + ((leaf - first_leaf + lane - 29) << a.leaf_shift));
        }
        const int beg = __shfl_sync(0xFFFFFFFFu, range, 29);
        const int end = __shfl_sync(0xFFFFFFFFu, range, 30);
        if (__shfl_sync(0xFFFFFFFFu, bound, 31) <= wl.worst.dist()) {
            T p[W];
            if (beg + lane < end) load_row<T, W>(a.pts + size_t(beg + lane) * W, p);
            for (int j = beg + lane; j - lane < end; j += 32) {
                T d = T(0);
                if (j < end) d = sqdist_w<T, W>(q, p);
                if (j + 32 < end) load_row<T, W>(a.pts + size_t(j + 32) * W, p);
                Key<T> mine = Key<T>::sentinel();
                if (j < end && d <= wl.worst.dist()) mine = Key<T>::make(d, uint32_t(__ldg(a.perm + j)));
                wl.offer(mine, lane);
            }
            wl.flush(lane);
        }
        const unsigned m = __ballot_sync(0xFFFFFFFFu, pending && bound <= wl.worst.dist());
        if (!m) break;
        const int t = 31 - __clz(m);
        pending = pending && lane < t;
        leaf = warp_descend(a.medians, path_sibling(leaf, L, t), t + 1, L, dims, lane, qa);
        fresh = t + 1;
    }
    wl.list.store(a.k, lane, out_d, out_i, 0);
}

// A warp per query at 5 blocks of 256 per SM (48 registers): 7% faster at 6
// and 8 dims than the 62 registers it takes freely; the next rows loaded
// while the last are offered: 4%.
template <typename T, int W, int G, int R>
__global__ void __launch_bounds__(256, G == 1 ? 0 : (sizeof(T) == 4 ? (R < 4 ? 5 : 4) : 1)) k_kd_wide(const KdWideArgs<T> a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* s_med = reinterpret_cast<T*>(smem_raw);
    Key<T>* buf = nullptr;
    if constexpr (G == 32) {
        __shared__ Key<T> bufs[8][64];
        buf = bufs[threadIdx.x >> 5];
    } else {
        const int n_smem = (1 << a.smem_levels) - 1;
        for (int i = threadIdx.x; i < n_smem; i += blockDim.x) s_med[i] = a.medians[i];
        __syncthreads();
    }

    const int lane = threadIdx.x & 31;
    constexpr int kGroupsPerWarp = 32 / G;
    const int gid = lane / G;
    for (int round = 0;;) {
        const int base = next_queries(a.work, kGroupsPerWarp, a.nq, round);
        if (base >= a.nq) break;
        const int t = base + gid;
        if (t < a.nq) {
            const int qi = a.order ? __ldg(a.order + t) : t;
            T q[W];
#pragma unroll
            for (int c = 0; c < W; ++c) q[c] = c < a.dims ? a.q[(long long)qi * a.dims + c] : T(0);
            T* out_d = a.out_d + (long long)qi * a.k;
            int32_t* out_i = a.out_i + (long long)qi * a.k;
            if constexpr (G == 32) kd_search_wide_warp<T, W, R>(a, q, out_d, out_i, buf, lane);
            else kd_search_wide<T, W, R>(a, s_med, q, out_d, out_i);
        }
        __syncwarp();
    }
}

// Cell id at depth B of every query (axis cycling over the real dims), its
// arrival rank within the cell, and (with `boxes`, rows of width W) its cost
// class from the home leaf at depth L, as k_bin_count for narrow trees:
// bin_of = cell | class << 16.  Ordering the launch by class took 7-8% off
// the 4- and 8-dim searches of 262,144 queries in 1,048,576 N(0,1) points.
template <typename T>
__global__ void k_bin_count_wide(const T* __restrict__ q, int nq, int dims, const T* __restrict__ medians, int B,
                                 int L, const T* __restrict__ boxes, int W, int* __restrict__ counts,
                                 int* __restrict__ bin_of, int* __restrict__ pos_of) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nq) return;
    const T* p = q + (long long)i * dims;
    int node = 0, ax = 0, bin = 0;
    const int stop = boxes ? L : B;
    for (int depth = 0; depth < stop; ++depth) {
        if (depth == B) bin = node - ((1 << B) - 1);
        const T m = __ldg(medians + node);
        node = 2 * node + (p[ax] < m ? 1 : 2);
        ax = (ax + 1 == dims) ? 0 : ax + 1;
    }
    if (stop == B) bin = node - ((1 << B) - 1);
    uint32_t cls = 0;
    if (boxes) {
        const T* lo = boxes + size_t(2 * node) * W;
        const T* hi = lo + W;
        float far2 = 0.f;
        for (int c = 0; c < dims; ++c) {
            const T x = p[c];
            const float f = float(fmax(fabs(x - __ldg(lo + c)), fabs(x - __ldg(hi + c))));
            far2 += f * f;
        }
        cls = cost_class(far2);
    }
    bin_of[i] = bin | int(cls << 16);
    pos_of[i] = atomicAdd(counts + bin, 1);
}

// Launchers (kd_wide_f32.cu, kd_wide_f64.cu): G in {1, 32}; R in {1, 2, 4, 8,
// 16} for G = 1, {0, 1, 2, 4} for G = 32.
template <typename T>
const void* kd_wide_kernel(int W, int G, int R);
template <typename T>
int kd_wide_launch(const KdWideArgs<T>& a, int W, int G, int R, int grid, int block, size_t smem, cudaStream_t s);
template <typename T>
void bin_count_wide_launch(const T* q, int nq, int dims, const T* medians, int B, int L, const T* boxes, int W,
                           int* counts, int* bin_of, int* pos_of, cudaStream_t s);

}  // namespace tk
