// Building blocks of the searches that give a whole warp to one query
// (kd_query.cuh: trees of 1-3 dims; kd_wide.cuh: 4-8 dims).
//
// The walk is depth first.  The path from the root to the current leaf
// follows from the leaf's heap index, and lane t looks after the sibling of
// the path's node at depth t + 1: when the path changes below some depth,
// the lanes below it load their new siblings' boxes and compute their bounds
// side by side, in one round trip to memory that also fetches the leaf's own
// box and point range (lane 31; leaves are at depth <= 24).  A bound never
// changes, so choosing the next node is one ballot: the deepest lane whose
// bound is within reach of the current k-th distance.  Descending to the near
// leaf reads the split values of five levels at once, one per lane, and
// walks them with shuffles.  A leaf visit so costs about three dependent
// round trips; checking one pending sibling after the other, with every lane
// loading the same box, and descending a level per load cost up to ten.
//
// Pruning is exact (see box_bound): a node is skipped only when its bound
// exceeds the current k-th distance.
#pragma once

#include <cuda_runtime.h>

#include "tk_device.cuh"

namespace tk {

// Leaf (depth L) of the subtree under `node` (at depth `depth`) that the
// query falls into (src/kdtree.cpp:30 rule); qa(axis) is its coordinate.
template <typename T, typename QAt>
__device__ __forceinline__ int warp_descend(const T* __restrict__ medians, int node, int depth, int L, int dims,
                                            int lane, QAt qa) {
    int ax = depth % dims;
    while (depth < L) {
        const int steps = min(5, L - depth);
        const int r = 31 - __clz(lane | 1);  // level of the subtree's heap entry `lane` (entry 1 is `node`)
        T m = T(0);
        if (lane > 0 && r < steps) m = __ldg(medians + ((node + 1) << r) - 1 + (lane - (1 << r)));
        int h = 1;
        for (int s = 0; s < steps; ++s) {
            const T split = __shfl_sync(0xFFFFFFFFu, m, h);
            h = 2 * h + (qa(ax) < split ? 0 : 1);
            ax = ax + 1 == dims ? 0 : ax + 1;
        }
        node = ((node + 1) << steps) - 1 + (h - (1 << steps));
        depth += steps;
    }
    return node;
}

// Sibling of the depth-(t + 1) node on the path to `leaf` (a node of depth L).
__device__ __forceinline__ int path_sibling(int leaf, int L, int t) { return ((leaf + 1) >> (L - 1 - t) ^ 1) - 1; }

// A warp's sorted list of the k best keys plus the candidates that beat its
// worst key and wait to be merged: 32 at a time in one sorted batch, or at
// the end of a leaf as a batch (from kBatch on) or one by one.  Inserting
// every candidate at once, unless 8 of 32 came together, was most of the work
// of large k.
template <typename T, int R>
struct WarpList {
    static constexpr int kBatch = 6;  // a batch costs about as much as six single insertions
    TopK<T, 32, R> list;
    Key<T> worst;
    Key<T>* buf;  // [64] in shared memory, this warp's
    int waiting;

    __device__ __forceinline__ void init(int k, Key<T>* shared, int lane) {
        list.init(k, lane);
        worst = Key<T>::sentinel();
        buf = shared;
        waiting = 0;
    }
    __device__ __forceinline__ void merge(const Key<T>& x, int lane) {
        list.merge_warp_batch(x, lane);
        worst = list.worst(0xFFFFFFFFu);
    }
    // One candidate per lane (sentinel where there is none).
    __device__ __forceinline__ void offer(const Key<T>& mine, int lane) {
        const bool hit = mine.lt(worst);
        const unsigned m = __ballot_sync(0xFFFFFFFFu, hit);
        if (!m) return;
        const int c = __popc(m);
        if (waiting == 0 && c >= 16) {  // while the list fills
            merge(hit ? mine : Key<T>::sentinel(), lane);
            return;
        }
        if (hit) buf[waiting + __popc(m & ((1u << lane) - 1u))] = mine;
        waiting += c;
        __syncwarp();
        if (waiting >= 32) {
            const Key<T> x = buf[lane];
            const Key<T> rest = buf[32 + lane];
            __syncwarp();
            waiting -= 32;
            if (lane < waiting) buf[lane] = rest;
            merge(x, lane);
        }
    }
    __device__ __forceinline__ void flush(int lane) {
        if (waiting == 0) return;
        __syncwarp();
        if (waiting >= kBatch) {
            merge(lane < waiting ? buf[lane] : Key<T>::sentinel(), lane);
        } else {
            for (int i = 0; i < waiting; ++i) {
                const Key<T> c = buf[i];
                if (c.lt(worst)) {
                    list.insert(c, 0xFFFFFFFFu, lane);
                    worst = list.worst(0xFFFFFFFFu);
                }
            }
        }
        waiting = 0;
        __syncwarp();
    }
};

// k = 1 (kernels of R = 0): the nearest of a batch's candidates is the new
// worst key at once.  Buffered until the end of a leaf they kept the reach wide
// and cost a sort of 32 where one exchange does (1M queries in 1,000 points, 500
// a leaf, 1.27 -> 0.82 ms; 262,144 in 4M, 512 a leaf 0.58 -> 0.41).
template <typename T>
struct WarpList<T, 0> {
    struct Nearest {
        Key<T> key;
        __device__ __forceinline__ void store(int, int lane, T* out_d, int32_t* out_i, long long row) const {
            if (lane == 0) {
                out_d[row] = key.dist();
                out_i[row] = int32_t(key.index());
            }
        }
    } list;
    Key<T> worst;

    __device__ __forceinline__ void init(int, Key<T>*, int) { worst = list.key = Key<T>::sentinel(); }
    __device__ __forceinline__ void offer(const Key<T>& mine, int lane) {
        Key<T> x = mine.lt(worst) ? mine : worst;
        if (!__any_sync(0xFFFFFFFFu, mine.lt(worst))) return;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const Key<T> y = x.shfl(0xFFFFFFFFu, lane ^ o, 32);
            x = y.lt(x) ? y : x;
        }
        worst = list.key = x;
    }
    __device__ __forceinline__ void flush(int) {}
};

}  // namespace tk
