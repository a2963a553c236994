// KD-tree construction on the GPU, in exactly the layout build_host_tree
// produces (the reference's createKDTree, src/kdtree.hpp:392-534): node at
// depth t splits on axis t % dims, its points ordered along that axis by
// (coordinate, original index) send the first floor(n/2) left, split value =
// middle element or 0.5 * (a + b) of the two middle ones, leaves contiguous,
// points inside a leaf ordered along the leaf parent's axis.
//
// Presorted-axes construction instead of per-node sorting:
//   1. for every axis a, P_a = all point ids stably radix-sorted by the
//      coordinate's order-preserving key (ties keep ascending ids), all axes
//      in the same launches;
//   2. every node's points occupy the same range [lo, lo + c) in every P_a,
//      and node ranges depend only on n (left child = floor(c / 2)), so a
//      position finds its node by arithmetic (locate).  The split axis's
//      array gives the split value and each point's side, and the first and
//      last entry of a node's range in each P_a give its bounding box.  The
//      other axes' arrays are stably partitioned by side within their nodes,
//      which keeps both children's ranges sorted.  While nodes hold more than
//      kSub points this takes three launches a level for the whole array;
//   3. from there on a block per node does all remaining levels in shared
//      memory (k_subtrees) and writes split values, leaf offsets, node boxes
//      and point records straight into the tree's device image.
//
// What bounds it: launches and dependent gathers for small clouds, then the
// level passes' L2 traffic (a gather of the split coordinate per point, axis
// and level).  One sort per axis, seven launches per axis and level, boxes
// bottom-up and seventeen allocations took (1M / 4M points, default levels,
// build_kd_tree with the synchronisation) 2.7 / 4.7 ms and 0.93 ms for 10,000
// points; this takes 0.49 / 1.73 ms and 0.20 ms.
#include <algorithm>
#include <cstring>
#include <limits>
#include <string>
#include <vector>

#include "kd_filter.cuh"
#include "launch.cuh"
#include "tk_device.cuh"
#include "tk_internal.h"

namespace tk {
namespace {

constexpr int kSortThreads = 512;
constexpr int kScanThreads = 256;
constexpr int kTile = 1024;        // positions per block of the partition passes
constexpr int kSub = 4096;         // points of a subtree that one block finishes in shared memory
constexpr int kSubThreads = 1024;
constexpr int kSubItems = kSub / kSubThreads;

// A build is a chain of some 30 short launches, each on the results of the one
// before: all but the first are set up ahead of time (launch.cuh; 65,536 points
// 0.28 -> 0.23 ms, 1M 0.55 -> 0.49).

template <typename T>
struct KeyBits;
template <>
struct KeyBits<float> {
    using type = uint32_t;
    static constexpr int kItems = 8;  // per thread and radix tile: 41 KiB of shared memory
};
template <>
struct KeyBits<double> {
    using type = unsigned long long;
    static constexpr int kItems = 4;
};
template <typename T>
constexpr int radix_tile() {
    return kSortThreads * KeyBits<T>::kItems;
}

// One id array per axis (or per axis of a group), as a kernel argument: equal
// arrays of one buffer, array a in slot `slots` byte a.  (An array of pointers
// that a kernel indexes at run time is copied to every thread's local memory;
// that copy was most of the memory traffic of the level passes.)
struct Arrays {
    uint32_t* base = nullptr;
    int64_t stride = 0;
    uint64_t slots = 0;
    __host__ __device__ __forceinline__ uint32_t* operator[](int a) const {
        return base + int64_t((slots >> (8 * a)) & 255u) * stride;
    }
    void set(int a, int slot) {
        slots &= ~(uint64_t(255) << (8 * a));
        slots |= uint64_t(slot) << (8 * a);
    }
    int slot(int a) const { return int((slots >> (8 * a)) & 255u); }
};

// Order-preserving unsigned keys; -0 and +0 get the same key (they compare
// equal on the host, so their order falls to the original index).
__device__ __forceinline__ uint32_t coord_key(float v) {
    const uint32_t b = __float_as_uint(v == 0.0f ? 0.0f : v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ unsigned long long coord_key(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v == 0.0 ? 0.0 : v);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

// odd[0]: some coordinate is NaN; odd[1]: some coordinate is NaN or infinite.
template <typename T>
__device__ __forceinline__ void mark_odd(T v, int* odd) {
    if (v - v != T(0)) {
        odd[1] = 1;
        if (v != v) odd[0] = 1;
    }
}

// Lanes of the warp whose 8-bit digit equals this lane's, among the valid
// ones (an invalid lane gets the other invalid lanes).  Eight ballots: faster
// here than __match_any_sync.
__device__ __forceinline__ unsigned same_digit(int digit, bool valid) {
    unsigned peers = __ballot_sync(0xFFFFFFFFu, valid);
    if (!valid) peers = ~peers;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool bit = (digit >> b) & 1;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, bit);
        peers &= bit ? m : ~m;
    }
    return peers;
}

// Exclusive sum over the block of one value per thread; warp_sums holds 32 ints.
__device__ __forceinline__ int block_exclusive(int v, int* warp_sums, int* total = nullptr) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= o) x += t;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int w = lane < nw ? warp_sums[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= o) w += t;
        }
        if (lane < nw) warp_sums[lane] = w;
    }
    __syncthreads();
    const int excl = x - v + (wid > 0 ? warp_sums[wid - 1] : 0);
    if (total) *total = warp_sums[nw - 1];
    __syncthreads();
    return excl;
}

// ----------------------------------------------------------- radix sort --
//
// Stable LSD radix sort by 8-bit digits, every axis of a group in the same
// launches (blockIdx.y): per pass a histogram per tile, an exclusive scan of
// each digit's row of tiles, and a scatter that ranks a tile's items in
// registers (ballots within a warp, a table across warps) and
// reorders them in shared memory so that equal digits leave as runs.

template <typename T, bool FIRST>
__global__ void __launch_bounds__(kSortThreads) k_radix_hist(const T* __restrict__ pts, int64_t n, int dims, int ax0,
                                                             const typename KeyBits<T>::type* keys,
                                                             int shift, int ntiles, int* hist,
                                                             int* __restrict__ odd) {
    begin();
    __shared__ int h[256];
    const int t = threadIdx.x, a = blockIdx.y;
    if (t < 256) h[t] = 0;
    __syncthreads();
    const int64_t base = int64_t(blockIdx.x) * radix_tile<T>();
#pragma unroll
    for (int i = 0; i < KeyBits<T>::kItems; ++i) {
        const int64_t e = base + i * kSortThreads + t;
        if (e < n) {
            typename KeyBits<T>::type k;
            if constexpr (FIRST) {
                const T v = pts[e * dims + ax0 + a];
                mark_odd(v, odd);
                k = coord_key(v);
            } else {
                k = keys[a * n + e];
            }
            atomicAdd(&h[int(k >> shift) & 255], 1);
        }
    }
    __syncthreads();
    if (t < 256) hist[(int64_t(a) * 256 + t) * ntiles + blockIdx.x] = h[t];
}

// Exclusive scan of every row (blockIdx.y * gridDim.x + blockIdx.x) of `len`
// counts in place; the row's total goes to totals.
__global__ void __launch_bounds__(kScanThreads) k_row_scan(int* rows, int len, int* totals) {
    begin();
    __shared__ int warp_sums[32];
    const int64_t row = int64_t(blockIdx.y) * gridDim.x + blockIdx.x;
    int* d = rows + row * len;
    int carry = 0;
    for (int base = 0; base < len; base += 4 * kScanThreads) {
        const int e = base + 4 * int(threadIdx.x);
        int v[4], s = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            v[i] = e + i < len ? d[e + i] : 0;
            s += v[i];
        }
        int total = 0;
        int run = carry + block_exclusive(s, warp_sums, &total);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            if (e + i < len) d[e + i] = run;
            run += v[i];
        }
        carry += total;
    }
    if (threadIdx.x == 0) totals[row] = carry;
}

// Up to kOwnScanTiles tiles there is no scan (totals null): a scatter block
// adds up its digits' rows of the histogram itself, which saves a launch per
// pass (30,000 points built in 0.208 -> 0.195 ms; with 64 tiles the rows cost
// more than the launch, 260,000 points 0.26 -> 0.30).
constexpr int kOwnScanTiles = 32;

template <typename T, bool FIRST, bool LAST>
__global__ void __launch_bounds__(kSortThreads, 2) k_radix_scatter(
    const T* __restrict__ pts, int64_t n, int dims, int ax0, const typename KeyBits<T>::type* kin,
    const Arrays vin, int shift, int ntiles, const int* hist, const int* totals,
    typename KeyBits<T>::type* kout, const Arrays vout) {
    begin();
    using K = typename KeyBits<T>::type;
    constexpr int ITEMS = KeyBits<T>::kItems, TILE = radix_tile<T>(), WARPS = kSortThreads / 32;
    __shared__ K skey[TILE];
    __shared__ uint32_t sval[TILE];
    __shared__ uint16_t cnt[WARPS][256];
    __shared__ int gbase[256];
    __shared__ int warp_sums[32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, a = blockIdx.y;
    const int64_t base = int64_t(blockIdx.x) * TILE;
    const int64_t e0 = base + w * (32 * ITEMS) + lane;
    for (int i = t; i < WARPS * 128; i += kSortThreads) reinterpret_cast<uint32_t*>(&cnt[0][0])[i] = 0;
    __syncthreads();
    K key[ITEMS];
    uint32_t val[ITEMS];
    int rank[ITEMS];
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const int64_t e = e0 + i * 32;
        key[i] = 0;
        val[i] = 0;
        if (e < n) {
            key[i] = FIRST ? coord_key(pts[e * dims + ax0 + a]) : kin[a * n + e];
            val[i] = FIRST ? uint32_t(e) : vin[a][e];
        }
    }
    // of digit t: items in tiles before this one, and in all
    int tiles_before = 0, row_total = 0;
    if (t < 256) {
        const int* row = hist + (int64_t(a) * 256 + t) * ntiles;
        if (totals) {
            tiles_before = row[blockIdx.x];
            row_total = totals[a * 256 + t];
        } else {
#pragma unroll 4
            for (int i = 0; i < ntiles; ++i) {
                const int c = row[i];
                tiles_before += i < int(blockIdx.x) ? c : 0;
                row_total += c;
            }
        }
    }
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        const bool valid = e0 + i * 32 < n;
        const int digit = int(key[i] >> shift) & 255;
        const unsigned peers = same_digit(digit, valid);
        const int before = cnt[w][digit];
        __syncwarp();
        if (valid && (peers & below) == 0) cnt[w][digit] = uint16_t(before + __popc(peers));
        __syncwarp();
        rank[i] = before + __popc(peers & below);
    }
    __syncthreads();
    // thread t < 256 owns digit t: place of every warp's run within the tile
    int run = 0;
    if (t < 256)
        for (int i = 0; i < WARPS; ++i) {
            const int c = cnt[i][t];
            cnt[i][t] = uint16_t(run);
            run += c;
        }
    const int lstart = block_exclusive(run, warp_sums);
    const int gstart = block_exclusive(row_total, warp_sums);
    if (t < 256) {
        gbase[t] = gstart + tiles_before - lstart;
        for (int i = 0; i < WARPS; ++i) cnt[i][t] = uint16_t(cnt[i][t] + lstart);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < ITEMS; ++i) {
        if (e0 + i * 32 < n) {
            const int pos = cnt[w][int(key[i] >> shift) & 255] + rank[i];
            skey[pos] = key[i];
            sval[pos] = val[i];
        }
    }
    __syncthreads();
    const int m = int(min(int64_t(TILE), n - base));
    for (int j = t; j < m; j += kSortThreads) {
        const K k = skey[j];
        const int64_t dst = int64_t(gbase[int(k >> shift) & 255]) + j;
        if (!LAST) kout[a * n + dst] = k;
        vout[a][dst] = sval[j];
    }
}

// Clouds of up to kSub points: one block per axis sorts in shared memory, all
// digits in one launch.
template <typename T>
__global__ void __launch_bounds__(kSubThreads) k_small_sort(const T* __restrict__ pts, int n, int dims,
                                                            const Arrays out, int* __restrict__ odd) {
    using K = typename KeyBits<T>::type;
    constexpr int WARPS = kSubThreads / 32;
    extern __shared__ __align__(16) unsigned char smem[];
    K* skey = reinterpret_cast<K*>(smem);                                      // [kSub]
    uint16_t* sval = reinterpret_cast<uint16_t*>(skey + kSub);                 // [kSub]
    uint16_t* cnt = sval + kSub;                                               // [WARPS][256]
    __shared__ int warp_sums[32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5, a = blockIdx.x;
    for (int i = t; i < n; i += kSubThreads) {
        const T v = pts[int64_t(i) * dims + a];
        mark_odd(v, odd);
        skey[i] = coord_key(v);
        sval[i] = uint16_t(i);
    }
    __syncthreads();
    const int e0 = w * (32 * kSubItems) + lane;
    const unsigned below = (1u << lane) - 1u;
    for (int shift = 0; shift < int(sizeof(K)) * 8; shift += 8) {
        for (int i = t; i < WARPS * 256; i += kSubThreads) cnt[i] = 0;
        K key[kSubItems];
        uint16_t val[kSubItems];
        int rank[kSubItems];
#pragma unroll
        for (int i = 0; i < kSubItems; ++i) {
            const int e = e0 + i * 32;
            key[i] = e < n ? skey[e] : K(0);
            val[i] = e < n ? sval[e] : uint16_t(0);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kSubItems; ++i) {
            const bool valid = e0 + i * 32 < n;
            const int digit = int(key[i] >> shift) & 255;
            const unsigned peers = same_digit(digit, valid);
            const int before = cnt[w * 256 + digit];
            __syncwarp();
            if (valid && (peers & below) == 0) cnt[w * 256 + digit] = uint16_t(before + __popc(peers));
            __syncwarp();
            rank[i] = before + __popc(peers & below);
        }
        __syncthreads();
        int run = 0;
        if (t < 256) {
            for (int i = 0; i < WARPS; ++i) {
                const int c = cnt[i * 256 + t];
                cnt[i * 256 + t] = uint16_t(run);
                run += c;
            }
        }
        const int start = block_exclusive(t < 256 ? run : 0, warp_sums);
        if (t < 256)
            for (int i = 0; i < WARPS; ++i) cnt[i * 256 + t] = uint16_t(cnt[i * 256 + t] + start);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kSubItems; ++i) {
            if (e0 + i * 32 < n) {
                const int pos = cnt[w * 256 + (int(key[i] >> shift) & 255)] + rank[i];
                skey[pos] = key[i];
                sval[pos] = val[i];
            }
        }
        __syncthreads();
    }
    for (int i = t; i < n; i += kSubThreads) out[a][i] = sval[i];
}

template <typename T>
size_t small_sort_smem() {
    return kSub * sizeof(typename KeyBits<T>::type) + kSub * sizeof(uint16_t) + (kSubThreads / 32) * 256 * sizeof(uint16_t);
}

// --------------------------------------------------------- node arithmetic --

// Node of depth t that position p of the n points falls into: index j in its
// level, first position lo, point count c, and the number of points that go
// left at depth t in all nodes before it (`lefts`).  A node of c points gives
// floor(c / 2) to its left child, so the 2^r nodes r levels below a node of c
// points hold floor(c / 2^r) points each, the last c mod 2^r in bit-reversed
// order one more: the number of odd ones among them follows.
struct NodeAt {
    int j, lo, c, lefts;
};
__device__ __forceinline__ int lefts_below(int c, int r) {
    const int f = c >> r, m = c & ((1 << r) - 1);
    const int odd = (f & 1) ? (1 << r) - m : m;
    return (c - odd) >> 1;
}
__device__ __forceinline__ NodeAt locate(int n, int t, int p) {
    NodeAt a{0, 0, n, 0};
    for (int s = 0; s < t; ++s) {
        const int h = a.c >> 1;
        a.j <<= 1;
        if (p - a.lo >= h) {
            a.lefts += lefts_below(h, t - 1 - s);
            a.lo += h;
            a.c -= h;
            a.j |= 1;
        } else {
            a.c = h;
        }
    }
    return a;
}
// First position and point count of node j of depth t.
__device__ __forceinline__ void node_range(int n, int t, int j, int& lo, int& c) {
    lo = 0;
    c = n;
    for (int s = t - 1; s >= 0; --s) {
        const int h = c >> 1;
        if ((j >> s) & 1) {
            lo += h;
            c -= h;
        } else {
            c = h;
        }
    }
}

__device__ __forceinline__ float half_sum(float a, float b) {
    return __double2float_rn(__dmul_rn(0.5, double(__fadd_rn(a, b))));
}
__device__ __forceinline__ double half_sum(double a, double b) { return __dmul_rn(0.5, __dadd_rn(a, b)); }
__device__ __forceinline__ float index_bits(uint32_t v, float) { return __uint_as_float(v); }
__device__ __forceinline__ double index_bits(uint32_t v, double) { return __longlong_as_double((long long)v); }

// The tree's device image (see tk_internal.h).
template <typename T>
struct Image {
    T* pts;             // point records, or rows of W coordinates (trees of 4-8 dims)
    int32_t* perm;      // trees of 4-8 dims
    T* medians;
    int32_t* leaf_off;
    T* boxes;
    int levels;         // depth of the leaves
    int W;              // record_width(dims)
};

// One of the node_parts(dims) entries of node j of depth s, whose c points
// stand in positions lo .. lo + c of every axis's order: the lower and upper
// bound of each axis (its order starts at the minimum and ends at the
// maximum), then the rest (point range, split value or leaf offset).  A
// thread per entry: a thread per node waited for one gather after the other.
// id_at(axis, i): id of the i-th point of the node along the axis.
// compMedian (src/kdtree.hpp:392-401): odd n -> element h, even n -> 0.5 *
// (element h-1 + element h), the sum rounded in T and the product in double.
__device__ __forceinline__ int node_parts(int dims) { return 2 * dims + 1; }
template <typename T, typename IdAt>
__device__ __forceinline__ void write_node_part(const T* __restrict__ pts, int dims, const Image<T>& im, int s, int j,
                                                int lo, int c, int part, IdAt id_at) {
    const int64_t node = (int64_t(1) << s) - 1 + j;
    const T inf = std::numeric_limits<T>::infinity();
    const bool wide = dims > 3;
    const int bs = wide ? im.W : 4;  // coordinates per box row
    T* lo_row = im.boxes + (2 * node) * bs;
    T* hi_row = lo_row + bs;
    if (part < 2 * dims) {
        const int a = part >> 1, upper = part & 1;
        const T v = c > 0 ? pts[int64_t(id_at(a, upper ? c - 1 : 0)) * dims + a] : (upper ? -inf : inf);
        (upper ? hi_row : lo_row)[a] = v;
        return;
    }
    for (int a = dims; a < im.W; ++a) {
        lo_row[a] = c > 0 ? T(0) : inf;
        hi_row[a] = c > 0 ? T(0) : -inf;
    }
    if (!wide) {  // the box records also carry the node's point range [begin, end)
        lo_row[3] = index_bits(uint32_t(lo), T(0));
        hi_row[3] = index_bits(uint32_t(lo + c), T(0));
    }
    if (s < im.levels) {
        const int ax = s % dims, h = c / 2;
        if (c > 0) {
            const T upper = pts[int64_t(id_at(ax, h)) * dims + ax];
            const T lower = pts[int64_t(id_at(ax, h > 0 ? h - 1 : 0)) * dims + ax];
            im.medians[node] = (c & 1) ? upper : half_sum(lower, upper);
        }
    } else {
        im.leaf_off[j] = lo;
        if (j == (1 << s) - 1) im.leaf_off[j + 1] = lo + c;
    }
}

template <typename T>
__device__ __forceinline__ void write_point(const T* __restrict__ pts, int dims, const Image<T>& im, int64_t p,
                                            uint32_t id) {
    const T* src = pts + int64_t(id) * dims;
    if (dims > 3) {
        for (int d = 0; d < im.W; ++d) im.pts[p * im.W + d] = d < dims ? src[d] : T(0);
        im.perm[p] = int32_t(id);
    } else {
        PointRec<T> r;
        r.x = src[0];
        r.y = dims > 1 ? src[1] : T(0);
        r.z = dims > 2 ? src[2] : T(0);
        r.w = index_bits(id, T(0));
        reinterpret_cast<PointRec<T>*>(im.pts)[p] = r;
    }
}

// ------------------------------------------------------------ top levels --

// Level s over the whole array.  Slice blockIdx.y < naxes: which points of a
// group of axes' orders go left -- those before the middle element of their
// node's order along the split axis, by (coordinate, id) -- as bits, with
// their count per tile.  The slice after them writes the nodes' entries of
// the image.  (Marking each point's side in an array by id first, to be
// gathered here instead of the coordinate, cost another pass of scattered
// byte writes: 22 us a level at 1M points.)
template <typename T>
__global__ void __launch_bounds__(256) k_level_count(const T* __restrict__ pts, int n, int dims, int s, const Arrays P,
                                                     const Image<T> im, const Arrays in, int naxes,
                                                     uint32_t* bits, int words, int ntiles,
                                                     int* counts) {
    begin();
    __shared__ int warp_cnt[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, b = blockIdx.y;
    if (b == naxes) {
        const int64_t v = int64_t(blockIdx.x) * 256 + threadIdx.x;
        if (v < (int64_t(1) << s) * node_parts(dims)) {
            const int j = int(v / node_parts(dims)), part = int(v % node_parts(dims));
            int lo, c;
            node_range(n, s, j, lo, c);
            write_node_part<T>(pts, dims, im, s, j, lo, c, part, [&](int ax, int i) { return P[ax][lo + i]; });
        }
        return;
    }
    const int ax = s % dims;
    const uint32_t* pa = P[ax];
    const uint32_t* pb = in[b];
    int c = 0;
#pragma unroll
    for (int i = 0; i < kTile / 256; ++i) {
        const int word = blockIdx.x * (kTile / 32) + w * (kTile / 256) + i;
        const int64_t p = int64_t(word) * 32 + lane;
        bool left = false;
        if (p < n) {
            const NodeAt a = locate(n, s, int(p));
            const uint32_t id = pb[p], mid = pa[a.lo + (a.c >> 1)];
            // by the sort's keys: exactly h of a node's points go left whatever
            // the values (NaN compares false with everything; with it the
            // places below would run past the node's range)
            const auto v = coord_key(pts[int64_t(id) * dims + ax]), m = coord_key(pts[int64_t(mid) * dims + ax]);
            left = v < m || (v == m && id < mid);
        }
        const unsigned m = __ballot_sync(0xFFFFFFFFu, left);
        if (lane == 0 && word < words) bits[int64_t(b) * words + word] = m;
        c += __popc(m);
    }
    if (lane == 0) warp_cnt[w] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int sum = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) sum += warp_cnt[i];
        counts[int64_t(b) * ntiles + blockIdx.x] = sum;
    }
}

// Stable partition of every node's range by side (lefts first); counts holds
// the tiles' left counts or, `scanned`, their exclusive scan.  Up to
// kCountedTiles tiles a block adds up the counts before its own (a few
// kilobytes from L2, while its own bits arrive), which saves the scan's launch
// (1M points 0.57 -> 0.55 ms).
constexpr int kCountedTiles = 2048;

__global__ void __launch_bounds__(256) k_level_partition(int n, int s, const Arrays in, const Arrays out,
                                                         const uint32_t* bits, int words, int ntiles, bool scanned,
                                                         const int* counts) {
    begin();
    __shared__ int warp_cnt[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, b = blockIdx.y;
    const uint32_t* pb = in[b];
    uint32_t* po = out[b];
    constexpr int WORDS = kTile / 256;
    const int word0 = blockIdx.x * (kTile / 32) + w * WORDS;
    const uint32_t mine = lane < WORDS && word0 + lane < words ? bits[int64_t(b) * words + word0 + lane] : 0u;
    int c = __popc(mine);
    c = __reduce_add_sync(0xFFFFFFFFu, c);
    if (lane == 0) warp_cnt[w] = c;
    int run = 0;
    if (!scanned) {
        __shared__ int before[8];
        int sum = 0;
        for (int i = threadIdx.x; i < int(blockIdx.x); i += 256) sum += counts[int64_t(b) * ntiles + i];
        sum = __reduce_add_sync(0xFFFFFFFFu, sum);
        if (lane == 0) before[w] = sum;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 8; ++i) run += before[i];
    } else {
        __syncthreads();
        run = counts[int64_t(b) * ntiles + blockIdx.x];
    }
    for (int i = 0; i < w; ++i) run += warp_cnt[i];
    const unsigned below = (1u << lane) - 1u;
#pragma unroll
    for (int i = 0; i < WORDS; ++i) {
        const unsigned m = __shfl_sync(0xFFFFFFFFu, mine, i);
        const int64_t p64 = int64_t(word0 + i) * 32 + lane;
        if (p64 < n) {
            const int p = int(p64);
            const NodeAt a = locate(n, s, p);
            const int before = run + __popc(m & below) - a.lefts;  // lefts before p in its node
            const int dst = (m >> lane) & 1 ? a.lo + before : a.lo + (a.c >> 1) + (p - a.lo - before);
            po[dst] = pb[p];
        }
        run += __popc(m);
    }
}

template <typename T>
__global__ void __launch_bounds__(256) k_write_points(const T* __restrict__ pts, int n, int dims,
                                                      const uint32_t* order, const Image<T> im) {
    begin();
    const int64_t p = int64_t(blockIdx.x) * 256 + threadIdx.x;
    if (p < n) write_point<T>(pts, dims, im, p, order[p]);
}

// -------------------------------------------------------------- subtrees --

// One block per node of depth t0 (at most kSub points): all levels below it.
// The node's ids and, per axis, its order as 16-bit places live in shared
// memory; a thread keeps the node range of its kSubItems consecutive places
// in registers.  Two axes' left counts share one block scan (16 bits each).
template <typename T>
__global__ void __launch_bounds__(kSubThreads) k_subtrees(const T* __restrict__ pts, int n, int dims, int t0,
                                                          const Arrays P, const Image<T> im,
                                                          uint16_t* __restrict__ place) {
    begin();
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* ids = reinterpret_cast<uint32_t*>(smem);                    // [kSub]
    uint32_t* start = ids + kSub;                                         // [kSub] scan at each node's start
    uint16_t* arr = reinterpret_cast<uint16_t*>(start + kSub);            // [dims][kSub]
    uint8_t* side = reinterpret_cast<uint8_t*>(arr + dims * kSub);        // [kSub]
    __shared__ int warp_sums[32];
    int glo, cnt;
    node_range(n, t0, blockIdx.x, glo, cnt);
    const int t = threadIdx.x;
    for (int i = t; i < cnt; i += kSubThreads) {
        const uint32_t id = P[0][glo + i];
        ids[i] = id;
        arr[i] = uint16_t(i);
        if (dims > 1) place[id] = uint16_t(i);
    }
    __syncthreads();  // the block's own writes to `place` are visible to all its threads
    for (int a = 1; a < dims; ++a)
        for (int i = t; i < cnt; i += kSubThreads) arr[a * kSub + i] = place[P[a][glo + i]];

    int lo[kSubItems], c[kSubItems], j[kSubItems];
#pragma unroll
    for (int e = 0; e < kSubItems; ++e) {
        lo[e] = 0;
        c[e] = cnt;
        j[e] = 0;
    }
    __syncthreads();
    for (int s = t0;; ++s) {
        const int entries = node_parts(dims) << (s - t0);
        for (int v = t; v < entries; v += kSubThreads) {
            const int nj = v / node_parts(dims), part = v % node_parts(dims);
            int nlo, nc;
            node_range(cnt, s - t0, nj, nlo, nc);
            write_node_part<T>(pts, dims, im, s, (int(blockIdx.x) << (s - t0)) + nj, glo + nlo, nc, part,
                               [&](int ax, int i) { return ids[arr[ax * kSub + nlo + i]]; });
        }
        if (s == im.levels) break;
        const int ax = s % dims;
#pragma unroll
        for (int e = 0; e < kSubItems; ++e) {
            const int p = t * kSubItems + e;
            if (p < cnt) side[arr[ax * kSub + p]] = uint8_t(p - lo[e] >= (c[e] >> 1));
        }
        __syncthreads();
        for (int o = 1; o < dims; o += 2) {
            // the next two axes after the split axis (cyclically); the second may not exist
            const int b0 = (ax + o) % dims, b1 = (ax + o + 1) % dims;
            const bool two = o + 1 < dims;
            uint16_t v0[kSubItems], v1[kSubItems];
            uint32_t f[kSubItems], sum = 0;
#pragma unroll
            for (int e = 0; e < kSubItems; ++e) {
                const int p = t * kSubItems + e;
                v0[e] = v1[e] = 0;
                f[e] = 0;
                if (p < cnt) {
                    v0[e] = arr[b0 * kSub + p];
                    f[e] = side[v0[e]] ^ 1u;
                    if (two) {
                        v1[e] = arr[b1 * kSub + p];
                        f[e] |= uint32_t(side[v1[e]] ^ 1u) << 16;
                    }
                }
                sum += f[e];
            }
            uint32_t run = uint32_t(block_exclusive(int(sum), warp_sums));
            uint32_t ex[kSubItems];
#pragma unroll
            for (int e = 0; e < kSubItems; ++e) {
                const int p = t * kSubItems + e;
                ex[e] = run;
                if (p < cnt && p == lo[e]) start[j[e]] = run;
                run += f[e];
            }
            __syncthreads();
#pragma unroll
            for (int e = 0; e < kSubItems; ++e) {
                const int p = t * kSubItems + e;
                if (p < cnt) {
                    const uint32_t d = ex[e] - start[j[e]];  // both halves: lefts before p in its node
                    const int h = c[e] >> 1, d0 = int(d & 0xFFFFu), d1 = int(d >> 16);
                    arr[b0 * kSub + ((f[e] & 1u) ? lo[e] + d0 : lo[e] + h + (p - lo[e] - d0))] = v0[e];
                    if (two) arr[b1 * kSub + ((f[e] >> 16) ? lo[e] + d1 : lo[e] + h + (p - lo[e] - d1))] = v1[e];
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int e = 0; e < kSubItems; ++e) {
            const int p = t * kSubItems + e, h = c[e] >> 1;
            j[e] *= 2;
            if (p - lo[e] >= h) {
                lo[e] += h;
                c[e] -= h;
                j[e] += 1;
            } else {
                c[e] = h;
            }
        }
    }
    // points in leaf order: the leaf parent's axis (left as it was by the last partition)
    const int fa = (im.levels - 1) % dims;
    for (int i = t; i < cnt; i += kSubThreads) write_point<T>(pts, dims, im, glo + i, ids[arr[fa * kSub + i]]);
}

// ---------------------------------------------------------- float filter --

// Centre and scale of the cloud from its root box; a cloud with infinite
// coordinates keeps its own.
__device__ __forceinline__ Frame cloud_frame(const PointRec<double>* boxes) {
    const PointRec<double> lo = boxes[0], hi = boxes[1];
    const double l[3] = {lo.x, lo.y, lo.z}, h[3] = {hi.x, hi.y, hi.z};
    Frame f;
    double extent = 0.0;
    for (int c = 0; c < 3; ++c) {
        f.centre[c] = l[c] + 0.5 * (h[c] - l[c]);
        if (!(fabs(f.centre[c]) <= 1.7e308)) f.centre[c] = 0.0;
        extent = fmax(extent, h[c] - l[c]);
    }
    int e = 0;
    if (extent > 0.0 && extent <= 1.7e308) e = -ilogb(extent);
    f.scale = ldexp(1.0, max(-400, min(400, e)));
    return f;
}

// Float images of points, boxes (rounded outwards) and split values.
__global__ void __launch_bounds__(256) k_fill_filter(const PointRec<double>* pts, int64_t n,
                                                     const PointRec<double>* boxes, int64_t nodes,
                                                     const double* medians, int64_t splits, int dims,
                                                     PointRec<float>* __restrict__ f_pts,
                                                     PointRec<float>* __restrict__ f_boxes,
                                                     float* __restrict__ f_medians, Frame* __restrict__ frame) {
    begin();
    __shared__ Frame f;
    if (threadIdx.x == 0) f = cloud_frame(boxes);
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) *frame = f;
    const int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x;
    if (i < n) {
        const PointRec<double> p = pts[i];
        f_pts[i] = PointRec<float>{__double2float_rn((p.x - f.centre[0]) * f.scale),
                                   __double2float_rn((p.y - f.centre[1]) * f.scale),
                                   __double2float_rn((p.z - f.centre[2]) * f.scale), 0.f};
    }
    if (i < nodes) {
        const PointRec<double> lo = boxes[2 * i], hi = boxes[2 * i + 1];
        f_boxes[2 * i] = PointRec<float>{__double2float_rd(frame_down(lo.x, f.centre[0], f.scale)),
                                         __double2float_rd(frame_down(lo.y, f.centre[1], f.scale)),
                                         __double2float_rd(frame_down(lo.z, f.centre[2], f.scale)),
                                         __uint_as_float(rec_index(lo))};
        f_boxes[2 * i + 1] = PointRec<float>{__double2float_ru(frame_up(hi.x, f.centre[0], f.scale)),
                                             __double2float_ru(frame_up(hi.y, f.centre[1], f.scale)),
                                             __double2float_ru(frame_up(hi.z, f.centre[2], f.scale)),
                                             __uint_as_float(rec_index(hi))};
    }
    if (i < splits) {
        const int ax = (31 - __clz(int(i) + 1)) % dims;
        f_medians[i] = __double2float_rn((medians[i] - f.centre[ax]) * f.scale);
    }
}

size_t subtree_smem(int dims) { return size_t(kSub) * (4 + 4 + 2 * dims + 1); }

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

// Axes sorted (and partitioned) in one launch: all of them up to 32M points,
// above that one after the other, with the scratch of one.
int axes_at_once(int64_t n, int dims) { return n <= (int64_t(32) << 20) ? dims : 1; }

// Scratch of a build: id orders (one per axis), then spare orders, two key
// arrays (whose space the level passes use afterwards), digit histograms.
struct BuildWs {
    size_t orders = 0, key_a = 0, key_b = 0, hist = 0, totals = 0, odd = 0, total = 0;
    size_t order_bytes = 0;
    int at_once = 1;
};
BuildWs build_ws(int64_t n, int dims, size_t key_bytes) {
    BuildWs w;
    const bool small = n <= kSub;
    const int A = w.at_once = axes_at_once(n, dims);
    w.order_bytes = align256(4 * size_t(n));
    size_t o = 0;
    w.odd = o;
    o += 256;
    w.orders = o;
    o += w.order_bytes * (small ? dims : dims + A);
    w.key_b = o;  // small clouds: the places of k_subtrees only
    o += small ? align256(2 * size_t(n)) : align256(key_bytes * size_t(n) * A);
    if (!small) {
        w.key_a = o;
        o += align256(key_bytes * size_t(n) * A);
        const size_t tile = key_bytes == 4 ? radix_tile<float>() : radix_tile<double>();
        const size_t ntiles = (size_t(n) + tile - 1) / tile;
        w.hist = o;  // the level passes' tile counts use it too
        o += align256(sizeof(int) * 256 * ntiles * A);
        w.totals = o;
        o += align256(sizeof(int) * 256 * A);
    }
    w.total = o;
    return w;
}

#define TK_TRY(expr)                                                                          \
    do {                                                                                      \
        cudaError_t e_ = (expr);                                                              \
        if (e_ != cudaSuccess) return fail(TK_ECUDA, std::string("device build: ") + cudaGetErrorString(e_)); \
    } while (0)

}  // namespace

size_t build_workspace_bytes(int64_t n, int dims, int dtype) {
    return build_ws(n, dims, dtype == TK_F32 ? 4 : 8).total;
}

TreeImage tree_image(int64_t n, int dims, int dtype, int levels) {
    TreeImage im;
    const size_t es = dtype == TK_F32 ? 4 : 8;
    const size_t nleaves = size_t(1) << levels;
    const bool wide = dims > 3;
    const size_t row = es * (wide ? record_width(dims) : 4);
    size_t o = 0;
    im.pts = o;
    o += align256(row * size_t(n));
    im.boxes = o;
    o += align256(row * 2 * (2 * nleaves - 1));
    im.medians = o;
    o += align256(es * nleaves);
    im.leaf_off = o;
    o += align256(sizeof(int32_t) * (nleaves + 1));
    im.perm = o;
    if (wide) o += align256(sizeof(int32_t) * size_t(n));
    if (!wide && dtype == TK_F64) {
        im.f_pts = o;
        o += align256(sizeof(PointRec<float>) * size_t(n));
        im.f_boxes = o;
        o += align256(sizeof(PointRec<float>) * 2 * (2 * nleaves - 1));
        im.f_medians = o;
        o += align256(sizeof(float) * nleaves);
        im.f_frame = o;
        o += align256(sizeof(Frame));
    }
    im.total = o;
    return im;
}

template <typename T>
int enqueue_device_tree(const T* pts, int64_t n, int dims, void* stream, const tk_tree* t, void* workspace,
                        const int** odd_out) {
    using K = typename KeyBits<T>::type;
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int L = t->search_levels;
    const BuildWs w = build_ws(n, dims, sizeof(K));
    char* ws = static_cast<char*>(workspace);
    int* odd = reinterpret_cast<int*>(ws + w.odd);
    *odd_out = odd;
    Arrays P, spare;  // P's arrays, then the spares
    P.base = spare.base = reinterpret_cast<uint32_t*>(ws + w.orders);
    P.stride = spare.stride = int64_t(w.order_bytes / 4);
    const int A = w.at_once;
    for (int a = 0; a < dims; ++a) P.set(a, a);
    for (int a = 0; a < A; ++a) spare.set(a, dims + a);
    const int n32 = int(n);

    Image<T> im;
    im.pts = static_cast<T*>(t->d_pts);
    im.perm = t->d_perm;
    im.medians = static_cast<T*>(t->d_medians);
    im.leaf_off = t->d_leaf_off;
    im.boxes = static_cast<T*>(t->d_boxes);
    im.levels = L;
    im.W = record_width(dims);

    // 1. presorted axes
    TK_TRY(cudaMemsetAsync(odd, 0, 2 * sizeof(int), s));
    int t0 = 0;  // depth from which a block finishes a node
    if (n <= kSub) {
        const size_t smem = small_sort_smem<T>();
        TK_TRY(cudaFuncSetAttribute(k_small_sort<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        k_small_sort<T><<<dims, kSubThreads, smem, s>>>(pts, n32, dims, P, odd);
        TK_TRY(cudaGetLastError());
    } else {
        while (t0 < L && ((n - 1) >> t0) + 1 > kSub) ++t0;
        K* key_a = reinterpret_cast<K*>(ws + w.key_a);
        K* key_b = reinterpret_cast<K*>(ws + w.key_b);
        int* hist = reinterpret_cast<int*>(ws + w.hist);
        const int rtiles = int((n + radix_tile<T>() - 1) / radix_tile<T>());
        int* totals = rtiles > kOwnScanTiles ? reinterpret_cast<int*>(ws + w.totals) : nullptr;
        const int passes = int(sizeof(K));
        for (int a0 = 0; a0 < dims; a0 += A) {
            const int na = std::min(A, dims - a0);
            const dim3 grid(rtiles, na);
            Arrays dst = P;
            for (int a = 0; a < na; ++a) dst.set(a, P.slot(a0 + a));
            for (int pass = 0; pass < passes; ++pass) {
                const K* kin = pass & 1 ? key_a : key_b;  // pass 0 reads the points
                K* kout = pass & 1 ? key_b : key_a;
                const Arrays& vin = pass & 1 ? spare : dst;
                const Arrays& vout = pass & 1 ? dst : spare;  // an even number of passes ends in dst
                const int shift = 8 * pass;
                if (pass == 0) TK_TRY(launch(a0 > 0, k_radix_hist<T, true>, grid, kSortThreads, 0, s, pts, n, dims, a0, kin, shift, rtiles, hist, odd));
                else TK_TRY(launch(true, k_radix_hist<T, false>, grid, kSortThreads, 0, s, pts, n, dims, a0, kin, shift, rtiles, hist, odd));
                if (totals) TK_TRY(launch(true, k_row_scan, dim3(256, na), kScanThreads, 0, s, hist, rtiles, totals));
                if (pass == 0) TK_TRY(launch(true, k_radix_scatter<T, true, false>, grid, kSortThreads, 0, s, pts, n, dims, a0, kin, vin, shift, rtiles, hist, totals, kout, vout));
                else if (pass + 1 < passes) TK_TRY(launch(true, k_radix_scatter<T, false, false>, grid, kSortThreads, 0, s, pts, n, dims, a0, kin, vin, shift, rtiles, hist, totals, kout, vout));
                else TK_TRY(launch(true, k_radix_scatter<T, false, true>, grid, kSortThreads, 0, s, pts, n, dims, a0, kin, vin, shift, rtiles, hist, totals, kout, vout));
                TK_TRY(cudaGetLastError());
            }
        }
    }

    // 2. levels whose nodes exceed a block's capacity
    const int ntiles = int((n + kTile - 1) / kTile);
    if (t0 > 0) {
        uint32_t* bits = reinterpret_cast<uint32_t*>(ws + w.key_a);  // the keys' space
        int* counts = reinterpret_cast<int*>(ws + w.hist);
        int* totals = reinterpret_cast<int*>(ws + w.totals);
        const int words = int((n + 31) / 32);
        for (int lev = 0; lev < t0; ++lev) {
            int axes[kMaxDims], na = 0;
            for (int b = 0; b < dims; ++b)
                if (b != lev % dims) axes[na++] = b;
            int g = 0;
            do {
                const int m = std::min(A, na - g);
                Arrays in = P;
                const Arrays out = spare;
                for (int i = 0; i < m; ++i) in.set(i, P.slot(axes[g + i]));
                // the nodes' entries need every axis's order as it was before this level: with the first group
                TK_TRY(launch(true, k_level_count<T>, dim3(ntiles, m + (g == 0)), 256, 0, s, pts, n32, dims, lev, P, im, in, m, bits, words, ntiles, counts));
                if (m > 0) {
                    const bool scan = ntiles > kCountedTiles;
                    if (scan) TK_TRY(launch(true, k_row_scan, dim3(1, m), kScanThreads, 0, s, counts, ntiles, totals));
                    TK_TRY(launch(true, k_level_partition, dim3(ntiles, m), 256, 0, s, n32, lev, in, out, bits, words, ntiles, scan, counts));
                }
                for (int i = 0; i < m; ++i) {
                    P.set(axes[g + i], out.slot(i));
                    spare.set(i, in.slot(i));
                }
                g += A;
            } while (g < na);
            TK_TRY(cudaGetLastError());
        }
    }

    // 3. the rest, a block per node
    if (n > kSub && ((n - 1) >> t0) + 1 > kSub) {  // leaves larger than a block's capacity
        TK_TRY(launch(true, k_level_count<T>, dim3(ntiles, 1), 256, 0, s, pts, n32, dims, L, P, im, P, 0, nullptr, 0, ntiles, nullptr));
        TK_TRY(launch(true, k_write_points<T>, dim3(unsigned((n + 255) / 256)), 256, 0, s, pts, n32, dims, P[(L - 1) % dims], im));
    } else {
        const size_t smem = subtree_smem(dims);
        TK_TRY(cudaFuncSetAttribute(k_subtrees<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        TK_TRY(launch(true, k_subtrees<T>, dim3(1u << t0), kSubThreads, smem, s, pts, n32, dims, t0, P, im,
                      reinterpret_cast<uint16_t*>(ws + w.key_b)));
    }
    TK_TRY(cudaGetLastError());
    if constexpr (sizeof(T) == 8) {
        if (t->d_filter[0]) {
            const int64_t nodes = (int64_t(2) << L) - 1, splits = (int64_t(1) << L) - 1;
            const int64_t work = std::max(n, nodes);
            TK_TRY(launch(true, k_fill_filter, dim3(unsigned((work + 255) / 256)), 256, 0, s,
                static_cast<const PointRec<double>*>(t->d_pts), n, static_cast<const PointRec<double>*>(t->d_boxes), nodes,
                static_cast<const double*>(t->d_medians), splits, dims,
                static_cast<PointRec<float>*>(const_cast<void*>(t->d_filter[0])),
                static_cast<PointRec<float>*>(const_cast<void*>(t->d_filter[1])),
                static_cast<float*>(const_cast<void*>(t->d_filter[2])),
                static_cast<Frame*>(const_cast<void*>(t->d_filter[3]))));
            TK_TRY(cudaGetLastError());
        }
    }
    return TK_OK;
}

template <typename T>
int build_device_tree(const T* pts, int64_t n, int dims, void* stream, tk_tree* t, void* workspace) {
    const cudaStream_t s = static_cast<cudaStream_t>(stream);
    const int* odd = nullptr;
    const int rc = enqueue_device_tree<T>(pts, n, dims, stream, t, workspace, &odd);
    if (rc != TK_OK) return rc;
    int nan_host = 0;
    TK_TRY(cudaMemcpyAsync(&nan_host, odd, sizeof(int), cudaMemcpyDeviceToHost, s));
    TK_TRY(cudaStreamSynchronize(s));
    if (nan_host) return fail(TK_EINVAL, "reference points contain NaN");
    return TK_OK;
}

template int enqueue_device_tree<float>(const float*, int64_t, int, void*, const tk_tree*, void*, const int**);
template int enqueue_device_tree<double>(const double*, int64_t, int, void*, const tk_tree*, void*, const int**);
template int build_device_tree<float>(const float*, int64_t, int, void*, tk_tree*, void*);
template int build_device_tree<double>(const double*, int64_t, int, void*, tk_tree*, void*);

}  // namespace tk
