// Exhaustive ("brute force") exact KNN: the nn_distance op.
//
// The reference's kernel (NmDistanceKernelDynamic, src/nndistance_g.cu:74-140)
// runs as ONE block for the whole problem, hard-codes d = 3 and keeps each
// thread's top-k list in a global scratch array.  Here:
//   * a block owns a tile of queries (one query per group of G lanes) and one
//     slice of the reference cloud; the grid is queries x slices so every SM
//     is busy even for few queries;
//   * reference points stream through shared memory in tiles, zero-padded to
//     DP dimensions (padding adds exact zeros, so distances are unchanged);
//   * distances use the reference's CPU arithmetic (sqdist order, no fused
//     multiply-add), so results match the KD-tree query bit for bit;
//   * each slice keeps the k best (distance, index) keys in registers (TopK);
//     with several slices a merge kernel combines the per-slice lists;
//   * with one lane per query a candidate is first tested as a float against
//     the list's worst distance (one compare), and only the rare survivors
//     build and compare the 64-bit (distance, index) key.
#pragma once

#include <cuda_runtime.h>

#include "tk_device.cuh"
#include "tk_internal.h"

namespace tk {

template <typename T>
struct BruteArgs {
    const T* ref;   // [n, d]
    const T* q;     // [nq, d]
    int n, nq, d, k;
    int nsplit;     // reference slices (gridDim.y)
    T* out_d;       // [nq, k]   (nsplit == 1)
    int32_t* out_i; // [nq, k]
    Key<T>* part;   // [nq, nsplit, k] per-slice lists (nsplit > 1)
    // Optional gather: when qlist is set, the queries are qlist[0..*qcount)
    // and results go to their rows (the caller merges the slices).
    const int* qlist = nullptr;
    const int* qcount = nullptr;
    const int* gate = nullptr;  // do nothing while *gate is 0
    int qmore = 0;  // a list of at most this many queries is not served here
};

// Slices of a listed search, at most `most`: as many as the launched blocks
// can search at one (query tile, slice) pair each; with one, its lists go
// straight to the outputs.
__host__ __device__ __forceinline__ int list_slices(int count, int blocks, int per_tile, int most) {
    const int s = blocks / ((count + per_tile - 1) / per_tile);
    return s < 1 ? 1 : (s > most ? most : s);
}

// Reference rows per shared-memory tile: 32 KiB of coordinates, 32 to 256 rows.
template <typename T, int DP>
struct BruteTile {
    static constexpr int kElems = 32768 / int(sizeof(T));
    static constexpr int kRefs = (kElems / DP) > 256 ? 256 : ((kElems / DP) < 32 ? 32 : (kElems / DP));
};

template <typename T, int DP>
__device__ __forceinline__ T sqdist_padded(const T (&q)[DP], const T* r) {
    T d0 = sub_rn(q[0], r[0]);
    T acc = mul_rn(d0, d0);
#pragma unroll
    for (int c = 1; c < DP; ++c) {
        const T dc = sub_rn(q[c], r[c]);
        acc = add_rn(acc, mul_rn(dc, dc));
    }
    return acc;
}

// A block's share: query tile, slice, and how many there are of queries and
// slices.  Of a list only the device knows; it is kept in shared memory (`at`)
// and read again after the search, where its registers cost up to a seventh
// (262,144 x 65,536, all listed, d = 32, k = 32: 79 -> 69 ms).
struct BrutePlace {
    int live, nsplit, qtile, slice;
};
template <typename T, bool LIST>
__device__ __forceinline__ BrutePlace brute_place(const BruteArgs<T>& a, const volatile int* at) {
    if constexpr (LIST) return BrutePlace{at[0], at[1], at[2], at[3]};
    else return BrutePlace{a.nq, a.nsplit, int(blockIdx.x), int(blockIdx.y)};
}

// One query tile against one slice (LIST: of the listed queries).
template <typename T, int DP, int G, int R, bool LIST>
__device__ __forceinline__ void brute_block(const BruteArgs<T>& a, T* tile, const volatile int* at) {
    constexpr int TR = BruteTile<T, DP>::kRefs;
    const int lane = threadIdx.x & 31;
    const int gl = lane & (G - 1);
    const int gbase = lane & ~(G - 1);
    const unsigned gmask = group_mask<G>(lane);
    const BrutePlace b = brute_place<T, LIST>(a, at);
    const int slot = b.qtile * (blockDim.x / G) + threadIdx.x / G;
    const bool active = slot < b.live;
    const int qi = active ? (LIST ? a.qlist[slot] : slot) : 0;

    T q[DP];
#pragma unroll
    for (int c = 0; c < DP; ++c) q[c] = (active && c < a.d) ? a.q[(long long)qi * a.d + c] : T(0);

    TopK<T, G, R> list;
    list.init(a.k, gl);
    Key<T> worst = Key<T>::sentinel();

    const long long per = ((long long)a.n + b.nsplit - 1) / b.nsplit;
    const int r0 = int(min((long long)a.n, per * b.slice));
    const int r1 = int(min((long long)a.n, per * (b.slice + 1)));
    for (int t0 = r0; t0 < r1; t0 += TR) {
        const int len = min(TR, r1 - t0);
        __syncthreads();
        for (int e = threadIdx.x; e < TR * DP; e += blockDim.x) {
            const int j = e / DP, c = e - j * DP;
            tile[e] = (j < len && c < a.d) ? a.ref[(long long)(t0 + j) * a.d + c] : T(0);
        }
        __syncthreads();
        if constexpr (G == 1 && DP % 4 == 0 && sizeof(T) == 4) {
            // One lane per query: every lane reads the same reference row, so
            // a 16-byte shared load broadcasts four coordinates to the warp;
            // four references per step give four independent chains.  Same
            // accumulation order as sqdist (dimension by dimension).
            constexpr int U = 4;
            static_assert(TR % U == 0, "tile rows must be a multiple of the step");
            // two steps at once where the list is one key (k = 1, 20,000 x 2,000,
            // d = 8 0.155 -> 0.125 ms; with more keys 2% slower to 20%)
            constexpr int kSteps = R == 1 ? 2 : 1;
            if (active) {
                const float4* rows = reinterpret_cast<const float4*>(tile);
#pragma unroll kSteps
                for (int j0 = 0; j0 < len; j0 += U) {
                    T acc[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const float4 v = rows[(j0 + u) * (DP / 4)];
                        const T d0 = sub_rn(q[0], v.x), d1 = sub_rn(q[1], v.y);
                        const T d2 = sub_rn(q[2], v.z), d3 = sub_rn(q[3], v.w);
                        acc[u] = mul_rn(d0, d0);
                        acc[u] = add_rn(acc[u], mul_rn(d1, d1));
                        acc[u] = add_rn(acc[u], mul_rn(d2, d2));
                        acc[u] = add_rn(acc[u], mul_rn(d3, d3));
                    }
#pragma unroll
                    for (int c4 = 1; c4 < DP / 4; ++c4) {
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const float4 v = rows[(j0 + u) * (DP / 4) + c4];
                            const T d0 = sub_rn(q[4 * c4], v.x), d1 = sub_rn(q[4 * c4 + 1], v.y);
                            const T d2 = sub_rn(q[4 * c4 + 2], v.z), d3 = sub_rn(q[4 * c4 + 3], v.w);
                            acc[u] = add_rn(acc[u], mul_rn(d0, d0));
                            acc[u] = add_rn(acc[u], mul_rn(d1, d1));
                            acc[u] = add_rn(acc[u], mul_rn(d2, d2));
                            acc[u] = add_rn(acc[u], mul_rn(d3, d3));
                        }
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        if (j0 + u < len && acc[u] <= worst.dist())
                            worst = offer<T, G, R>(list, Key<T>::make(acc[u], uint32_t(t0 + j0 + u)), worst, gmask,
                                                   gl, gbase);
                    }
                }
            }
        } else if (active) {
            // four references per lane step: four independent accumulation chains
            constexpr int U = DP <= 4 ? 1 : ((DP > 32 || R >= 16) ? 2 : 4);
            for (int j0 = 0; j0 < len; j0 += G * U) {
                T acc[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int j = min(j0 + u * G + gl, TR - 1);  // rows past len are padding zeros
                    const T* r = tile + j * DP;
                    const T d0 = sub_rn(q[0], r[0]);
                    acc[u] = mul_rn(d0, d0);
                }
#pragma unroll
                for (int c = 1; c < DP; ++c) {
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const int j = min(j0 + u * G + gl, TR - 1);
                        const T dc = sub_rn(q[c], tile[j * DP + c]);
                        acc[u] = add_rn(acc[u], mul_rn(dc, dc));
                    }
                }
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int j = j0 + u * G + gl;
                    if constexpr (G == 1) {
                        if (j < len && acc[u] <= worst.dist())
                            worst = offer<T, G, R>(list, Key<T>::make(acc[u], uint32_t(t0 + j)), worst, gmask, gl,
                                                   gbase);
                    } else {
                        Key<T> mine = Key<T>::sentinel();
                        if (j < len) mine = Key<T>::make(acc[u], uint32_t(t0 + j));
                        worst = offer<T, G, R>(list, mine, worst, gmask, gl, gbase);
                    }
                }
            }
        }
    }
    const BrutePlace e = brute_place<T, LIST>(a, at);
    const int row = e.qtile * (blockDim.x / G) + threadIdx.x / G;
    if (row >= e.live) return;
    if (e.nsplit == 1) {
        list.store(a.k, gl, a.out_d, a.out_i, LIST ? a.qlist[row] : row);
    } else {
        Key<T>* dst = a.part + ((long long)row * e.nsplit + e.slice) * a.k;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int s = r * G + gl;
            const int o = s - (G * R - a.k);
            if (o >= 0) dst[o] = list.slot[r];
        }
    }
}

template <typename T, int DP, int G, int R>
__global__ void __launch_bounds__(256) k_brute(const BruteArgs<T> a) {
    __shared__ __align__(16) T tile[BruteTile<T, DP>::kRefs * DP];
    if (a.gate && *a.gate == 0) return;
    brute_block<T, DP, G, R, false>(a, tile, nullptr);
}

// The queries of a list: a block per (query tile, slice) pair, the rest exit.
// (Blocks that looped over the pairs took 1.4 to 1.9 times as long.)
template <typename T, int DP, int G, int R>
__global__ void __launch_bounds__(256) k_brute_list(const BruteArgs<T> a) {
    __shared__ __align__(16) T tile[BruteTile<T, DP>::kRefs * DP];
    __shared__ int at[4];
    const int live = *a.qcount;
    if (live <= a.qmore) return;
    const int per_tile = blockDim.x / G, qtiles = (live + per_tile - 1) / per_tile;
    const int nsplit = list_slices(live, gridDim.x, per_tile, a.nsplit);
    if (int(blockIdx.x) >= qtiles * nsplit) return;
    if (threadIdx.x == 0) {
        at[0] = live;
        at[1] = nsplit;
        at[2] = int(blockIdx.x) % qtiles;
        at[3] = int(blockIdx.x) / qtiles;
    }
    __syncthreads();
    brute_block<T, DP, G, R, true>(a, tile, at);
}

// Combine the per-slice lists of every query (group of G lanes per query).
template <typename T, int G, int R>
__global__ void __launch_bounds__(256) k_brute_merge(const BruteArgs<T> a) {
    const int lane = threadIdx.x & 31;
    const int gl = lane & (G - 1);
    const int gbase = lane & ~(G - 1);
    const unsigned gmask = group_mask<G>(lane);
    const int slot = blockIdx.x * (blockDim.x / G) + threadIdx.x / G;
    if (slot >= a.nq || (a.gate && *a.gate == 0)) return;  // whole groups leave together
    TopK<T, G, R> list;
    list.init(a.k, gl);
    Key<T> worst = Key<T>::sentinel();
    const Key<T>* src = a.part + (long long)slot * a.nsplit * a.k;
    const int total = a.nsplit * a.k;
    for (int e0 = 0; e0 < total; e0 += G) {
        const int e = e0 + gl;
        const Key<T> mine = e < total ? src[e] : Key<T>::sentinel();
        worst = offer<T, G, R>(list, mine, worst, gmask, gl, gbase);
    }
    list.store(a.k, gl, a.out_d, a.out_i, slot);
}

// Exact search for the queries listed on the device (qlist[0..*qcount)),
// results written to their rows of dists / idx (brute.cu).
size_t brute_fallback_workspace_bytes(int64_t n, int64_t nq, int d, int k);
int brute_fallback(const float* ref, int64_t n, const float* q, int64_t nq, int d, int k, float* dists,
                   int32_t* idx, const int* qlist, const int* qcount, void* ws, size_t ws_bytes, cudaStream_t s);

// Launch shape of an exhaustive search (brute.cu: plan_brute).
struct BrutePlan {
    int DP, G, R, nsplit, qtiles;
    int list_blocks = 0;  // blocks of a search of listed queries
};

template <typename T, int DP>
int launch_dp(const BruteArgs<T>& a, const BrutePlan& p, cudaStream_t s) {
    dim3 grid(p.qtiles, p.nsplit);
    bool done = false;
#define TK_BR(g, r)                                                          \
    if (!done && p.G == g && p.R == r) {                                     \
        if (p.list_blocks) {                                                 \
            if constexpr (sizeof(T) == 4) k_brute_list<T, DP, g, r><<<p.list_blocks, 256, 0, s>>>(a); \
        } else {                                                             \
            k_brute<T, DP, g, r><<<grid, 256, 0, s>>>(a);                    \
            if (p.nsplit > 1) k_brute_merge<T, g, r><<<p.qtiles, 256, 0, s>>>(a); \
        }                                                                    \
        done = true;                                                         \
    }
    TK_BR(1, 1) TK_BR(1, 4) TK_BR(1, 16) TK_BR(2, 16) TK_BR(4, 16) TK_BR(8, 16)
    if constexpr (sizeof(T) == 4 && DP % 4 == 0 && DP <= 32) {
        TK_BR(1, 32)
    }
#undef TK_BR
    if (!done) return fail(TK_EUNSUPPORTED, "no brute-force kernel for this k");
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(TK_ECUDA, std::string("brute-force launch: ") + cudaGetErrorString(e));
    return TK_OK;
}

// float64 searches of 5 to 128 dimensions (brute_f64.cu, a unit of its own).
int launch_brute_f64_wide(const BruteArgs<double>& a, const BrutePlan& p, cudaStream_t s);

}  // namespace tk
