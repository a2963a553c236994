// nn_distance: exhaustive exact KNN on CUDA cores (see brute.cuh), plus the
// C entry points for every brute-force mode.
#include <algorithm>
#include <mutex>
#include <string>
#include <vector>

#include "brute.cuh"
#include "brute_tc.cuh"
#include "kd_warp.cuh"

namespace tk {
namespace {

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

int pow2_ceil(int v) {
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

int sm_count_dev() {
    static std::mutex mu;
    static std::vector<int> cache;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if ((int)cache.size() <= dev) cache.resize(dev + 1, 0);
    if (!cache[dev]) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 1;
        cache[dev] = v;
    }
    return cache[dev];
}

// padded dimension for d
int padded_dims(int d) {
    if (d <= 4) return d;
    if (d <= 8) return 8;
    if (d <= 16) return 16;
    if (d <= 32) return 32;
    if (d <= 64) return 64;
    return 128;
}

BrutePlan plan_brute(int64_t n, int64_t nq, int d, int k, bool f32) {
    BrutePlan p;
    p.DP = padded_dims(d);
    // long lists of narrow points: padded to 4 they fit the path below
    // (262,144 x 65,536, d=3, k=32: 131 ms on two lanes per query, 24 ms)
    if (f32 && d < 4 && k > 16 && k <= 32) p.DP = 4;
    if (f32 && p.DP % 4 == 0 && p.DP <= 32 && k <= 32) {
        // one lane per query with broadcast 16-byte row loads (brute.cuh)
        p.G = 1;
        p.R = k <= 1 ? 1 : (k <= 4 ? 4 : (k <= 16 ? 16 : 32));
    } else {
        p.G = std::max(1, pow2_ceil((k + 15) / 16));
        p.R = pow2_ceil((k + p.G - 1) / p.G);
        if (p.G == 1) p.R = p.R <= 1 ? 1 : (p.R <= 4 ? 4 : 16);
    }
    const int per_block = 256 / p.G;
    p.qtiles = int((nq + per_block - 1) / per_block);
    const int target = 8 * sm_count_dev();
    int ns = std::max(1, (target + p.qtiles - 1) / std::max(1, p.qtiles));
    ns = int(std::min<int64_t>(ns, std::max<int64_t>(1, n / 2048)));
    p.nsplit = ns;
    return p;
}

template <typename T>
size_t brute_ws_bytes(const BrutePlan& p, int64_t nq, int k) {
    if (p.nsplit <= 1) return 256;
    return align256(sizeof(Key<T>) * size_t(nq) * p.nsplit * k);
}

template <typename T>
int launch_brute(const BruteArgs<T>& a, const BrutePlan& p, cudaStream_t s) {
    switch (p.DP) {
        case 1: return launch_dp<T, 1>(a, p, s);
        case 2: return launch_dp<T, 2>(a, p, s);
        case 3: return launch_dp<T, 3>(a, p, s);
        case 4: return launch_dp<T, 4>(a, p, s);
        default: break;
    }
    if constexpr (sizeof(T) == 4) {
        switch (p.DP) {
            case 8: return launch_dp<T, 8>(a, p, s);
            case 16: return launch_dp<T, 16>(a, p, s);
            case 32: return launch_dp<T, 32>(a, p, s);
            case 64: return launch_dp<T, 64>(a, p, s);
            case 128: return launch_dp<T, 128>(a, p, s);
            default: break;
        }
    } else {
        return launch_brute_f64_wide(a, p, s);  // brute_f64.cu: d = 5 .. 128
    }
    return fail(TK_EUNSUPPORTED, "no brute-force kernel for this dimension");
}

template <typename T>
int run_brute(const T* ref, int64_t n, const T* q, int64_t nq, int d, int k, T* dists, int32_t* idx, void* ws,
              size_t ws_bytes, cudaStream_t s, const int* gate = nullptr) {
    const BrutePlan p = plan_brute(n, nq, d, k, sizeof(T) == 4);
    if (ws_bytes < brute_ws_bytes<T>(p, nq, k) || (p.nsplit > 1 && !ws))
        return fail(TK_EWORKSPACE, "workspace too small");
    BruteArgs<T> a;
    a.ref = ref;
    a.q = q;
    a.n = int(n);
    a.nq = int(nq);
    a.d = d;
    a.k = k;
    a.nsplit = p.nsplit;
    a.out_d = dists;
    a.out_i = idx;
    a.part = static_cast<Key<T>*>(ws);
    a.gate = gate;
    return launch_brute<T>(a, p, s);
}

// Route of a call that only wants the exact answer (TK_BRUTE_ROUTED).
enum class Route { kCudaCores, kTensorCores, kTree };

// Queries per pass over the tensor cores: bounds the workspace (4.6 KB of hit
// lists per query and slice).
constexpr int64_t kRoutePass = 262144;
constexpr size_t kRouteBytes = size_t(4) << 30;

// Up to three dimensions a tree that is built for the call pays from the
// pairs on at which the comparisons cost more than its build (ms, exhaustive /
// tree: 65,536 x 65,536, d=3, k=1 1.87 / 0.29; 20,000 x 20,000 k=1 0.22 / 0.21,
// k=4 0.33 / 0.23, k=16 1.24 / 0.26; 65,536 x 2,000 k=4 0.18 / 0.23; float64
// 10,000 x 10,000 3.4 / 0.28).  Otherwise the tensor-core search (BF16 hi/lo:
// an error bound 60 times smaller than TF32's leaves hardly any query without
// a certificate) beats the CUDA cores wherever it applies but for the smallest
// calls, whose launches cost more than the work (ms, CUDA cores / tensor
// cores: 262,144 x 65,536, k=32, d=32 69 / 4.7, d=8 30 / 3.8; 20,000 x 20,000,
// d=8, k=1 0.44 / 0.45, k=8 1.02 / 0.45; 1,000 x 128, d=8, k=1 0.06 / 0.07,
// k=8 0.11 / 0.07, d=32, k=8 0.17 / 0.07; d=3, k=4 1,000 x 1,000 0.08 / 0.07,
// 10,000 x 10,000 0.19 / 0.18; k=1 0.13 / 0.18).
Route route_of(int64_t n, int64_t nq, int d, int k, int dtype) {
    const double pairs = double(n) * double(nq);
    const bool narrow = d <= 3;
    if (narrow && n >= 512) {
        const double worth = dtype == TK_F64 ? 3e5 : (k == 1 ? 4e8 : (k < 8 ? 2.5e8 : 1e8));
        if (pairs >= worth) return Route::kTree;
    }
    if (dtype != TK_F32 || d > 47 || k > 32 || n < 512 || pairs < 6e4) return Route::kCudaCores;
    if (narrow && (k < 4 || (k < 8 && pairs > 5e7))) return Route::kCudaCores;
    if (k < 4 && pairs < (d <= 8 ? 5e8 : 1e6)) return Route::kCudaCores;
    if (brute_tc_workspace_bytes(n, nq, d, k, TK_BRUTE_BF16_SPLIT, kRoutePass) > kRouteBytes) return Route::kCudaCores;
    return Route::kTensorCores;
}

// Workspace of the tree route: the exhaustive search's (for clouds with NaN
// or infinite coordinates), then the tree's.
size_t exact_ws_bytes(int64_t n, int64_t nq, int d, int k, int dtype) {
    const BrutePlan p = plan_brute(n, nq, d, k, dtype != TK_F64);
    return dtype == TK_F64 ? brute_ws_bytes<double>(p, nq, k) : brute_ws_bytes<float>(p, nq, k);
}

template <typename T>
int run_tree_route(const T* ref, int64_t n, const T* q, int64_t nq, int d, int k, int dtype, T* dists, int32_t* idx,
                   char* ws, size_t ws_bytes, cudaStream_t s) {
    const size_t eb = exact_ws_bytes(n, nq, d, k, dtype);
    if (!ws || ws_bytes < eb + transient_tree_workspace_bytes(n, nq, d, k, dtype))
        return fail(TK_EWORKSPACE, "workspace too small");
    const int* odd = nullptr;
    const int rc = transient_tree_query(ref, n, q, nq, d, k, dtype, dists, idx, ws + eb, s, &odd);
    if (rc != TK_OK) return rc;
    return run_brute<T>(ref, n, q, nq, d, k, dists, idx, ws, eb, s, odd + 1);
}

int check_common(const void* ref, int64_t n, const void* q, int64_t nq, int d, int k, int dtype, const void* dists,
                 const void* idx) {
    if (n < 1 || n >= (int64_t(1) << 31)) return fail(TK_EINVAL, "reference count must be in [1, 2^31)");
    if (nq < 0 || nq >= (int64_t(1) << 31)) return fail(TK_EINVAL, "query count must be in [0, 2^31)");
    if (d < 1 || d > 128) return fail(TK_EINVAL, "dims must be in [1, 128]");
    if (k < 1) return fail(TK_EINVAL, "k must be >= 1");
    if (k > n) return fail(TK_EINVAL, "You requested more nearest neighbors than there are reference points");
    if (k > kMaxK) return fail(TK_EINVAL, "k is limited to 128");
    if (dtype != TK_F32 && dtype != TK_F64) return fail(TK_EINVAL, "dtype must be TK_F32 or TK_F64");
    if (nq > 0 && (!ref || !q || !dists || !idx)) return fail(TK_EINVAL, "null pointer");
    return TK_OK;
}

}  // namespace

// ------------------------------------------------- listed queries --
//
// The exact answers of the queries on a device-side list, whose length only
// the device knows.  Usually it is empty or short: up to kFew queries are
// searched in (query, slice) pairs, a lane per reference row read from global
// memory -- a chain of such reads, so up to kVeryFew queries a block's eight
// warps share a pair (one query in 262,144 references, d=32: 0.2 ms -> 0.04),
// above that a warp takes one (0.8 us per query).  Longer lists go through the
// tiled kernel above, a block per (query tile, slice) pair.  A
// last kernel merges a query's slices, a block per query or for long lists a
// warp; whichever kernel is not meant exits at once.  (The tiled kernel for any
// list, with a lane merging a query's 128 slices, took 1.0 ms for a few dozen
// queries.)
namespace {

constexpr int kFew = 256;
constexpr int kFewSlices = 64;
constexpr int kVeryFew = 32;
constexpr int kMaxSlices = 128;

// The tiled kernel's plan for a list: enough blocks for the tiles of all
// queries, and for 8 an SM.
BrutePlan plan_list(int64_t n, int64_t nq, int d, int k) {
    BrutePlan p = plan_brute(n, nq, d, k, true);
    p.nsplit = int(std::max<int64_t>(1, std::min<int64_t>(kMaxSlices, n / 256)));
    p.list_blocks = std::max(p.qtiles, 8 * sm_count_dev());
    return p;
}

struct ListArgs {
    const float* ref;
    const float* q;
    int n, d, k;
    const int* qlist;
    const int* qcount;
    Key<float>* part;  // [listed query][slice][k]
    int max_slices, tile_blocks, per_tile;  // of the tiled kernel
    float* out_d;
    int32_t* out_i;
};

// Rows of d floats, 16 bytes at a time when `vec`; the reference's order.
__device__ __forceinline__ float row_dist(const float* __restrict__ q, const float* __restrict__ r, int d, bool vec) {
    float acc = 0.f;
    if (vec) {
        for (int c = 0; c < d; c += 4) {
            const float4 a = __ldg(reinterpret_cast<const float4*>(q + c)), b = __ldg(reinterpret_cast<const float4*>(r + c));
            const float d0 = sub_rn(a.x, b.x), d1 = sub_rn(a.y, b.y), d2 = sub_rn(a.z, b.z), d3 = sub_rn(a.w, b.w);
            acc = add_rn(add_rn(add_rn(add_rn(acc, mul_rn(d0, d0)), mul_rn(d1, d1)), mul_rn(d2, d2)), mul_rn(d3, d3));
        }
    } else {
        for (int c = 0; c < d; ++c) {
            const float t = sub_rn(q[c], r[c]);
            acc = add_rn(acc, mul_rn(t, t));
        }
    }
    return acc;
}

// The lists of a block's eight warps, joined in the first warp's.  Every
// thread of the block calls it.
template <int R>
__device__ __forceinline__ void join_lists(WarpList<float, R>& wl, Key<float> (*all)[32 * R], int k, int lane, int w) {
    if (w > 0) {
#pragma unroll
        for (int i = 0; i < R; ++i) all[w][i * 32 + lane] = wl.list.slot[i];
    }
    __syncthreads();
    if (w == 0) {
        for (int o = 1; o < 8; ++o) {
#pragma unroll
            for (int i = 0; i < R; ++i)
                wl.offer(i * 32 + lane >= 32 * R - k ? all[o][i * 32 + lane] : Key<float>::sentinel(), lane);
        }
        wl.flush(lane);
    }
    __syncthreads();
}

template <int R>
__global__ void __launch_bounds__(256) k_few_search(const ListArgs a) {
    __shared__ Key<float> bufs[8][64];
    __shared__ Key<float> all[8][32 * R];
    const int count = *a.qcount;
    if (count == 0 || count > kFew) return;
    const int share = count <= kVeryFew ? 8 : 1;  // warps of a pair
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const bool vec = (a.d & 3) == 0 && ((reinterpret_cast<uintptr_t>(a.ref) | reinterpret_cast<uintptr_t>(a.q)) & 15) == 0;
    const int per = (a.n + kFewSlices - 1) / kFewSlices;
    const int first = share == 8 ? int(blockIdx.x) : int(blockIdx.x) * 8 + w;
    for (int item = first; item < count * kFewSlices; item += int(gridDim.x) * 8 / share) {
        const int slot = item / kFewSlices, slice = item % kFewSlices;
        const float* q = a.q + (long long)a.qlist[slot] * a.d;
        int r0 = int(min((long long)a.n, (long long)per * slice)), r1 = int(min((long long)a.n, (long long)r0 + per));
        if (share == 8) {
            const int sub = (r1 - r0 + 7) / 8;
            r0 = min(r1, r0 + sub * w);
            r1 = min(r1, r0 + sub);
        }
        WarpList<float, R> wl;
        wl.init(a.k, bufs[w], lane);
        for (int r = r0; r < r1; r += 32) {
            Key<float> mine = Key<float>::sentinel();
            if (r + lane < r1) mine = Key<float>::make(row_dist(q, a.ref + (long long)(r + lane) * a.d, a.d, vec), uint32_t(r + lane));
            wl.offer(mine, lane);
        }
        wl.flush(lane);
        if (share == 8) {
            join_lists<R>(wl, all, a.k, lane, w);
            if (w > 0) continue;
        }
        Key<float>* out = a.part + (long long)item * a.k;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int o = i * 32 + lane - (32 * R - a.k);
            if (o >= 0) out[o] = wl.list.slot[i];
        }
    }
}

template <int R>
__global__ void __launch_bounds__(256) k_list_merge(const ListArgs a) {
    __shared__ Key<float> bufs[8][64];
    __shared__ Key<float> all[8][32 * R];
    const int count = *a.qcount;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (count <= kFew) {  // a block per query
        const int total = kFewSlices * a.k;
        for (int slot = blockIdx.x; slot < count; slot += gridDim.x) {
            WarpList<float, R> wl;
            wl.init(a.k, bufs[w], lane);
            const Key<float>* src = a.part + (long long)slot * total;
            for (int e = threadIdx.x; e - lane < total; e += 256)
                wl.offer(e < total ? src[e] : Key<float>::sentinel(), lane);
            wl.flush(lane);
            join_lists<R>(wl, all, a.k, lane, w);
            if (w == 0) wl.list.store(a.k, lane, a.out_d, a.out_i, a.qlist[slot]);
        }
        return;
    }
    const int slices = list_slices(count, a.tile_blocks, a.per_tile, a.max_slices);
    if (slices == 1) return;  // already in the outputs
    for (int slot = blockIdx.x * 8 + w; slot < count; slot += gridDim.x * 8) {
        WarpList<float, R> wl;
        wl.init(a.k, bufs[w], lane);
        const Key<float>* src = a.part + (long long)slot * slices * a.k;
        const int total = slices * a.k;
        for (int e = lane; e - lane < total; e += 32) wl.offer(e < total ? src[e] : Key<float>::sentinel(), lane);
        wl.flush(lane);
        wl.list.store(a.k, lane, a.out_d, a.out_i, a.qlist[slot]);
    }
}

}  // namespace

// Both kernels share one buffer of per-slice lists, some 80 MB for k = 32
// however many queries there are: a list per query of each of the tiled
// kernel's blocks, or of the slices of a short list.
size_t brute_fallback_workspace_bytes(int64_t n, int64_t nq, int d, int k) {
    nq = std::max<int64_t>(nq, 1);
    const BrutePlan p = plan_list(n, nq, d, k);
    const int64_t tiled = std::min(nq * p.nsplit, int64_t(p.list_blocks) * (256 / p.G));
    const int64_t few = std::min<int64_t>(nq, kFew) * kFewSlices;
    return align256(sizeof(Key<float>) * size_t(std::max(tiled, few)) * k);
}

int brute_fallback(const float* ref, int64_t n, const float* q, int64_t nq, int d, int k, float* dists,
                   int32_t* idx, const int* qlist, const int* qcount, void* ws, size_t ws_bytes, cudaStream_t s) {
    if (ws_bytes < brute_fallback_workspace_bytes(n, nq, d, k)) return fail(TK_EWORKSPACE, "fallback workspace");
    const int sms = sm_count_dev(), few = int(std::min<int64_t>(nq, kFew));
    const BrutePlan p = plan_list(n, nq, d, k);
    ListArgs l{ref, q, int(n), d, k, qlist, qcount, static_cast<Key<float>*>(ws), p.nsplit, p.list_blocks, 256 / p.G,
               dists, idx};
    const unsigned gs = unsigned(std::min(4 * sms, few * kFewSlices));
    const unsigned gm = unsigned(std::min<int64_t>(4 * sms, std::max<int64_t>(few, (nq + 7) / 8)));
    if (k <= 32) k_few_search<1><<<gs, 256, 0, s>>>(l);
    else if (k <= 64) k_few_search<2><<<gs, 256, 0, s>>>(l);
    else k_few_search<4><<<gs, 256, 0, s>>>(l);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(TK_ECUDA, std::string("listed queries: ") + cudaGetErrorString(e));
    if (nq > kFew) {
        BruteArgs<float> a;
        a.ref = ref;
        a.q = q;
        a.n = int(n);
        a.nq = int(nq);
        a.d = d;
        a.k = k;
        a.nsplit = p.nsplit;
        a.out_d = dists;
        a.out_i = idx;
        a.part = static_cast<Key<float>*>(ws);
        a.qlist = qlist;
        a.qcount = qcount;
        a.qmore = kFew;
        const int rc = launch_brute<float>(a, p, s);
        if (rc != TK_OK) return rc;
    }
    if (k <= 32) k_list_merge<1><<<gm, 256, 0, s>>>(l);
    else if (k <= 64) k_list_merge<2><<<gm, 256, 0, s>>>(l);
    else k_list_merge<4><<<gm, 256, 0, s>>>(l);
    e = cudaGetLastError();
    if (e != cudaSuccess) return fail(TK_ECUDA, std::string("listed queries: ") + cudaGetErrorString(e));
    return TK_OK;
}

}  // namespace tk

using namespace tk;

extern "C" {

size_t tk_nn_distance_workspace_size(int64_t n, int64_t nq, int dims, int k, int dtype, int mode) {
    if (n < 1 || nq < 0 || k < 1 || dims < 1) return 0;
    if (mode == TK_BRUTE_TF32 || mode == TK_BRUTE_BF16_SPLIT) return brute_tc_workspace_bytes(n, nq, dims, k, mode, kTcPass);
    nq = std::max<int64_t>(nq, 1);
    const Route route = mode == TK_BRUTE_ROUTED ? route_of(n, nq, dims, k, dtype) : Route::kCudaCores;
    if (route == Route::kTensorCores) return brute_tc_workspace_bytes(n, nq, dims, k, TK_BRUTE_BF16_SPLIT, kRoutePass);
    return exact_ws_bytes(n, nq, dims, k, dtype) +
           (route == Route::kTree ? transient_tree_workspace_bytes(n, nq, dims, k, dtype) : 0);
}

int tk_nn_distance(const void* ref, int64_t n, const void* q, int64_t nq, int dims, int k, int dtype, int mode,
                   void* dists, int32_t* idx, void* workspace, size_t workspace_bytes, void* stream) {
    clear_error();
    int rc = check_common(ref, n, q, nq, dims, k, dtype, dists, idx);
    if (rc != TK_OK) return rc;
    if (nq == 0) return TK_OK;
    if (ws_misaligned(workspace)) return fail(TK_EINVAL, "workspace must be 256-byte aligned");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const Route route = mode == TK_BRUTE_ROUTED ? route_of(n, nq, dims, k, dtype) : Route::kCudaCores;
    if (route == Route::kTree) {
        char* ws = static_cast<char*>(workspace);
        if (dtype == TK_F32)
            return run_tree_route<float>(static_cast<const float*>(ref), n, static_cast<const float*>(q), nq, dims, k,
                                         dtype, static_cast<float*>(dists), idx, ws, workspace_bytes, s);
        return run_tree_route<double>(static_cast<const double*>(ref), n, static_cast<const double*>(q), nq, dims, k,
                                      dtype, static_cast<double*>(dists), idx, ws, workspace_bytes, s);
    }
    if (route == Route::kTensorCores)
        return run_brute_tc(static_cast<const float*>(ref), n, static_cast<const float*>(q), nq, dims, k,
                            TK_BRUTE_BF16_SPLIT, static_cast<float*>(dists), idx, workspace, workspace_bytes,
                            kRoutePass, s);
    if (mode == TK_BRUTE_EXACT || mode == TK_BRUTE_ROUTED) {
        if (dtype == TK_F32)
            return run_brute<float>(static_cast<const float*>(ref), n, static_cast<const float*>(q), nq, dims, k,
                                    static_cast<float*>(dists), idx, workspace, workspace_bytes, s);
        return run_brute<double>(static_cast<const double*>(ref), n, static_cast<const double*>(q), nq, dims, k,
                                 static_cast<double*>(dists), idx, workspace, workspace_bytes, s);
    }
    if (mode == TK_BRUTE_TF32 || mode == TK_BRUTE_BF16_SPLIT) {
        if (dtype != TK_F32) return fail(TK_EINVAL, "tensor-core modes take float32 inputs");
        return run_brute_tc(static_cast<const float*>(ref), n, static_cast<const float*>(q), nq, dims, k, mode,
                            static_cast<float*>(dists), idx, workspace, workspace_bytes, kTcPass, s);
    }
    return fail(TK_EINVAL, "unknown brute-force mode");
}

}  // extern "C"
