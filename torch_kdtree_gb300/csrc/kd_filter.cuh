// Single-precision filter of float64 trees of 1-3 dimensions.
//
// Double precision runs at 1/64 of the float rate here, and a search spends
// it on boxes and points that are far out of reach.  A tree built on the GPU
// therefore also holds float images of its points, node boxes and split
// values, relative to the cloud's centre and scaled by a power of two to an
// extent near 1 (Frame).  The search walks those: a float lower bound on the
// exact distance -- directed rounding throughout -- discards a node or point
// when it exceeds the current k-th distance, rounded up; what is left is
// computed in double, 32 points at a time, with the reference's arithmetic.
// The answer is the exact search's, bit for bit: nothing is discarded whose
// computed distance could reach the k-th (a computed distance is at least the
// real one less 2^-51 of it; the comparison allows 2^-21).  Which child a
// descent takes is free, since siblings are tested by their boxes.
//
// 65,536 queries in 200,000 points, k=8: 0.77 ms without the filter (1.06 ms on
// four lanes per query), 0.27 ms with it; the image grows from 32 to 48 bytes
// per point.  The double pipe was still 75% busy at 0.32 ms, a good part of it
// with the query's place in the frame, now an axis per lane, and the reach,
// now in integers.  What is left is the survivors' distances; keeping those of
// several leaves for one batch costs more in reach (4 or more: 2-10% slower).
#pragma once

#include <cuda_runtime.h>

#include "kd_warp.cuh"
#include "tk_device.cuh"
#include "tk_internal.h"

namespace tk {

struct Frame {
    double centre[3];
    double scale;  // a power of two, 2^-400 .. 2^400 (its square neither overflows nor lets squares underflow)
};

struct FilterView {
    const PointRec<float>* pts = nullptr;    // in leaf order (w unused); null: the tree has no filter
    const PointRec<float>* boxes = nullptr;  // rounded outwards; w: point range as in the double boxes
    const float* medians = nullptr;
    const Frame* frame = nullptr;
};

struct FilterArgs {
    FilterView f;
    const PointRec<double>* pts;
    int levels;
    const double* q;  // [nq, D]
    int nq, k;
    const int32_t* order;
    double* out_d;
    int32_t* out_i;
    int* work;
};

__device__ __forceinline__ double frame_down(double v, double c, double s) { return __dmul_rd(__dsub_rd(v, c), s); }
__device__ __forceinline__ double frame_up(double v, double c, double s) { return __dmul_ru(__dsub_ru(v, c), s); }

// A float no less than d 2^e, d a distance given by its bits (never negative,
// never NaN): at most an ulp more than the next float, at least 2^-126.  In
// integers: a search asks for it at every leaf.
__device__ __forceinline__ float scaled_up(unsigned long long d, int e) {
    const int field = int(d >> 52);
    if (field == 0x7FF) return __int_as_float(0x7f800000);
    const int f = max(field, 1) - 1023 + e + 127;
    if (f <= 0) return __int_as_float(0x00800000);
    if (f >= 255) return __int_as_float(0x7f800000);
    return __int_as_float((f << 23) + int((d >> 29) & 0x7FFFFFull) + 1);
}

template <int D, int R>
__device__ __forceinline__ void kd_search_filtered(const FilterArgs& a, const double (&q)[D], double* out_d,
                                                   int32_t* out_i, Key<double>* buf, uint32_t* todo, int lane) {
    WarpList<double, R> wl;
    wl.init(a.k, buf, lane);
    const int L = a.levels;
    const double scale = a.f.frame->scale;
    bool nan_q = false;  // all distances are NaN and enter no list: the home leaf is enough
    float lo[D], hi[D];  // the query's place in the frame, an axis per lane
    {
        const int c = lane < D ? lane : 0;
        double qc = q[0];
        if (D > 1) qc = c == 1 ? q[D > 1 ? 1 : 0] : qc;
        if (D > 2) qc = c == 2 ? q[D > 2 ? 2 : 0] : qc;
        const double centre = a.f.frame->centre[c];
        const float down = __double2float_rd(frame_down(qc, centre, scale));
        const float up = __double2float_ru(frame_up(qc, centre, scale));
#pragma unroll
        for (int i = 0; i < D; ++i) {
            nan_q |= (__double_as_longlong(q[i]) & 0x7FFFFFFFFFFFFFFFll) > 0x7FF0000000000000ll;
            lo[i] = __shfl_sync(0xFFFFFFFFu, down, i);
            hi[i] = __shfl_sync(0xFFFFFFFFu, up, i);
        }
    }
    const int scale_exp = 2 * (int((__double_as_longlong(scale) >> 52) & 0x7FF) - 1023);
    float reach = __int_as_float(0x7f800000);  // the k-th distance in the frame, rounded up
    auto set_reach = [&]() { reach = __fmul_ru(scaled_up(wl.worst.d, scale_exp), 1.0f + 0x1p-21f); };
    // sum of squares of lower bounds on the per-axis distances
    auto sum_sq = [&](const float (&g)[D]) {
        float s = 0.f;
#pragma unroll
        for (int c = 0; c < D; ++c) {
            const float p = fmaxf(g[c], 0.f);
            s = __fadd_rd(s, __fmul_rd(p, p));
        }
        return s;
    };
    auto point_bound = [&](const PointRec<float>& p) {
        const float x[3] = {p.x, p.y, p.z};
        float g[D];
#pragma unroll
        for (int c = 0; c < D; ++c)  // a coordinate was rounded by at most 2^-24 of itself
            g[c] = __fmaf_rd(-0x1p-23f, fabsf(x[c]), fmaxf(__fsub_rd(lo[c], x[c]), __fsub_rd(x[c], hi[c])));
        return sum_sq(g);
    };
    auto box_bound_f = [&](const PointRec<float>& bl, const PointRec<float>& bh) {
        const float l[3] = {bl.x, bl.y, bl.z}, h[3] = {bh.x, bh.y, bh.z};
        float g[D];
#pragma unroll
        for (int c = 0; c < D; ++c) g[c] = fmaxf(__fsub_rd(l[c], hi[c]), __fsub_rd(lo[c], h[c]));
        return sum_sq(g);
    };
    auto qa = [&](int ax) {
        float r = lo[0];
        if (D > 1) r = ax == 1 ? lo[D > 1 ? 1 : 0] : r;
        if (D > 2) r = ax == 2 ? lo[D > 2 ? 2 : 0] : r;
        return r;
    };
    int waiting = 0;
    // exact distances of the first m points on the list
    auto evaluate = [&](int m) {
        Key<double> mine = Key<double>::sentinel();
        if (lane < m) {
            const PointRec<double> p = load_rec(a.pts + todo[lane]);
            mine = Key<double>::make(sqdist<double, D>(q, p), rec_index(p));
        }
        wl.offer(mine, lane);
    };
    auto collect = [&](int j, bool valid, const PointRec<float>& p) {
        const bool hit = valid && point_bound(p) <= reach;
        const unsigned m = __ballot_sync(0xFFFFFFFFu, hit);
        if (!m) return;
        if (hit) todo[waiting + __popc(m & ((1u << lane) - 1u))] = uint32_t(j);
        waiting += __popc(m);
        __syncwarp();
        if (waiting >= 32) {
            evaluate(32);
            const uint32_t rest = todo[32 + lane];
            __syncwarp();
            waiting -= 32;
            if (lane < waiting) todo[lane] = rest;
            __syncwarp();
            set_reach();
        }
    };

    int leaf = warp_descend(a.f.medians, 0, 0, L, D, lane, qa);
    float bound = 0.f;  // of this lane's sibling (lane 31: of the leaf)
    bool pending = false;
    int range = 0, range_end = 0;
    for (int fresh = 0;;) {  // lanes fresh .. L - 1 have new siblings
        if ((lane >= fresh && lane < L) || lane == 31) {
            const int node = lane == 31 ? leaf : path_sibling(leaf, L, lane);
            const PointRec<float> bl = load_rec(a.f.boxes + 2 * node);
            const PointRec<float> bh = load_rec(a.f.boxes + 2 * node + 1);
            bound = box_bound_f(bl, bh);
            range = int(rec_index(bl));
            range_end = int(rec_index(bh));
            pending = lane != 31 && !nan_q;
        }
        const int beg = __shfl_sync(0xFFFFFFFFu, range, 31);
        const int end = __shfl_sync(0xFFFFFFFFu, range_end, 31);
        if (__shfl_sync(0xFFFFFFFFu, bound, 31) <= reach) {
            for (int j = beg + lane; j - lane < end; j += 64) {
                PointRec<float> p0{}, p1{};
                if (j < end) p0 = load_rec(a.f.pts + j);
                if (j + 32 < end) p1 = load_rec(a.f.pts + j + 32);
                collect(j, j < end, p0);
                if (j - lane + 32 < end) collect(j + 32, j + 32 < end, p1);
            }
            if (waiting > 0) {
                evaluate(waiting);
                waiting = 0;
                __syncwarp();
            }
            wl.flush(lane);
            set_reach();
        }
        const unsigned m = __ballot_sync(0xFFFFFFFFu, pending && bound <= reach);
        if (!m) break;
        const int t = 31 - __clz(m);
        pending = pending && lane < t;
        leaf = warp_descend(a.f.medians, path_sibling(leaf, L, t), t + 1, L, D, lane, qa);
        fresh = t + 1;
    }
    wl.list.store(a.k, lane, out_d, out_i, 0);
}

template <int D, int R>
__global__ void __launch_bounds__(256) k_kd_query_filtered(const FilterArgs a) {
    __shared__ Key<double> bufs[8][64];
    __shared__ uint32_t todo[8][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int round = 0;;) {
        const int t = next_queries(a.work, 1, a.nq, round);
        if (t >= a.nq) break;
        const int qi = a.order ? __ldg(a.order + t) : t;
        double q[D];
#pragma unroll
        for (int c = 0; c < D; ++c) q[c] = a.q[(long long)qi * D + c];
        kd_search_filtered<D, R>(a, q, a.out_d + (long long)qi * a.k, a.out_i + (long long)qi * a.k, bufs[w], todo[w],
                                 lane);
        __syncwarp();
    }
}

// kd_filter.cu
const void* kd_filtered_kernel(int D, int R);
int kd_filtered_launch(const FilterArgs& a, int D, int R, int grid, cudaStream_t s);

}  // namespace tk
