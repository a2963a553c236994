// Tensor-core brute force: kernels and launch templates, shared by the units
// that instantiate them (brute_tc5_tf32.cu, brute_tc5_tf32_deep.cu,
// brute_tc5_bf16.cu: the tcgen05 candidate search per operand mode and row
// depth; brute_tc_mma.cu: the mma.sync search for deeper rows or larger k;
// brute_tc.cu: packing, re-rank and the host side).
// The algorithm is described at the top of brute_tc.cu.
#pragma once

#include <cuda_bf16.h>

#include <string>

#include "brute.cuh"
#include "kd_warp.cuh"
#include "launch.cuh"
#include "tc_sm100.cuh"
#include "tk_internal.h"

namespace tk {
namespace tcx {


constexpr int kRows = 128;   // queries per block
constexpr int kCols = 128;   // references per tile
constexpr int kThreads = 256;

inline size_t align256(size_t v) { return (v + 255) / 256 * 256; }

// The certificate below reasons about finite scores: a slice whose list never
// filled (tau = +inf) holds every reference of the slice.  NaN scores (from
// non-finite coordinates) enter no list, and overflowing ones break the error
// bound, so a query is certified only when |q|^2 < 2^125 and every reference
// has |r|^2 < 2^125 (the pack kernel flags any other reference in `err`,
// which certifies nothing; the tcgen05 path packs references with infinite or
// NaN coordinates as padding).  Then every partial sum of a score is below
// |r|^2 + 2|q||r| <= 2 (|q|^2 + |r|^2) < 2^127: finite.  Uncertified queries
// are answered by the exact kernel.
constexpr float kTcNormLimit = 0x1p125f;
// Bits of the candidate search's error word (any bit: certify nothing, so
// the exact kernel recomputes every query and the answer stays exact).
constexpr int kTcErrTimeout = 1;  // a bounded wait of the tcgen05 kernel ran out
constexpr int kTcErrRange = 2;    // an input outside the certificate's range (kTcNormLimit)

__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}

// Row-major packed operands: TF32 -> one uint32 per element, BF16 split ->
// hi and lo bf16 planes.  Rows are zero-padded to KP elements.
template <int MODE>
__global__ void k_tc_pack(const float* __restrict__ x, int rows, int d, int KP, uint32_t* __restrict__ tf,
                          __nv_bfloat16* __restrict__ hi, __nv_bfloat16* __restrict__ lo, float* __restrict__ norm,
                          int* __restrict__ err) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    float s = 0.f;
    for (int c = 0; c < KP; ++c) {
        const float v = c < d ? x[(long long)r * d + c] : 0.f;
        s = fmaf(v, v, s);
        if (MODE == TK_BRUTE_TF32) {
            tf[(long long)r * KP + c] = to_tf32(v);
        } else {
            const __nv_bfloat16 h = __float2bfloat16_rn(v);
            hi[(long long)r * KP + c] = h;
            lo[(long long)r * KP + c] = __float2bfloat16_rn(v - __bfloat162float(h));
        }
    }
    norm[r] = s;
    if (err && !(s < kTcNormLimit)) atomicOr(err, kTcErrRange);  // see kTcNormLimit
}

struct TcArgs {
    const uint32_t* a_tf;  // queries (TF32)
    const uint32_t* b_tf;  // references (TF32)
    const __nv_bfloat16 *a_hi, *a_lo, *b_hi, *b_lo;
    const float* rnorm;    // |r|^2
    int n, nq, KP, C;
    int nsplit;
    float* cand_s;         // [nq, nsplit, C] scores
    int32_t* cand_i;       // [nq, nsplit, C] indices (-1 = empty)
    float* tau;            // [nq, nsplit]
};

__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// KP: padded depth (TF32: multiple of 8; BF16: multiple of 16).  C: over-fetch.
template <int MODE, int KP, int C>
__global__ void __launch_bounds__(kThreads, 1) k_tc_select(const TcArgs a) {
    constexpr int KW = (MODE == TK_BRUTE_TF32) ? KP : KP / 2;  // 32-bit words per packed row
    constexpr int BS = KW + 4;                                  // smem row stride (bank-conflict free)
    constexpr int SS = kCols + 4;                               // score tile row stride
    constexpr int PLANES = (MODE == TK_BRUTE_TF32) ? 1 : 2;
    extern __shared__ __align__(1024) unsigned char smem[];  // one declaration per unit: k_tc5_select's alignment
    uint32_t* Bs = reinterpret_cast<uint32_t*>(smem);                        // [PLANES][kCols][BS]
    float* rn = reinterpret_cast<float*>(Bs + PLANES * kCols * BS);          // [kCols]
    float* S = rn + kCols;                                                   // [kRows][SS]
    float* Ls = S + kRows * SS;                                              // [C][kRows]
    int32_t* Li = reinterpret_cast<int32_t*>(Ls + C * kRows);                // [C][kRows]

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int q0 = blockIdx.x * kRows;
    const long long per = ((long long)a.n + a.nsplit - 1) / a.nsplit;
    const int r0 = int(min((long long)a.n, per * blockIdx.y));
    const int r1 = int(min((long long)a.n, per * (blockIdx.y + 1)));

    // A fragments of this warp's 16 rows, all k-steps, kept in registers
    constexpr int KSTEPS = (MODE == TK_BRUTE_TF32) ? KP / 8 : KP / 16;
    uint32_t af[PLANES][KSTEPS][4];
    {
        const int ra = q0 + warp * 16 + g, rb = ra + 8;
#pragma unroll
        for (int p = 0; p < PLANES; ++p) {
#pragma unroll
            for (int ks = 0; ks < KSTEPS; ++ks) {
                if (MODE == TK_BRUTE_TF32) {
                    const uint32_t* A = a.a_tf;
                    const int c0 = ks * 8 + t, c1 = c0 + 4;
                    af[p][ks][0] = ra < a.nq ? A[(long long)ra * KP + c0] : 0u;
                    af[p][ks][1] = rb < a.nq ? A[(long long)rb * KP + c0] : 0u;
                    af[p][ks][2] = ra < a.nq ? A[(long long)ra * KP + c1] : 0u;
                    af[p][ks][3] = rb < a.nq ? A[(long long)rb * KP + c1] : 0u;
                } else {
                    const uint32_t* A = reinterpret_cast<const uint32_t*>(p == 0 ? a.a_hi : a.a_lo);
                    const int w0 = ks * 8 + t, w1 = w0 + 4;  // 32-bit words: element pairs
                    af[p][ks][0] = ra < a.nq ? A[(long long)ra * KW + w0] : 0u;
                    af[p][ks][1] = rb < a.nq ? A[(long long)rb * KW + w0] : 0u;
                    af[p][ks][2] = ra < a.nq ? A[(long long)ra * KW + w1] : 0u;
                    af[p][ks][3] = rb < a.nq ? A[(long long)rb * KW + w1] : 0u;
                }
            }
        }
    }

    // per-row candidate lists (threads 0..127 own one row each)
    int cnt = 0;
    float tau = __int_as_float(0x7f800000);
    for (int c = 0; c < C && tid < kRows; ++c) {
        Ls[c * kRows + tid] = tau;
        Li[c * kRows + tid] = -1;
    }

    for (int c0 = r0; c0 < r1; c0 += kCols) {
        const int len = min(kCols, r1 - c0);
        __syncthreads();
        // reference tile -> shared memory (zero rows past the slice end)
        for (int e = tid; e < PLANES * kCols * KW; e += kThreads) {
            const int p = e / (kCols * KW);
            const int rem = e - p * kCols * KW;
            const int j = rem / KW, w = rem - j * KW;
            uint32_t v = 0u;
            if (j < len) {
                const uint32_t* B = MODE == TK_BRUTE_TF32 ? a.b_tf
                                                          : reinterpret_cast<const uint32_t*>(p == 0 ? a.b_hi : a.b_lo);
                v = B[(long long)(c0 + j) * KW + w];
            }
            Bs[(p * kCols + j) * BS + w] = v;
        }
        for (int j = tid; j < kCols; j += kThreads) rn[j] = j < len ? a.rnorm[c0 + j] : __int_as_float(0x7f800000);
        __syncthreads();
        // 16 x 128 scores per warp
        float acc[kCols / 8][4];
#pragma unroll
        for (int nt = 0; nt < kCols / 8; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[nt][i] = 0.f;
#pragma unroll
        for (int ks = 0; ks < KSTEPS; ++ks) {
#pragma unroll
            for (int nt = 0; nt < kCols / 8; ++nt) {
                const int j = nt * 8 + g;
                if (MODE == TK_BRUTE_TF32) {
                    const uint32_t b0 = Bs[j * BS + ks * 8 + t];
                    const uint32_t b1 = Bs[j * BS + ks * 8 + t + 4];
                    mma_tf32(acc[nt], af[0][ks], b0, b1);
                } else {
                    const uint32_t bh0 = Bs[j * BS + ks * 8 + t];
                    const uint32_t bh1 = Bs[j * BS + ks * 8 + t + 4];
                    const uint32_t bl0 = Bs[(kCols + j) * BS + ks * 8 + t];
                    const uint32_t bl1 = Bs[(kCols + j) * BS + ks * 8 + t + 4];
                    mma_bf16(acc[nt], af[0][ks], bh0, bh1);  // hi * hi
                    mma_bf16(acc[nt], af[0][ks], bl0, bl1);  // hi * lo
                    mma_bf16(acc[nt], af[PLANES - 1][ks], bh0, bh1);  // lo * hi
                }
            }
        }
        // scores -> shared memory
        {
            const int ra = warp * 16 + g;
#pragma unroll
            for (int nt = 0; nt < kCols / 8; ++nt) {
                const int cc = nt * 8 + 2 * t;
                S[ra * SS + cc] = acc[nt][0];
                S[ra * SS + cc + 1] = acc[nt][1];
                S[(ra + 8) * SS + cc] = acc[nt][2];
                S[(ra + 8) * SS + cc + 1] = acc[nt][3];
            }
        }
        __syncthreads();
        // one thread per row: filter by tau, insert the rare survivors
        if (tid < kRows) {
            const float* row = S + tid * SS;
            for (int j = 0; j < len; ++j) {
                const float sc = fmaf(-2.f, row[j], rn[j]);
                if (sc < tau) {
                    int pos = cnt < C ? cnt : C - 1;
                    while (pos > 0 && Ls[(pos - 1) * kRows + tid] > sc) {
                        Ls[pos * kRows + tid] = Ls[(pos - 1) * kRows + tid];
                        Li[pos * kRows + tid] = Li[(pos - 1) * kRows + tid];
                        --pos;
                    }
                    Ls[pos * kRows + tid] = sc;
                    Li[pos * kRows + tid] = c0 + j;
                    cnt = min(cnt + 1, C);
                    if (cnt == C) tau = Ls[(C - 1) * kRows + tid];
                }
            }
        }
    }
    // write the lists
    if (tid < kRows) {
        const int q = q0 + tid;
        if (q < a.nq) {
            const long long base = ((long long)q * a.nsplit + blockIdx.y) * C;
            for (int c = 0; c < C; ++c) {
                a.cand_s[base + c] = Ls[c * kRows + tid];
                a.cand_i[base + c] = Li[c * kRows + tid];
            }
            a.tau[(long long)q * a.nsplit + blockIdx.y] = cnt == C ? tau : __int_as_float(0x7f800000);
        }
    }
}

// ---------------------------------------------------------------------------
// tcgen05 path (d <= 39 for TF32, d <= 47 for BF16 split; k <= 32).
//
// The score is produced by the MMA itself by augmenting K with one column:
//   A = [-2 q, 1, 0...],  B = [r, |r|^2, 0...]  =>  A.B = |r|^2 - 2 q.r.
// Operands are packed in global memory in the tensor core's canonical
// no-swizzle K-major layout (8-row x 16-byte core matrices; core matrices
// adjacent along K 128 bytes apart, 8-row groups 8*KB bytes apart), one
// contiguous block per 128 query rows / 256 reference rows, so each tile is
// a single bulk copy.  Reference r sits in tile r % tiles, at column r / tiles
// turned by a step per tile (packed_ref): references that are neighbours in
// memory, often neighbours in space, fall into different tiles (see the sample
// below) and different column groups (see the lists).  Padding rows carry a
// huge |r|^2.
constexpr int kT5MaxDims = 47;
constexpr int kT5Rows = 128;   // M (queries per block)
constexpr int kT5Cols = 256;   // N (references per tile)
constexpr int kT5EpiWarps = 16; // 4 per 32-lane quarter of the accumulator when reading tensor memory
constexpr int kT5Parts = kT5EpiWarps / 4;           // column groups of 64: lists per row and slice
constexpr int kT5Minima = 128;                      // sample minima per row
constexpr int kT5MinStride = kT5Minima + 2;         // their row stride (16-bit words): lanes of a read on other banks
constexpr int kT5Threads = 32 * (kT5EpiWarps + 1);
// |r|^2 of a padding row, and the highest threshold: a power of two, exact in
// TF32 and in BF16, so that a padding row scores just that, never below it
// (rounded down it would let r >= n into the lists).
constexpr float kT5PadNorm = 0x1p99f;
constexpr uint32_t kT5MaxTries = 1u << 22;  // bounded mbarrier polls (default; Tc5Args::max_tries)

__device__ __forceinline__ uint32_t core_offset(int row, int kb, int KB) {
    return uint32_t((row >> 3) * (8 * KB) + (kb >> 4) * 128 + (row & 7) * 16 + (kb & 15));
}

// Reference at column `col` of tile `tile`; padding when >= n.
__device__ __forceinline__ uint32_t packed_ref(uint32_t tile, uint32_t col, uint32_t tiles) {
    return ((col - 67u * tile) & uint32_t(kT5Cols - 1)) * tiles + tile;
}

// The point that queries and references are taken relative to: a score's error
// grows with their squared norms, so a cloud far from the origin (its mean 30
// times its spread) would get no certificate.  Per coordinate the median of 32
// references, where it exceeds half their interquartile range, else 0 (a cloud
// around the origin keeps its operands).  A warp per coordinate, a lane per
// reference, one block; it also zeroes the words of the report.
static __global__ void __launch_bounds__(1024) k_tc5_centre(const float* __restrict__ ref, int n, int d,
                                                            float* __restrict__ centre, int* __restrict__ err,
                                                            int* __restrict__ fail_count) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) *err = *fail_count = 0;
    for (int c = threadIdx.x >> 5; c < d; c += 32) {
        float v = ref[(long long)lane * n / 32 * d + c];
        if (!(fabsf(v) < 0x1p60f)) v = 0.f;  // infinite and NaN coordinates, too
        int rank = 0;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const float o = __shfl_sync(0xFFFFFFFFu, v, j);
            rank += o < v || (o == v && j < lane) ? 1 : 0;
        }
        auto ranked = [&](int r) { return __shfl_sync(0xFFFFFFFFu, v, __ffs(__ballot_sync(0xFFFFFFFFu, rank == r)) - 1); };
        const float lower = ranked(8), median = ranked(16), upper = ranked(24);
        if (lane == 0) centre[c] = fabsf(median) >= 0.5f * (upper - lower) ? median : 0.f;
    }
}

// One side's points and where they go.
struct Tc5Pack {
    const float* x;
    int rows, tiles;
    unsigned char *hi, *lo;
};

// A thread per 16 bytes of a packed row, [-2q, 1] (tiles of kT5Rows rows) in
// the first q_blocks blocks, [r, |r|^2] (tiles of kT5Cols rows) in the others,
// q and r relative to `centre`; |q|^2 goes to qnorm.
template <int MODE>
__global__ void __launch_bounds__(256) k_tc5_pack(const Tc5Pack queries, const Tc5Pack refs, int q_blocks, int d,
                                                  int KP, const float* centre, float* qnorm, int* err) {
    begin();
    const bool is_query = int(blockIdx.x) < q_blocks;
    const Tc5Pack& side = is_query ? queries : refs;
    const float* __restrict__ x = side.x;
    const int rows = side.rows, tiles = side.tiles;
    unsigned char *hi = side.hi, *lo = side.lo;
    __shared__ float mid[kT5MaxDims];
    if (threadIdx.x < d) mid[threadIdx.x] = centre[threadIdx.x];
    __syncthreads();
    constexpr int ESZ = MODE == TK_BRUTE_TF32 ? 4 : 2;
    constexpr int E = 16 / ESZ;  // elements of 16 bytes
    const int KB = KP * ESZ, chunks = KB / 16;
    const int tile_rows = is_query ? kT5Rows : kT5Cols;
    const long long i = (long long)(int(blockIdx.x) - (is_query ? 0 : q_blocks)) * 256 + threadIdx.x;
    const long long p = i / chunks;
    const int cb = int(i - p * chunks);
    if (p >= (long long)tiles * tile_rows) return;
    const int tile = int(p / tile_rows), c = int(p - (long long)tile * tile_rows);
    const long long r = is_query ? p : (long long)packed_ref(uint32_t(tile), uint32_t(c), uint32_t(tiles));
    const bool real = r < rows;
    const float* row = x + r * d;
    // A reference with an infinite or NaN coordinate is at distance inf or NaN:
    // it is in no certified answer (those have k finite distances), and all of
    // its row becomes padding's.  Packed as it is, its products are infinite,
    // scores of -inf take the sample's threshold down to -inf, and tau with it.
    float nrm = 0.f, odd = 0.f;  // odd: NaN if a coordinate is not finite
    const bool norm = !is_query || d / E == cb;  // a query's only where it is written
    for (int j = 0; real && norm && j < d; ++j) {
        const float v = __fsub_rn(row[j], mid[j]);
        nrm = fmaf(v, v, nrm);
        odd += row[j] - row[j];
    }
    const bool used = real && (is_query || odd == 0.f);
    float v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int k = cb * E + e;
        v[e] = 0.f;
        if (k < d) {
            v[e] = used ? __fsub_rn(row[k], mid[k]) : 0.f;
            if (is_query) v[e] = -2.f * v[e];
        } else if (k == d) {
            if (is_query) {
                v[e] = real ? 1.f : 0.f;
                if (real) qnorm[r] = nrm;
            } else {
                if (used && !(nrm < kTcNormLimit)) atomicOr(err, kTcErrRange);  // see kTcNormLimit
                v[e] = used ? nrm : kT5PadNorm;
            }
        }
    }
    const long long off = (long long)tile * tile_rows * KB + core_offset(c, cb * 16, KB);
    if constexpr (MODE == TK_BRUTE_TF32) {
        *reinterpret_cast<uint4*>(hi + off) = make_uint4(to_tf32(v[0]), to_tf32(v[1]), to_tf32(v[2]), to_tf32(v[3]));
    } else {
        __align__(16) __nv_bfloat16 h[E], l[E];
#pragma unroll
        for (int e = 0; e < E; ++e) {
            h[e] = __float2bfloat16_rn(v[e]);
            l[e] = __float2bfloat16_rn(v[e] - __bfloat162float(h[e]));
        }
        *reinterpret_cast<uint4*>(hi + off) = *reinterpret_cast<const uint4*>(h);
        *reinterpret_cast<uint4*>(lo + off) = *reinterpret_cast<const uint4*>(l);
    }
}

// Slices of the references of a row block, and how their thresholds come about
// (see k_tc5_select).
struct Tc5Slices {
    int nsplit;
    int pstride;  // every pstride-th tile of a slice is sampled
    int rank;     // the threshold is the rank-th smallest of the sample's minima
};

// The row blocks before `split_from` and those from there on may have
// different slices; lists are kept by query, then slice, then part.
__host__ __device__ inline long long first_slice(long long row, int split_from, int head, int tail) {
    const long long b = (long long)split_from * kT5Rows;
    return row < b ? row * head : b * head + (row - b) * tail;
}

struct Tc5Args {
    const unsigned char* a_hi;  // packed queries, blocks of 128 rows
    const unsigned char* a_lo;
    const unsigned char* b_hi;  // packed references, tiles of 256 rows
    const unsigned char* b_lo;
    int nq, tiles, split_from;  // row blocks with the head's slices
    Tc5Slices head, tail;
    uint2* hits;                // [slices of all rows, see first_slice][kT5Parts][CAP]: score bits, reference
    int* counts;                // [slices of all rows][kT5Parts]
    float* thr;                 // same shape: every reference of the part scoring below it is in its list
    const float* qnorm;         // |q|^2
    float eps_dot;              // see RerankArgs
    int d;
    int* err;                   // kTcErrTimeout set when a bounded wait ran out
    uint32_t max_tries;         // polls of each mbarrier wait before giving up
};

// Whether a query's certificate holds: |q|^2 = qq, the k-th exact distance among
// the recomputed references is D, every other reference scores at or above
// tau.  In single precision: E already doubles the bound on the score's error,
// and its second term covers the rounding of this arithmetic, below 2 (d + 16) u of
// the largest operand, and that of taking q and r relative to the centre (u of
// each coordinate, which moves |q - r|^2 by at most 4.1 u (|q|^2 + |r|^2)).  (In
// double it kept the slow pipe busy for a third of the re-rank.)  Overflow or
// NaN anywhere, and tau = -inf, refuse it; what fails for some D and tau fails
// for every larger D and smaller tau.
struct ScoreBound {
    float Dp;  // at least the real |q-r|^2 of any r with dist(r) <= D
    float E;   // bound on the error of any such r's score, and of the comparison
};
__device__ __forceinline__ ScoreBound score_bound(float eps_dot, int d, float qq, float tau, float D) {
    const float u = 1.0f / 16777216.0f;           // 2^-24
    const float m = float(d + 4) * u;             // rounding of the exact FP32 distance
    const float Dp = D * (1.0f + 2.0f * m);
    const float qn = sqrtf(qq);
    const float rho = qn + sqrtf(Dp);             // |r|
    const float eps = 2.0f * eps_dot + m;         // score error, relative
    const float big = qn * rho + rho * rho + fmaxf(Dp, qq);
    // first term: x2 safety; the last: operands, products and sums below 2^-126
    // may be taken for zero, each of the at most 3 (d + 1) <= 195 products and
    // sums at a loss of that much (relative bounds say nothing down there)
    const float E = 2.0f * eps * big + 4.0f * float(d + 18) * u * (big + fabsf(tau)) + 0x1p-112f;
    return ScoreBound{Dp, E};
}
__device__ __forceinline__ bool certifies(float eps_dot, int d, float qq, float tau, float D) {
    const ScoreBound b = score_bound(eps_dot, d, qq, tau, D);
    return (qq + tau) - b.E > b.Dp;               // false for NaN
}

// Order-preserving uint32 image of a score (negative scores included).
__device__ __forceinline__ uint32_t score_bits(float sc) {
    const uint32_t u = __float_as_uint(sc);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float bits_score(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// Entries of one part's list, and how many of them survive when it fills up
// (before it may lack room for 16 more).  Enough for every k the path takes.
constexpr int kT5Kept = 64;
constexpr int kT5Cap = 2 * kT5Kept + 16;

template <int MODE, int KP>
struct Tc5Shape {
    static constexpr int ESZ = MODE == TK_BRUTE_TF32 ? 4 : 2;
    static constexpr int KB = KP * ESZ;
    static constexpr int PL = MODE == TK_BRUTE_TF32 ? 1 : 2;
    static constexpr uint32_t A_BYTES = uint32_t(kT5Rows) * KB;
    static constexpr uint32_t B_BYTES = uint32_t(kT5Cols) * KB;
    static constexpr int KSTEPS = KB / 32;
    static constexpr size_t FIXED = size_t(PL) * A_BYTES + size_t(kT5Rows) * kT5MinStride * 2 + kT5Rows * sizeof(float);
    // reference tiles in flight: as many as fit, at most 4
    static constexpr int STAGES = (232448 - FIXED) / (PL * B_BYTES) < 4 ? int((232448 - FIXED) / (PL * B_BYTES)) : 4;
    static_assert(STAGES >= 3, "reference stages of the select kernel");
    static constexpr size_t SMEM = FIXED + size_t(STAGES) * PL * B_BYTES;
};

// A part's list of n >= kT5Kept entries (n <= kT5Cap), by the whole warp:
// lower its threshold to its kT5Kept-th smallest score and keep what scores
// below.  Returns (entries kept, threshold's bits).  By the list's own lane
// alone this took 0.5 ms.
static __device__ __noinline__ uint2 prune_hits(uint2* list, int n, int lane) {
    constexpr int E = (kT5Cap + 31) / 32;
    uint2 k[E];
    uint32_t u[E], lo = 0xFFFFFFFFu, hi = 0u;
    __syncwarp();
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const bool in = 32 * e + lane < n;
        k[e] = in ? list[32 * e + lane] : make_uint2(0u, 0u);
        u[e] = in ? score_bits(__uint_as_float(k[e].x)) : 0xFFFFFFFFu;
        lo = min(lo, u[e]);
        if (in) hi = max(hi, u[e]);
    }
    lo = __reduce_min_sync(0xFFFFFFFFu, lo);
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        int c = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) c += u[e] <= mid ? 1 : 0;
        c = __reduce_add_sync(0xFFFFFFFFu, c);
        if (c >= kT5Kept) hi = mid;
        else lo = mid + 1u;
    }
    int kept = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const unsigned m = __ballot_sync(0xFFFFFFFFu, u[e] < lo);
        if (u[e] < lo) list[kept + __popc(m & ((1u << lane) - 1u))] = k[e];
        kept += __popc(m);
    }
    __syncwarp();
    return make_uint2(uint32_t(kept), __float_as_uint(bits_score(lo)));
}

// 16 bits of a squared distance (the negative ones, errors of scores, are 0),
// ordered like it, and the largest distance with given bits.
constexpr uint32_t kT5CodeInf = 0xFF00u;
__device__ __forceinline__ uint16_t dist_code(float x) { return uint16_t(__float_as_uint(fmaxf(x, 0.f)) >> 15); }
__device__ __forceinline__ float code_end(uint32_t code) { return __uint_as_float((code << 15) | 0x7FFFu); }

// Threshold (a score) of a row whose minima's rank-th smallest has code `lo`,
// -inf where no certificate can come of it; see k_tc5_select.  By 4 lanes per
// row, each with a quarter of its minima, which stand for `groups` groups.
static __device__ __noinline__ float row_threshold(const uint16_t* mins, uint32_t lo, float qq, bool real, float eps_dot,
                                                   int d, int groups, int pstride) {
    float t = lo < kT5CodeInf ? code_end(lo) : kT5PadNorm;  // rounded up to the end of its 16-bit bucket
    // Where the scores' error is not small against t (clusters far apart), the
    // certificate may want lists that go on by that error; groups without a
    // reference that near tell whether they can hold what is there.  Where it
    // exceeds t there is none, see below.
    const float E = score_bound(eps_dot, d, qq, t - qq, t).E;
    const bool blurred = E > 0.0625f * t;
    if (__any_sync(0xFFFFFFFFu, blurred)) {
        const uint32_t end = min(uint32_t(dist_code(t + 1.01f * E)), kT5CodeInf - 1u);
        int c = 0;
        for (int i = 0; i < kT5Minima / 4; ++i) c += mins[i] <= end ? 1 : 0;
        c += __shfl_xor_sync(0xFFFFFFFFu, c, 1);
        c += __shfl_xor_sync(0xFFFFFFFFu, c, 2);
        const float most = float(groups) * (1.f - __expf(-float(kT5Parts * 96) / float(groups * pstride)));
        if (blurred && float(c) <= most) t = code_end(end);
    }
    // Low enough to keep the padding rows out.  (NaN scores have code 0 and are
    // no hits; such a row's |q|^2 is no certificate's.  Rows past the last query
    // take no hits: all their scores are equal.)
    const float low = fminf(t - qq, kT5PadNorm);
    return real && certifies(eps_dot, d, qq, low, 0.f) ? low : -__int_as_float(0x7f800000);
}

__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Candidate search of one block: 128 query rows against one slice of the
// references.
//
// A thread of the epilogue (warp w, lane l) reads 64 columns of one query row
// of every tile and keeps, by itself and without any barrier, the list of its
// references that score below a threshold: two instructions per score when
// there is no hit, which bounds the kernel together with the products.
//
// The threshold comes first.  Before its slice a block runs a sample of it,
// in which threads only keep minima of groups of scores, 128 per row, rounded
// up to 16 bits; the threshold is the rank-th smallest of a row's minima.  The
// groups being spread over the cloud, about rank * pstride references of the
// slice score below it; tc_layout picks both so that some 100 references (more
// for large k) of a row do over all slices.  Nothing depends on that: a list that fills up
// lowers its own threshold to its kT5Kept-th best, and whatever the threshold, the
// references that no list holds score at or above it, which is all that the
// certificate uses.  Rows whose threshold is too low for a certificate whatever
// the distances (clusters far apart: scores differ by less than their error)
// take no hits, and a block of such rows only waits for its products.
//
// 262,144 x 65,536, d=32, k=32, TF32: 3.1 ms; in whole waves of blocks 3.5 ms,
// of which it was measured: tensor pipe 45% busy, issue
// slots 51%: 4 epilogue warps per scheduler cannot cover the latency of their
// own minima, votes and branches.  (Before: a short sample, then per-row
// sorted lists kept up to date in the registers of 4-lane groups, a barrier
// per tile: 9.6 ms.)
template <int MODE, int KP>
__global__ void __launch_bounds__(kT5Threads, 1) k_tc5_select(const Tc5Args a) {
    using Sh = Tc5Shape<MODE, KP>;
    constexpr int PL = Sh::PL, KB = Sh::KB, KSTEPS = Sh::KSTEPS, STAGES = Sh::STAGES, CAP = kT5Cap;
    constexpr uint32_t A_BYTES = Sh::A_BYTES, B_BYTES = Sh::B_BYTES;
    constexpr uint32_t LBO = 128, SBO = 8 * KB;
    constexpr int NPROD = MODE == TK_BRUTE_TF32 ? 1 : 3;
    constexpr uint32_t IDESC = sm100::instr_desc(MODE == TK_BRUTE_TF32 ? 2u : 1u, kT5Rows, kT5Cols);

    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* sA = smem;                       // [PL][A_BYTES]
    unsigned char* sB = smem + PL * A_BYTES;        // [STAGES][PL][B_BYTES]
    uint16_t* sMin = reinterpret_cast<uint16_t*>(sB + STAGES * PL * B_BYTES);  // [kT5Rows][kT5MinStride]
    float* sThr = reinterpret_cast<float*>(sMin + kT5Rows * kT5MinStride);     // [kT5Rows]
    __shared__ __align__(8) uint64_t full_a, full_b[STAGES], mma_done[2], epi_done[2];
    __shared__ uint32_t tmem_base_sh;
    __shared__ volatile int some_row;  // whether a row of the block is searched
    constexpr int NEPI = 32 * kT5EpiWarps;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // row blocks of the head come first, one after another for each of its slices
    const bool in_tail = int(blockIdx.x) >= a.split_from * a.head.nsplit;
    const Tc5Slices sl = in_tail ? a.tail : a.head;
    const int in_part = int(blockIdx.x) - (in_tail ? a.split_from * a.head.nsplit : 0);
    const int part_rows = in_tail ? (a.nq + kT5Rows - 1) / kT5Rows - a.split_from : a.split_from;
    const int slice = in_part / part_rows;
    const int rblock = in_part - slice * part_rows + (in_tail ? a.split_from : 0);
    const int per = (a.tiles + sl.nsplit - 1) / sl.nsplit;
    const int tile0 = min(a.tiles, per * slice);
    const int ntiles = min(a.tiles, tile0 + per) - tile0;
    const int npre = (ntiles + sl.pstride - 1) / sl.pstride;  // sampled tiles
    const int nseq = npre + ntiles;  // tiles through the pipeline
    auto tile_of = [&](int t) { return tile0 + (t < npre ? t * sl.pstride : t - npre); };

    if (tid == 0) {
        some_row = 0;
        sm100::mbar_init(&full_a, 1);
        for (int i = 0; i < STAGES; ++i) sm100::mbar_init(&full_b[i], 1);
        sm100::mbar_init(&mma_done[0], 1);
        sm100::mbar_init(&mma_done[1], 1);
        sm100::mbar_init(&epi_done[0], kT5EpiWarps);
        sm100::mbar_init(&epi_done[1], kT5EpiWarps);
        sm100::mbar_fence_init();
    }
    for (int i = tid; i < kT5Rows * kT5MinStride; i += kT5Threads) sMin[i] = 0xFFFFu;
    if (warp == kT5EpiWarps) sm100::tmem_alloc(&tmem_base_sh, 512);
    sm100::tc_fence_before();
    __syncthreads();
    sm100::tc_fence_after();
    const uint32_t tmem = tmem_base_sh;

    if (warp == kT5EpiWarps) {
        // ------------------------------------------------ producer / MMA issuer
        if (lane == 0 && nseq > 0) {
            bool ok = true;
            // what this thread started and has not yet seen complete (waited
            // for, within bounds, if it gives up): tiles copied in, products
            bool a_pending = true;
            int b_issued = 0, b_waited = 0, m_issued = 0, m_waited = 0;
            auto load = [&](int t) {
                const int st = t % STAGES;
                const size_t tb = (size_t)tile_of(t) * B_BYTES;
                sm100::mbar_arrive_expect_tx(&full_b[st], PL * B_BYTES);
                sm100::bulk_g2s(sB + (st * PL) * B_BYTES, a.b_hi + tb, B_BYTES, &full_b[st]);
                if (PL == 2) sm100::bulk_g2s(sB + (st * PL + 1) * B_BYTES, a.b_lo + tb, B_BYTES, &full_b[st]);
                b_issued = t + 1;
            };
            sm100::mbar_arrive_expect_tx(&full_a, PL * A_BYTES);
            sm100::bulk_g2s(sA, a.a_hi + (size_t)rblock * A_BYTES, A_BYTES, &full_a);
            if (PL == 2) sm100::bulk_g2s(sA + A_BYTES, a.a_lo + (size_t)rblock * A_BYTES, A_BYTES, &full_a);
            for (int t = 0; t < STAGES && t < nseq; ++t) load(t);
            for (int t = 0; t < nseq; ++t) {
                const int st = t % STAGES, ac = t & 1;
                ok = sm100::mbar_wait(&full_b[st], (t / STAGES) & 1, a.max_tries);
                if (!ok) break;
                b_waited = t + 1;
                if (t == 0) {
                    ok = sm100::mbar_wait(&full_a, 0, a.max_tries);
                    if (!ok) break;
                    a_pending = false;
                }
                if (t >= 2) {
                    ok = sm100::mbar_wait(&epi_done[ac], ((t - 2) >> 1) & 1, a.max_tries);
                    if (!ok) break;
                }
                sm100::tc_fence_after();
                const uint32_t dtm = tmem + uint32_t(ac * kT5Cols);
                const uint32_t a0 = sm100::smem_u32(sA);
                const uint32_t b0 = sm100::smem_u32(sB + (st * PL) * B_BYTES);
#pragma unroll
                for (int ks = 0; ks < KSTEPS; ++ks) {
#pragma unroll
                    for (int pr = 0; pr < NPROD; ++pr) {
                        const uint32_t pa = pr == 2 ? A_BYTES : 0u;  // lo(A) for lo*hi
                        const uint32_t pb = pr == 1 ? B_BYTES : 0u;  // lo(B) for hi*lo
                        const uint64_t ad = sm100::smem_desc(a0 + pa + uint32_t(ks) * 256u, LBO, SBO);
                        const uint64_t bd = sm100::smem_desc(b0 + pb + uint32_t(ks) * 256u, LBO, SBO);
                        const uint32_t acc = (ks | pr) != 0 ? 1u : 0u;
                        if (MODE == TK_BRUTE_TF32) sm100::mma_tf32(dtm, ad, bd, IDESC, acc);
                        else sm100::mma_bf16(dtm, ad, bd, IDESC, acc);
                    }
                }
                sm100::mma_commit(&mma_done[ac]);
                m_issued = t + 1;
                // while these products run: the stage of the ones before them
                // takes its next tile
                if (t >= 1) {
                    ok = sm100::mbar_wait(&mma_done[ac ^ 1], ((t - 1) >> 1) & 1, a.max_tries);
                    if (!ok) break;
                    m_waited = t;
                    if (t - 1 + STAGES < nseq) load(t - 1 + STAGES);
                }
            }
            if (!ok) {
                // A wait ran out: flag it (the re-rank then certifies nothing
                // and the exact kernel answers every query), then let this
                // thread's own copies and matrix products still in flight
                // land -- each wait bounded by the default poll count --
                // before the block frees its tensor memory and exits.
                atomicOr(a.err, kTcErrTimeout);
                if (a_pending) sm100::mbar_wait(&full_a, 0, kT5MaxTries);
                for (int t = b_waited; t < b_issued; ++t)
                    sm100::mbar_wait(&full_b[t % STAGES], (t / STAGES) & 1, kT5MaxTries);
                for (int t = m_waited; t < m_issued; ++t)
                    sm100::mbar_wait(&mma_done[t & 1], (t >> 1) & 1, kT5MaxTries);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------- epilogue warps
        // Thread (warp w, lane l): accumulator lane 32 (w & 3) + l, i.e. query
        // row `myrow`, columns 64 (w >> 2) .. + 63.
        const int quarter = warp & 3, part = warp >> 2;
        const int myrow = 32 * quarter + lane;
        const uint32_t trow = tmem + (uint32_t(32 * quarter) << 16) + uint32_t(part * 64);
        auto bar_all = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(NEPI) : "memory"); };
        // |q|^2 of this thread's row, and of the row whose threshold it helps to find
        const int grow = 32 * quarter + 8 * part + (lane >> 2), gl = lane & 3;
        const float qq = rblock * kT5Rows + myrow < a.nq ? __ldg(a.qnorm + rblock * kT5Rows + myrow) : 0.f;
        bool alive = true;
        float va[32], vb[32];  // the thread's first and last 32 scores of a tile
        // Waits for pipeline step t's products; false when the wait ran out.
        auto products = [&](int t) {
            int ok = 1;
            if (lane == 0) ok = sm100::mbar_wait(&mma_done[t & 1], (t >> 1) & 1, a.max_tries);
            return __shfl_sync(0xFFFFFFFFu, ok, 0) != 0;
        };
        // The same, and loads both halves; the second is still on its way.
        auto begin = [&](int t) {
            if (!products(t)) return false;
            sm100::tc_fence_after();
            const uint32_t at = trow + uint32_t((t & 1) * kT5Cols);
            sm100::tmem_ld32(at, va);
            sm100::tmem_wait32(va);
            sm100::tmem_ld32(at + 32u, vb);
            return true;
        };
        // The second half has arrived: the accumulator goes back to the issuer.
        auto rest = [&](int t) {
            sm100::tmem_wait32(vb);
            sm100::tc_fence_before();
            __syncwarp();
            if (lane == 0) sm100::mbar_arrive(&epi_done[t & 1]);
        };
        // minima of columns 16 c + 3 j .. + 2 (j < 5) of a half, and of all 16
        auto min16 = [&](const float (&v)[32], int c, float (&g)[5]) {
            const float* x = v + 16 * c;
#pragma unroll
            for (int j = 0; j < 5; ++j) g[j] = min3(x[3 * j], x[3 * j + 1], x[3 * j + 2]);
            return fminf(min3(g[0], g[1], g[2]), min3(g[3], g[4], x[15]));
        };
        float g[5];
        // sample: minima of groups of `tpg` tiles' scores, of one tile, or (short slices) of 16 scores
        const int tpg = (npre + 31) / 32;
        float run = __int_as_float(0x7f800000);
        for (int t = 0; t < npre; ++t) {
            alive = begin(t);
            if (!alive) break;
            const float m0 = min16(va, 0, g), m1 = min16(va, 1, g);
            rest(t);
            const float m2 = min16(vb, 0, g), m3 = min16(vb, 1, g);
            uint16_t* out = sMin + myrow * kT5MinStride;
            if (npre <= 8) {
                out[(t * 4 + 0) * 4 + part] = dist_code(qq + m0);
                out[(t * 4 + 1) * 4 + part] = dist_code(qq + m1);
                out[(t * 4 + 2) * 4 + part] = dist_code(qq + m2);
                out[(t * 4 + 3) * 4 + part] = dist_code(qq + m3);
            } else {
                run = fminf(min3(run, m0, m1), fminf(m2, m3));
                if ((t + 1) % tpg == 0 || t + 1 == npre) {
                    out[(t / tpg) * 4 + part] = dist_code(qq + run);
                    run = __int_as_float(0x7f800000);
                }
            }
        }
        bar_all();
        {
            // the rank-th smallest of a row's minima, by 4 lanes: bisection on their 16-bit images
            const uint16_t* mins = sMin + grow * kT5MinStride + gl * (kT5Minima / 4);
            uint32_t m[kT5Minima / 8];
#pragma unroll
            for (int i = 0; i < kT5Minima / 8; ++i) m[i] = *reinterpret_cast<const uint32_t*>(mins + 2 * i);
            uint32_t lo = 0u, hi = 0xFFFFu;
#pragma unroll 1
            for (int it = 0; it < 16; ++it) {
                const uint32_t mid = (lo + hi) >> 1;
                int c = 0;
#pragma unroll
                for (int i = 0; i < kT5Minima / 8; ++i) c += ((m[i] & 0xFFFFu) <= mid ? 1 : 0) + ((m[i] >> 16) <= mid ? 1 : 0);
                c += __shfl_xor_sync(0xFFFFFFFFu, c, 1);
                c += __shfl_xor_sync(0xFFFFFFFFu, c, 2);
                if (c >= sl.rank) hi = mid;
                else lo = min(mid + 1u, 0xFFFFu);
            }
            const int grow_q = rblock * kT5Rows + grow;
            const bool real = grow_q < a.nq;
            const float low = row_threshold(mins, lo, real ? __ldg(a.qnorm + grow_q) : 0.f, real, a.eps_dot, a.d,
                                            npre <= 8 ? 16 * npre : 4 * ((npre + tpg - 1) / tpg), sl.pstride);
            if (gl == 0) sThr[grow] = low;
            if (__any_sync(0xFFFFFFFFu, low > -__int_as_float(0x7f800000)) && lane == 0) some_row = 1;
        }
        bar_all();
        const int row = rblock * kT5Rows + myrow;
        const long long lidx =
            (first_slice(row, a.split_from, a.head.nsplit, a.tail.nsplit) + slice) * kT5Parts + part;
        uint2* list = a.hits + lidx * CAP;
        float thr = sThr[myrow];
        int cnt = 0;
        // Hits of a half (32 columns from col0 on).  Branches are taken by the
        // whole warp (votes): few of its 512 scores of 16 columns are hits,
        // and the tests narrow down on them in two steps, 16 columns and 3.
        auto collect = [&](const float (&v)[32], uint32_t tile, uint32_t col0) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if (!__any_sync(0xFFFFFFFFu, min16(v, c, g) < thr)) continue;
#pragma unroll
                for (int j = 0; j < 6; ++j) {
                    if (!__any_sync(0xFFFFFFFFu, (j < 5 ? g[j < 5 ? j : 0] : v[16 * c + 15]) < thr)) continue;
#pragma unroll
                    for (int i = 16 * c + 3 * j; i < 16 * c + (j < 5 ? 3 * j + 3 : 16); ++i) {
                        if (v[i] < thr) {
                            list[cnt] = make_uint2(__float_as_uint(v[i]), packed_ref(tile, col0 + uint32_t(i), uint32_t(a.tiles)));
                            ++cnt;
                        }
                    }
                }
                unsigned full = __ballot_sync(0xFFFFFFFFu, cnt > CAP - 16);
                while (full) {
                    const int src = __ffs(full) - 1;
                    full &= full - 1u;
                    const int n = __shfl_sync(0xFFFFFFFFu, cnt, src);
                    uint2* at = reinterpret_cast<uint2*>(
                        __shfl_sync(0xFFFFFFFFu, reinterpret_cast<unsigned long long>(list), src));
                    const uint2 p = prune_hits(at, n, lane);
                    if (lane == src) {
                        cnt = int(p.x);
                        thr = __uint_as_float(p.y);
                    }
                }
            }
        };
        // A block without a row to search lets the products pass.  (The issuer
        // looking whether it could stop took every block 13% more time.)
        int next = npre;
        if (some_row == 0) {
            for (; alive && next < nseq; ++next) {
                alive = products(next);
                if (alive && lane == 0) sm100::mbar_arrive(&epi_done[next & 1]);
            }
        }
        for (int t = next; alive && t < nseq; ++t) {
            alive = begin(t);
            if (!alive) break;
            const uint32_t tile = uint32_t(tile_of(t)), col0 = uint32_t(64 * part);
            collect(va, tile, col0);
            rest(t);
            collect(vb, tile, col0 + 32u);
        }
        if (!alive && lane == 0) atomicOr(a.err, kTcErrTimeout);
        a.counts[lidx] = cnt;
        a.thr[lidx] = thr;
    }
    // teardown: everyone done with tensor memory
    sm100::tc_fence_before();
    __syncthreads();
    sm100::tc_fence_after();
    if (warp == kT5EpiWarps) sm100::tmem_dealloc(tmem, 512);
}

// Shared memory of the mma.sync candidate search for (mode, KP, C).
inline size_t select_smem_bytes(int mode, int KP, int C) {
    const int KW = (mode == TK_BRUTE_TF32) ? KP : KP / 2;
    const int PLANES = (mode == TK_BRUTE_TF32) ? 1 : 2;
    return sizeof(uint32_t) * PLANES * kCols * (KW + 4) + sizeof(float) * kCols +
           sizeof(float) * kRows * (kCols + 4) + (sizeof(float) + sizeof(int32_t)) * size_t(C) * kRows;
}
template <int MODE, int KP, int C>
size_t select_smem_bytes() {
    return select_smem_bytes(MODE, KP, C);
}

struct RerankArgs {
    const float* ref;     // [n, d] float32 originals
    const float* q;       // [nq, d]
    int n, nq, d, k, C, nsplit;
    int split_from, tail_nsplit;  // tcgen05 search, see first_slice (nsplit: the head's)
    const float* cand_s;  // mma.sync search: [nq, nsplit, C]
    const int32_t* cand_i;
    const float* tau;     // [nq, nsplit]
    const float* qnorm;   // |q|^2
    int keep;             // tcgen05 search: references per query worth recomputing
    const uint2* hits;    // see Tc5Args
    const int* counts;
    const float* thr;
    float eps_dot;        // relative error bound of the tensor-core dot product
    float* out_d;
    int32_t* out_i;
    int* fail_count;
    int* fail_list;
    const int* err;       // candidate kernel gave up (bounded wait ran out): certify nothing
};

// Exact FP32 squared distance of reference row rr to the query (the
// reference's arithmetic: coordinate differences squared and summed in
// coordinate order); rows read 16 bytes at a time when `vec` (d % 4 == 0,
// 16-byte aligned rows), which cut the re-rank of the 262,144 x 65,536, d=32
// workload from 0.96 to ~0.45 ms.
__device__ __forceinline__ float rerank_dist(const float* __restrict__ qrow, const float* __restrict__ rr, int d,
                                             bool vec) {
    float acc;
    if (vec) {
        const float4* q4 = reinterpret_cast<const float4*>(qrow);
        const float4* r4 = reinterpret_cast<const float4*>(rr);
        float4 qv = __ldg(q4), rv = __ldg(r4);
        float t = __fsub_rn(qv.x, rv.x);
        acc = __fmul_rn(t, t);
        t = __fsub_rn(qv.y, rv.y);
        acc = __fadd_rn(acc, __fmul_rn(t, t));
        t = __fsub_rn(qv.z, rv.z);
        acc = __fadd_rn(acc, __fmul_rn(t, t));
        t = __fsub_rn(qv.w, rv.w);
        acc = __fadd_rn(acc, __fmul_rn(t, t));
        for (int c = 1; c < (d >> 2); ++c) {
            qv = __ldg(q4 + c);
            rv = __ldg(r4 + c);
            t = __fsub_rn(qv.x, rv.x);
            acc = __fadd_rn(acc, __fmul_rn(t, t));
            t = __fsub_rn(qv.y, rv.y);
            acc = __fadd_rn(acc, __fmul_rn(t, t));
            t = __fsub_rn(qv.z, rv.z);
            acc = __fadd_rn(acc, __fmul_rn(t, t));
            t = __fsub_rn(qv.w, rv.w);
            acc = __fadd_rn(acc, __fmul_rn(t, t));
        }
    } else {
        float t = __fsub_rn(qrow[0], rr[0]);
        acc = __fmul_rn(t, t);
        for (int c = 1; c < d; ++c) {
            t = __fsub_rn(qrow[c], rr[c]);
            acc = __fadd_rn(acc, __fmul_rn(t, t));
        }
    }
    return acc;
}

// Certificate of a query (|q|^2 = qq) whose k-th exact distance among the
// recomputed references is D; every other reference scores at or above tau.
__device__ __forceinline__ bool certified(const RerankArgs& a, float qq, float tau, float D) {
    if (a.err && *a.err) return false;
    if (!(qq < kTcNormLimit)) return false;  // see kTcNormLimit (also NaN / inf coordinates)
    if (tau == __int_as_float(0x7f800000)) return true;  // every other reference was recomputed
    return certifies(a.eps_dot, a.d, qq, tau, D);
}

// One warp per query: exact distances of the candidates, top-k, certificate.
template <int R>
__global__ void __launch_bounds__(256) k_tc_rerank(const RerankArgs a) {
    const int lane = threadIdx.x & 31;
    const int qi = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
    if (qi >= a.nq) return;
    TopK<float, 32, R> list;
    list.init(a.k, lane);
    Key<float> worst = Key<float>::sentinel();
    const float* qrow = a.q + (long long)qi * a.d;
    const int total = a.C * a.nsplit;
    const long long base = (long long)qi * total;
    const bool vec =
        (a.d & 3) == 0 && ((reinterpret_cast<uintptr_t>(a.ref) | reinterpret_cast<uintptr_t>(a.q)) & 15) == 0;
    for (int e0 = 0; e0 < total; e0 += 32) {
        const int e = e0 + lane;
        Key<float> mine = Key<float>::sentinel();
        const int r = e < total ? a.cand_i[base + e] : -1;
        if (r >= 0) mine = Key<float>::make(rerank_dist(qrow, a.ref + (long long)r * a.d, a.d, vec), uint32_t(r));
        worst = offer<float, 32, R>(list, mine, worst, 0xFFFFFFFFu, lane, 0);
    }
    list.store(a.k, lane, a.out_d, a.out_i, qi);
    const float qq = a.qnorm[qi];
    if (lane == 0) {
        float tau = __int_as_float(0x7f800000);
        for (int s = 0; s < a.nsplit; ++s) tau = fminf(tau, a.tau[(long long)qi * a.nsplit + s]);
        if (!certified(a, qq, tau, worst.dist())) {
            const int slot = atomicAdd(a.fail_count, 1);
            a.fail_list[slot] = qi;
        }
    }
}

// The same for the lists of k_tc5_select (k <= 32).  Where they hold far more
// references than were wanted (clustered clouds), only those up to the
// keep-th best score are recomputed, and that score joins the lists'
// thresholds in tau.
//
// Bound by the gather of the listed rows (L1 92% busy at d=32).  From
// kStagedDims dimensions on, where a row is worth more than the arithmetic, the
// hits are held in registers and some k + 16 of the best scores are recomputed
// first; of the others only those that the certificate's bound, taken at their
// own score, does not put beyond the k-th distance.  262,144 x 65,536, d=32,
// k=32, whole call: TF32 3.59 -> 3.51 ms, BF16 4.02 -> 3.91; 20,000 x 30,000
// 0.52 -> 0.47; d=13 the same, d=8 1 to 7% slower.
constexpr int kStagedDims = 24;

static __global__ void __launch_bounds__(256, 4) k_tc5_rerank(const RerankArgs a) {
    constexpr int CAP = kT5Cap, HELD = 8;
    __shared__ Key<float> bufs[8][64];
    __shared__ uint32_t todo[8][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int qi = blockIdx.x * 8 + w;
    if (qi >= a.nq) return;
    const int nl = (qi < (long long)a.split_from * kT5Rows ? a.nsplit : a.tail_nsplit) * kT5Parts;
    const long long list0 = first_slice(qi, a.split_from, a.nsplit, a.tail_nsplit) * kT5Parts;
    const int* counts = a.counts + list0;
    const uint2* hits = a.hits + list0 * CAP;
    int total = 0;
    float tau = __int_as_float(0x7f800000);
    for (int l = lane; l < nl; l += 32) {
        total += counts[l];
        tau = fminf(tau, a.thr[list0 + l]);
    }
    total = __reduce_add_sync(0xFFFFFFFFu, total);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) tau = fminf(tau, __shfl_xor_sync(0xFFFFFFFFu, tau, o));
    uint32_t cut = 0xFFFFFFFFu;  // image of the last score recomputed
    if (total > 2 * a.keep) {
        uint32_t lo = 0xFFFFFFFFu, hi = 0u;
        for (int l = 0; l < nl; ++l) {
            const int c = counts[l];
            for (int e = lane; e < c; e += 32) {
                const uint32_t u = score_bits(__uint_as_float(hits[l * CAP + e].x));
                lo = min(lo, u);
                hi = max(hi, u);
            }
        }
        lo = __reduce_min_sync(0xFFFFFFFFu, lo);
        hi = __reduce_max_sync(0xFFFFFFFFu, hi);
        while (lo < hi) {
            const uint32_t mid = lo + ((hi - lo) >> 1);
            int below = 0;
            for (int l = 0; l < nl; ++l) {
                const int c = counts[l];
                for (int e = lane; e < c; e += 32)
                    below += score_bits(__uint_as_float(hits[l * CAP + e].x)) <= mid ? 1 : 0;
            }
            below = __reduce_add_sync(0xFFFFFFFFu, below);
            if (below >= a.keep) hi = mid;
            else lo = mid + 1u;
            if (below >= a.keep && below <= a.keep + 32) break;  // near enough
        }
        // (unless only the rest can give the certificate, see k_tc5_select)
        if (certifies(a.eps_dot, a.d, a.qnorm[qi], bits_score(hi), 0.f)) {
            cut = hi;
            tau = fminf(tau, bits_score(cut));
        }
    }
    WarpList<float, 1> wl;
    wl.init(a.k, bufs[w], lane);
    const float* qrow = a.q + (long long)qi * a.d;
    const bool vec =
        (a.d & 3) == 0 && ((reinterpret_cast<uintptr_t>(a.ref) | reinterpret_cast<uintptr_t>(a.q)) & 15) == 0;
    int waiting = 0;
    auto evaluate = [&](int m) {
        Key<float> mine = Key<float>::sentinel();
        if (lane < m) {
            const uint32_t r = todo[w][lane];
            mine = Key<float>::make(rerank_dist(qrow, a.ref + (long long)r * a.d, a.d, vec), r);
        }
        wl.offer(mine, lane);
    };
    auto collect = [&](bool take, uint32_t r) {
        const unsigned m = __ballot_sync(0xFFFFFFFFu, take);
        if (!m) return;
        if (take) todo[w][waiting + __popc(m & ((1u << lane) - 1u))] = r;
        waiting += __popc(m);
        __syncwarp();
        if (waiting >= 32) {
            evaluate(32);
            const uint32_t rest = todo[w][32 + lane];
            __syncwarp();
            waiting -= 32;
            if (lane < waiting) todo[w][lane] = rest;
            __syncwarp();
        }
    };
    auto finish = [&]() {
        if (waiting > 0) evaluate(waiting);
        waiting = 0;
        __syncwarp();
        wl.flush(lane);
    };
    const float qq = a.qnorm[qi];
    if (a.d >= kStagedDims && nl <= 8 && total > a.k + 48 && total <= 32 * HELD) {
        uint2 hit[HELD];  // hit h of all lists on lane h % 32
        const int mine = lane < nl ? counts[lane] : 0;
#pragma unroll
        for (int t = 0; t < HELD; ++t) {
            int e = t * 32 + lane, l = 0;
            for (int i = 0; i < nl; ++i) {
                const int c = __shfl_sync(0xFFFFFFFFu, mine, i);
                if (l == i && e >= c) {
                    e -= c;
                    ++l;
                }
            }
            hit[t] = make_uint2(0xFFFFFFFFu, 0u);
            if (l < nl) {
                hit[t] = hits[l * CAP + e];
                hit[t].x = score_bits(__uint_as_float(hit[t].x));
            }
        }
        // the score that some k + 16 hits reach
        uint32_t lo = 0xFFFFFFFFu, hi = 0u;
#pragma unroll
        for (int t = 0; t < HELD; ++t) {
            lo = min(lo, hit[t].x);
            hi = max(hi, t * 32 + lane < total ? hit[t].x : 0u);
        }
        lo = __reduce_min_sync(0xFFFFFFFFu, lo);
        hi = __reduce_max_sync(0xFFFFFFFFu, hi);
        while (lo < hi) {
            const uint32_t mid = lo + ((hi - lo) >> 1);
            int below = 0;
#pragma unroll
            for (int t = 0; t < HELD; ++t) below += hit[t].x <= mid ? 1 : 0;
            below = __reduce_add_sync(0xFFFFFFFFu, below);
            if (below >= a.k + 8) hi = mid;
            else lo = mid + 1u;
            if (below >= a.k + 8 && below <= a.k + 24) break;
        }
        const uint32_t first = hi;
#pragma unroll
        for (int t = 0; t < HELD; ++t) collect(t * 32 + lane < total && hit[t].x <= first, hit[t].y);
        finish();
        const float D = wl.worst.dist();
#pragma unroll
        for (int t = 0; t < HELD; ++t) {
            const float sc = bits_score(hit[t].x);
            collect(t * 32 + lane < total && hit[t].x > first && hit[t].x <= cut &&
                        (isinf(sc) || !certified(a, qq, sc, D)), hit[t].y);
        }
    } else {
        for (int l = 0; l < nl; ++l) {
            const int c = counts[l];
            for (int e0 = 0; e0 < c; e0 += 32) {
                const uint2 k = e0 + lane < c ? hits[l * CAP + e0 + lane] : make_uint2(0u, 0u);
                collect(e0 + lane < c && score_bits(__uint_as_float(k.x)) <= cut, k.y);
            }
        }
    }
    finish();
    wl.list.store(a.k, lane, a.out_d, a.out_i, qi);
    if (lane == 0 && !certified(a, qq, tau, wl.worst.dist())) {
        const int slot = atomicAdd(a.fail_count, 1);
        a.fail_list[slot] = qi;
    }
}

template <int MODE, int KP>
int launch_tc5(const Tc5Args& a, int qblocks, cudaStream_t s) {
    using Sh = Tc5Shape<MODE, KP>;
    const void* fn = reinterpret_cast<const void*>(&k_tc5_select<MODE, KP>);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(Sh::SMEM));
    if (e != cudaSuccess) return fail(TK_ECUDA, std::string("tcgen05 select smem: ") + cudaGetErrorString(e));
    const int grid = a.split_from * a.head.nsplit + (qblocks - a.split_from) * a.tail.nsplit;
    k_tc5_select<MODE, KP><<<grid, kT5Threads, Sh::SMEM, s>>>(a);
    return TK_OK;
}

template <int MODE, int KP, int C>
int launch_select(const TcArgs& a, int qblocks, cudaStream_t s) {
    const size_t smem = select_smem_bytes<MODE, KP, C>();
    const void* fn = reinterpret_cast<const void*>(&k_tc_select<MODE, KP, C>);
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e != cudaSuccess) return fail(TK_ECUDA, std::string("tc select smem: ") + cudaGetErrorString(e));
    k_tc_select<MODE, KP, C><<<dim3(qblocks, a.nsplit), kThreads, smem, s>>>(a);
    return TK_OK;
}

template <int MODE, int KP>
int dispatch_c(const TcArgs& a, int qblocks, cudaStream_t s) {
    switch (a.C) {
        case 16: return launch_select<MODE, KP, 16>(a, qblocks, s);
        case 32: return launch_select<MODE, KP, 32>(a, qblocks, s);
        case 64: return launch_select<MODE, KP, 64>(a, qblocks, s);
        case 128: return launch_select<MODE, KP, 128>(a, qblocks, s);
        default: return fail(TK_EUNSUPPORTED, "tensor-core modes support k <= 64");
    }
}

template <int MODE>
int dispatch_kp(const TcArgs& a, int qblocks, cudaStream_t s) {
    switch (a.KP) {
        case 8:
            if constexpr (MODE == TK_BRUTE_TF32) return dispatch_c<MODE, 8>(a, qblocks, s);
            break;
        case 16: return dispatch_c<MODE, 16>(a, qblocks, s);
        case 32: return dispatch_c<MODE, 32>(a, qblocks, s);
        case 64: return dispatch_c<MODE, 64>(a, qblocks, s);
        default: break;
    }
    return fail(TK_EUNSUPPORTED, "tensor-core modes support d <= 64");
}

// Entry points of the candidate kernels, one unit each.
int tc5_dispatch_tf32(const Tc5Args& a, int KP, int qblocks, cudaStream_t s);       // brute_tc5_tf32.cu
int tc5_dispatch_tf32_deep(const Tc5Args& a, int KP, int qblocks, cudaStream_t s);  // brute_tc5_tf32_deep.cu
int tc5_dispatch_bf16(const Tc5Args& a, int KP, int qblocks, cudaStream_t s);  // brute_tc5_bf16.cu
int tc_select_dispatch(const TcArgs& a, int mode, int qblocks, cudaStream_t s);          // brute_tc_mma.cu

}  // namespace tcx
}  // namespace tk
