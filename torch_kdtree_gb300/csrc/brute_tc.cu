// Tensor-core brute force: candidate search with q.r on tensor cores, exact
// FP32 re-rank, and a per-query certificate that the answer equals the exact
// search; uncertified queries are recomputed by the exact kernel.
//
//   score(q, r) = |r|^2 - 2 q.r   (ranks like |q - r|^2 for a fixed query)
//
// 0. k_tc5_centre: the point that q and r are taken relative to (tcgen05 path).
// 1. k_tc_pack: operands for the tensor cores (TF32 rounded to nearest, or a
//    BF16 hi/lo split x = hi + lo) and |x|^2 in FP32.
// 2. k_tc5_select (brute_tc_kernels.cuh): tcgen05 products of 128 queries and
//    256 references at a time; every row collects the references that score
//    below a sampled threshold tau.  Depths and k that it does not take go to
//    k_tc_select: a block owns 128 queries and one slice of the references;
//    tiles of 128 references are multiplied with mma.sync (TF32 m16n8k8 or
//    BF16 m16n8k16 with three products hi*hi + hi*lo + lo*hi, FP32 accumulate),
//    the score tile goes through shared memory, and one thread per query keeps
//    the C = over-fetch best scores of its row (C >= 2k) plus the row
//    threshold tau (the C-th score; +inf while fewer than C were seen).
// 3. k_tc5_rerank / k_tc_rerank: one warp per query recomputes the exact distance of every
//    candidate with the reference arithmetic (sqdist order, no fused
//    multiply-add), keeps the k best (distance, index) keys, and certifies:
//    with D = k-th exact distance, E = bound on |score_tc - score_exact| for
//    any reference that could reach D, and tau = min over slices, the answer
//    is the exact one if |q|^2 + tau - E > D / (1 - m).  (A reference outside
//    every list has score_tc >= tau, hence |q - r|^2 >= |q|^2 + tau - E.)
// 4. Uncertified queries are listed and recomputed by the exact kernel.
//
// Kernels and launch templates: brute_tc_kernels.cuh; the candidate kernels
// are instantiated in brute_tc5_tf32.cu, brute_tc5_tf32_deep.cu,
// brute_tc5_bf16.cu (tcgen05) and brute_tc_mma.cu (mma.sync), compiled in
// parallel.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <string>
#include <vector>

#include "brute_tc.cuh"
#include "brute_tc_kernels.cuh"

namespace tk {
using namespace tcx;
namespace {

struct TcWs {
    size_t a_pack, b_pack, a_lo, b_lo, rnorm, qnorm, centre, fail_list, brute, total;
    size_t cand_s, cand_i, tau;  // mma.sync search
    size_t hits, counts, thr;    // tcgen05 search
    int KP, C, nsplit, wanted;
    int split_from;          // tcgen05 search: see first_slice
    Tc5Slices head, tail;
    bool tc5;  // tcgen05 path
};

// tcgen05 path: K = d + 1 (augmented), padded to the MMA's K step.
bool tc5_eligible(int d, int k, int mode) {
    if (k > 32) return false;
    return mode == TK_BRUTE_TF32 ? (d + 1 <= 40) : (d + 1 <= 48);
}
int tc5_kp(int d, int mode) {
    const int step = mode == TK_BRUTE_TF32 ? 8 : 16;
    return (d + 1 + step - 1) / step * step;
}

int tc_kp(int d, int mode) {
    const int step = mode == TK_BRUTE_TF32 ? 8 : 16;
    int kp = (d + step - 1) / step * step;
    if (kp <= 16) return kp <= 8 && mode == TK_BRUTE_TF32 ? 8 : 16;
    if (kp <= 32) return 32;
    if (kp <= 64) return 64;
    return 128;
}

int tc_over(int k) {
    int c = 16;
    while (c < 2 * k) c <<= 1;
    return c;
}

TcWs tc_layout(int64_t n, int64_t nq, int d, int k, int mode, int sms) {
    TcWs w{};
    w.tc5 = tc5_eligible(d, k, mode);
    w.KP = w.tc5 ? tc5_kp(d, mode) : tc_kp(d, mode);
    w.C = tc_over(k);
    const size_t es = mode == TK_BRUTE_TF32 ? 4 : 2;
    size_t o = 0;
    if (w.tc5) {
        const int qblocks = int((nq + kT5Rows - 1) / kT5Rows);
        // Slices of the references per row block, and the sample that gives a
        // slice's threshold: `wanted` references of a row are to score below
        // the thresholds of its slices together (the certificate wants about
        // 2k with room), by the `rank`-th smallest minimum of every pstride-th
        // tile.  The threshold scatters by 1 / sqrt(rank), and every reference
        // below it costs a list entry and an exact distance.  262,144 x 65,536,
        // d=32, ms for (wanted, rank): TF32 k=16 (150, 25) 3.70, (100, 16)
        // 3.38, (100, 12) 3.27, (80, 12) 3.46, where some rows miss their
        // certificate; k=32 (5k, 25) 3.80, (4k, 20) 3.53, (4.5k, 12) 3.71;
        // BF16 k=32 (5k, 25) 4.34, (4k, 20) 4.12, (5k, 12) 4.00.
        const int64_t tiles = (n + kT5Cols - 1) / kT5Cols;
        const int most = int(std::min<int64_t>(24, std::max<int64_t>(1, tiles / 8)));
        // small calls, where it costs little, want more: their many short
        // slices scatter more, and TF32's error is large against the spacing
        // of near neighbours in few dimensions
        double wanted = std::max(100.0, (mode == TK_BRUTE_TF32 ? 4.0 : 5.0) * k);
        const double rank = mode == TK_BRUTE_TF32 && wanted < 6.0 * k ? 20.0 : 12.0;
        if (qblocks <= (mode == TK_BRUTE_TF32 && d <= 8 ? sms : sms / 8)) wanted = std::max(wanted, 16.0 * k);
        w.wanted = int(wanted);
        constexpr double kBlockTiles = 16.0;  // a block's start and its thresholds, in tiles
        auto slices = [&](int ns, double below) {
            const int64_t per = (tiles + ns - 1) / ns;
            Tc5Slices sl;
            sl.nsplit = ns;
            sl.pstride = per >= 64 ? std::max(1, std::min(16, int(below / rank))) : 1;
            // of at most 0.8 of the minima there are (see k_tc5_select)
            const int64_t pre = (per + sl.pstride - 1) / sl.pstride;
            const int minima = int(pre <= 8 ? 16 * pre : std::min<int64_t>(kT5Minima, 4 * std::min<int64_t>(pre, 32)));
            sl.rank = std::max(8, std::min({64, minima * 4 / 5, int(below / sl.pstride + 0.5)}));
            return sl;
        };
        // time of so many row blocks in ns slices each, in whole passes over the references
        auto cost = [&](int blocks, const Tc5Slices& sl) {
            return ((1.0 + 1.0 / sl.pstride) / sl.nsplit + kBlockTiles / double(tiles)) * std::ceil(double(blocks) * sl.nsplit / sms);
        };
        double best = 1e30;
        for (int ns = 1; ns <= most; ++ns) {
            const Tc5Slices sl = slices(ns, wanted / ns);
            const double c = cost(qblocks, sl);
            if (c < 0.98 * best) {
                best = c;
                w.head = w.tail = sl;
                w.split_from = qblocks;
            }
        }
        // Whole waves of row blocks, one block per SM, and slices for the blocks
        // left over, which would hold the chip for a wave that is nearly empty:
        // 512 row blocks on 152 SMs are 3 waves and half a wave of 56 x 2
        // slices (262,144 x 65,536, d=32, TF32, k=1 4.05 -> 3.26 ms with the
        // smaller sample above, of which the split 0.38; 20,000 queries 1.75 ->
        // 1.14).  The certificate takes the lowest threshold of a row's slices,
        // so they want more in all.
        const int whole = qblocks / sms * sms;
        for (int ns = 2; ns <= most && whole > 0 && whole < qblocks; ++ns) {
            const double below = wanted / ns + std::sqrt(2.0 * std::log(double(ns)) * wanted / ns);
            const Tc5Slices one = slices(1, wanted), sl = slices(ns, below);
            const double c = cost(whole, one) + cost(qblocks - whole, sl);
            if (c < 0.98 * best) {
                best = c;
                w.head = one;
                w.tail = sl;
                w.split_from = whole;
                w.wanted = int(std::max(wanted, ns * below));
            }
        }
        w.nsplit = w.head.nsplit;
        const size_t nq_pad = size_t(qblocks) * kT5Rows;
        const size_t n_pad = size_t((n + kT5Cols - 1) / kT5Cols) * kT5Cols;
        w.a_pack = o; o += align256(es * nq_pad * w.KP);
        w.b_pack = o; o += align256(es * n_pad * w.KP);
        w.a_lo = o; o += mode == TK_BRUTE_TF32 ? 0 : align256(es * nq_pad * w.KP);
        w.b_lo = o; o += mode == TK_BRUTE_TF32 ? 0 : align256(es * n_pad * w.KP);
        w.rnorm = o;
        w.qnorm = o; o += align256(4 * size_t(nq));
    } else {
        const int qblocks = int((nq + kRows - 1) / kRows);
        int ns = std::max(1, (2 * sms + qblocks - 1) / std::max(1, qblocks));
        ns = int(std::min<int64_t>(ns, std::max<int64_t>(1, n / (4 * kCols))));
        w.nsplit = ns;
        w.a_pack = o; o += align256(es * size_t(nq) * w.KP);
        w.b_pack = o; o += align256(es * size_t(n) * w.KP);
        w.a_lo = o; o += mode == TK_BRUTE_TF32 ? 0 : align256(es * size_t(nq) * w.KP);
        w.b_lo = o; o += mode == TK_BRUTE_TF32 ? 0 : align256(es * size_t(n) * w.KP);
        w.rnorm = o; o += align256(4 * size_t(n));
        w.qnorm = o; o += align256(4 * size_t(nq));
    }
    if (w.tc5) {
        w.centre = o; o += 256;
        const int64_t rows = (nq + kT5Rows - 1) / kT5Rows * kT5Rows;
        const size_t lists = size_t(first_slice(rows, w.split_from, w.head.nsplit, w.tail.nsplit)) * kT5Parts;
        w.hits = o; o += align256(8 * lists * kT5Cap);
        w.counts = o; o += align256(4 * lists);
        w.thr = o; o += align256(4 * lists);
    } else {
        w.cand_s = o; o += align256(4 * size_t(nq) * w.nsplit * w.C);
        w.cand_i = o; o += align256(4 * size_t(nq) * w.nsplit * w.C);
        w.tau = o; o += align256(4 * size_t(nq) * w.nsplit);
    }
    w.fail_list = o; o += align256(4 * size_t(nq));
    w.brute = o; o += brute_fallback_workspace_bytes(n, nq, d, k);
    w.total = o;
    return w;
}

// Every query on the fallback list: the tensor-core candidate search does
// not fit this shape (see run_brute_tc), the exact kernel answers them all.
__global__ void k_all_queries(int nq, int* list, int* count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nq) list[i] = i;
    if (i == 0) *count = nq;
}

// Poll budget of the candidate kernel's bounded waits (0 = kT5MaxTries); set
// by tk_set_device_wait_limit.
std::atomic<uint32_t> g_wait_polls{0};

int sm_count_now() {
    int dev = 0, v = 1;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v < 1) v = 1;
    return v;
}

}  // namespace

// The workspace starts with two words a pass (see kTcErrTimeout; queries
// recomputed), which tk_nn_distance_report reads; every pass uses the rest.
namespace {

int64_t pass_length(int d, int k, int mode, int64_t pass) {
    return tc5_eligible(d, k, mode) ? pass : int64_t(1) << 31;  // the mma.sync search's lists are short
}
int64_t pass_count(int64_t nq, int64_t len) { return (std::max<int64_t>(nq, 1) + len - 1) / len; }
size_t words_bytes(int64_t passes) { return align256(2 * sizeof(int) * size_t(passes)); }

}  // namespace

// A last, shorter pass may need more than a full one: rows left over after
// whole waves of blocks are searched in slices, each with lists of its own.
size_t brute_tc_workspace_bytes(int64_t n, int64_t nq, int d, int k, int mode, int64_t pass) {
    nq = std::max<int64_t>(nq, 1);
    const int64_t len = pass_length(d, k, mode, pass), rest = nq % len;
    const int sms = sm_count_now();
    size_t most = 0;
    if (nq >= len) most = tc_layout(n, len, d, k, mode, sms).total;
    if (rest > 0) most = std::max(most, tc_layout(n, rest, d, k, mode, sms).total);
    return words_bytes(pass_count(nq, len)) + most;
}

namespace {

int run_pass(const float* ref, int64_t n, const float* q, int64_t nq, int d, int k, int mode, float* dists,
             int32_t* idx, int* words, char* p, cudaStream_t s) {
    const TcWs w = tc_layout(n, nq, d, k, mode, sm_count_now());
    const int n32 = int(n), nq32 = int(nq);
    int* err = words;  // no certificates when set (see kTcNormLimit)
    int* fail_count = words + 1;
    if (!w.tc5) {
        // The mma.sync candidate search keeps 128 rows' lists and a score tile
        // in shared memory; for k > 32 with d > 32 (C = 128, KP = 64) that is
        // more than a block may have.  The answer is exact either way, so the
        // exact kernel answers every query (tk_nn_distance_report: all
        // recomputed) instead of failing the call.
        int dev = 0, optin = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) optin = 0;
        if (select_smem_bytes(mode, w.KP, w.C) > size_t(optin)) {
            int* list = reinterpret_cast<int*>(p + w.fail_list);
            cudaError_t e0 = cudaMemsetAsync(err, 0, sizeof(int), s);
            if (e0 != cudaSuccess) return fail(TK_ECUDA, std::string("memset: ") + cudaGetErrorString(e0));
            k_all_queries<<<(nq32 + 255) / 256, 256, 0, s>>>(nq32, list, fail_count);
            const cudaError_t e1 = cudaGetLastError();
            if (e1 != cudaSuccess) return fail(TK_ECUDA, std::string("fallback list: ") + cudaGetErrorString(e1));
            return brute_fallback(ref, n, q, nq, d, k, dists, idx, list, fail_count, p + w.brute,
                                  brute_fallback_workspace_bytes(n, nq, d, k), s);
        }
    }
    int crc = TK_OK;
    const float* centre = reinterpret_cast<const float*>(p + w.centre);
    float* qnorm = reinterpret_cast<float*>(p + w.qnorm);
    const double u = 1.0 / 16777216.0;
    const float eps_dot = float(mode == TK_BRUTE_TF32 ? (1.0 / 1024.0 + 1.0 / 4194304.0 + (d + 2) * 2.0 * u)
                                                      : (3.1 / 65536.0 + 3.0 * (d + 2) * 2.0 * u));
    if (w.tc5) {
        k_tc5_centre<<<1, 1024, 0, s>>>(ref, n32, d, reinterpret_cast<float*>(p + w.centre), err, fail_count);
    } else {
        const cudaError_t e0 = cudaMemsetAsync(words, 0, 2 * sizeof(int), s);
        if (e0 != cudaSuccess) return fail(TK_ECUDA, std::string("memset: ") + cudaGetErrorString(e0));
    }
    if (w.tc5) {
        // 1-2. pack into the core-matrix layout and run the tcgen05 candidate kernel
        const int qblocks = (nq32 + kT5Rows - 1) / kT5Rows, tiles = int((n + kT5Cols - 1) / kT5Cols);
        unsigned char* ahi = reinterpret_cast<unsigned char*>(p + w.a_pack);
        unsigned char* alo = reinterpret_cast<unsigned char*>(p + w.a_lo);
        unsigned char* bhi = reinterpret_cast<unsigned char*>(p + w.b_pack);
        unsigned char* blo = reinterpret_cast<unsigned char*>(p + w.b_lo);
        const int chunks = w.KP * (mode == TK_BRUTE_TF32 ? 4 : 2) / 16;  // 16-byte pieces of a packed row
        auto grid = [&](int64_t rows) { return unsigned((rows * chunks + 255) / 256); };
        const unsigned ga = grid(int64_t(qblocks) * kT5Rows), gb = grid(int64_t(tiles) * kT5Cols);
        const Tc5Pack pq{q, nq32, qblocks, ahi, alo}, pr{ref, n32, tiles, bhi, blo};
        // set up while the kernel before it runs
        const cudaError_t e0 =
            mode == TK_BRUTE_TF32
                ? launch(true, k_tc5_pack<TK_BRUTE_TF32>, dim3(ga + gb), 256, 0, s, pq, pr, int(ga), d, w.KP, centre, qnorm, err)
                : launch(true, k_tc5_pack<TK_BRUTE_BF16_SPLIT>, dim3(ga + gb), 256, 0, s, pq, pr, int(ga), d, w.KP, centre, qnorm, err);
        if (e0 != cudaSuccess) return fail(TK_ECUDA, std::string("packing: ") + cudaGetErrorString(e0));
        Tc5Args t5{};
        t5.a_hi = ahi;
        t5.a_lo = alo;
        t5.b_hi = bhi;
        t5.b_lo = blo;
        t5.nq = nq32;
        t5.tiles = tiles;
        t5.split_from = w.split_from;
        t5.head = w.head;
        t5.tail = w.tail;
        t5.hits = reinterpret_cast<uint2*>(p + w.hits);
        t5.counts = reinterpret_cast<int*>(p + w.counts);
        t5.thr = reinterpret_cast<float*>(p + w.thr);
        t5.qnorm = qnorm;
        t5.eps_dot = eps_dot;
        t5.d = d;
        t5.err = err;
        const uint32_t polls = g_wait_polls.load();
        t5.max_tries = polls ? polls : kT5MaxTries;
        crc = mode == TK_BRUTE_TF32 ? tc5_dispatch_tf32(t5, w.KP, qblocks, s)
                                    : tc5_dispatch_bf16(t5, w.KP, qblocks, s);
        if (crc != TK_OK) return crc;
    } else if (mode == TK_BRUTE_TF32) {
        k_tc_pack<TK_BRUTE_TF32><<<(nq32 + 255) / 256, 256, 0, s>>>(q, nq32, d, w.KP, reinterpret_cast<uint32_t*>(p + w.a_pack),
                                                                  nullptr, nullptr, qnorm,
                                                                  nullptr);
        k_tc_pack<TK_BRUTE_TF32><<<(n32 + 255) / 256, 256, 0, s>>>(ref, n32, d, w.KP, reinterpret_cast<uint32_t*>(p + w.b_pack),
                                                                 nullptr, nullptr, reinterpret_cast<float*>(p + w.rnorm),
                                                                 err);
    } else {
        k_tc_pack<TK_BRUTE_BF16_SPLIT><<<(nq32 + 255) / 256, 256, 0, s>>>(
            q, nq32, d, w.KP, nullptr, reinterpret_cast<__nv_bfloat16*>(p + w.a_pack),
            reinterpret_cast<__nv_bfloat16*>(p + w.a_lo), qnorm, nullptr);
        k_tc_pack<TK_BRUTE_BF16_SPLIT><<<(n32 + 255) / 256, 256, 0, s>>>(
            ref, n32, d, w.KP, nullptr, reinterpret_cast<__nv_bfloat16*>(p + w.b_pack),
            reinterpret_cast<__nv_bfloat16*>(p + w.b_lo), reinterpret_cast<float*>(p + w.rnorm), err);
    }
    // 2. candidates
    TcArgs a{};
    a.a_tf = reinterpret_cast<const uint32_t*>(p + w.a_pack);
    a.b_tf = reinterpret_cast<const uint32_t*>(p + w.b_pack);
    a.a_hi = reinterpret_cast<const __nv_bfloat16*>(p + w.a_pack);
    a.b_hi = reinterpret_cast<const __nv_bfloat16*>(p + w.b_pack);
    a.a_lo = reinterpret_cast<const __nv_bfloat16*>(p + w.a_lo);
    a.b_lo = reinterpret_cast<const __nv_bfloat16*>(p + w.b_lo);
    a.rnorm = reinterpret_cast<const float*>(p + w.rnorm);
    a.n = n32;
    a.nq = nq32;
    a.KP = w.KP;
    a.C = w.C;
    a.nsplit = w.nsplit;
    a.cand_s = reinterpret_cast<float*>(p + w.cand_s);
    a.cand_i = reinterpret_cast<int32_t*>(p + w.cand_i);
    a.tau = reinterpret_cast<float*>(p + w.tau);
    const int qblocks = (nq32 + kRows - 1) / kRows;
    if (!w.tc5) {
        crc = tc_select_dispatch(a, mode, qblocks, s);
        if (crc != TK_OK) return crc;
    }
    // 3. exact re-rank + certificate
    RerankArgs ra{};
    ra.ref = ref;
    ra.q = q;
    ra.n = n32;
    ra.nq = nq32;
    ra.d = d;
    ra.k = k;
    ra.C = w.C;
    ra.nsplit = w.nsplit;
    ra.split_from = w.split_from;
    ra.tail_nsplit = w.tail.nsplit;
    ra.cand_s = a.cand_s;
    ra.cand_i = a.cand_i;
    ra.tau = a.tau;
    ra.keep = w.wanted;
    ra.hits = reinterpret_cast<const uint2*>(p + w.hits);
    ra.counts = reinterpret_cast<const int*>(p + w.counts);
    ra.thr = reinterpret_cast<const float*>(p + w.thr);
    ra.eps_dot = eps_dot;
    ra.out_d = dists;
    ra.out_i = idx;
    ra.qnorm = qnorm;
    ra.fail_count = fail_count;
    ra.fail_list = reinterpret_cast<int*>(p + w.fail_list);
    ra.err = err;
    const int rb = (nq32 + 7) / 8;
    if (w.tc5) {
        k_tc5_rerank<<<rb, 256, 0, s>>>(ra);
    } else if (k <= 32) k_tc_rerank<1><<<rb, 256, 0, s>>>(ra);
    else k_tc_rerank<2><<<rb, 256, 0, s>>>(ra);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(TK_ECUDA, std::string("tc launch: ") + cudaGetErrorString(e));
    // 4. exact recomputation of the uncertified queries
    return brute_fallback(ref, n, q, nq, d, k, dists, idx, ra.fail_list, ra.fail_count, p + w.brute,
                          brute_fallback_workspace_bytes(n, nq, d, k), s);
}

}  // namespace

int run_brute_tc(const float* ref, int64_t n, const float* q, int64_t nq, int d, int k, int mode, float* dists,
                 int32_t* idx, void* ws, size_t ws_bytes, int64_t pass, cudaStream_t s) {
    if (k > 64) return fail(TK_EUNSUPPORTED, "tensor-core modes support k <= 64 (use TK_BRUTE_EXACT)");
    if (d > 64) return fail(TK_EUNSUPPORTED, "tensor-core modes support d <= 64 (use TK_BRUTE_EXACT)");
    if (!ws || ws_bytes < brute_tc_workspace_bytes(n, nq, d, k, mode, pass))
        return fail(TK_EWORKSPACE, "workspace too small");
    const int64_t len = pass_length(d, k, mode, pass), passes = pass_count(nq, len);
    char* rest = static_cast<char*>(ws) + words_bytes(passes);
    int rc = TK_OK;
    for (int64_t i = 0; i < passes && rc == TK_OK; ++i)
        rc = run_pass(ref, n, q + i * len * d, std::min(len, nq - i * len), d, k, mode, dists + i * len * k,
                      idx + i * len * k, static_cast<int*>(ws) + 2 * i, rest, s);
    return rc;
}

}  // namespace tk

extern "C" uint32_t tk_set_device_wait_limit(uint32_t polls) { return tk::g_wait_polls.exchange(polls); }

extern "C" int tk_nn_distance_report(const void* workspace, int64_t n, int64_t nq, int dims, int k, int dtype,
                                     int mode, int* flags, int* recomputed) {
    using namespace tk;
    using namespace tk::tcx;
    clear_error();
    if (!flags || !recomputed) return fail(TK_EINVAL, "null output pointer");
    *flags = 0;
    *recomputed = 0;
    if (mode != TK_BRUTE_TF32 && mode != TK_BRUTE_BF16_SPLIT) return TK_OK;  // the exact kernel has no certificate
    if (dtype != TK_F32) return fail(TK_EINVAL, "tensor-core modes take float32 inputs");
    if (!workspace || n < 1 || nq < 1 || k < 1 || dims < 1) return fail(TK_EINVAL, "bad shape or null workspace");
    std::vector<int> words(2 * size_t(pass_count(nq, pass_length(dims, k, mode, kTcPass))));
    const cudaError_t e = cudaMemcpy(words.data(), workspace, sizeof(int) * words.size(), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return fail(TK_ECUDA, std::string("report: ") + cudaGetErrorString(e));
    for (size_t i = 0; i < words.size(); i += 2) {
        *flags |= words[i];
        *recomputed += words[i + 1];
    }
    if (*flags & kTcErrTimeout)
        return fail(TK_ETIMEOUT, "a bounded device wait ran out; the exact kernel recomputed every query");
    return TK_OK;
}
