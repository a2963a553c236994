// tcgen05 candidate search, TF32 operands, rows of up to 24 (see brute_tc_kernels.cuh).
#include "brute_tc_kernels.cuh"

namespace tk {
namespace tcx {

int tc5_dispatch_tf32(const Tc5Args& a, int KP, int qblocks, cudaStream_t s) {
    switch (KP) {
        case 8: return launch_tc5<TK_BRUTE_TF32, 8>(a, qblocks, s);
        case 16: return launch_tc5<TK_BRUTE_TF32, 16>(a, qblocks, s);
        case 24: return launch_tc5<TK_BRUTE_TF32, 24>(a, qblocks, s);
        default: return tc5_dispatch_tf32_deep(a, KP, qblocks, s);  // 32, 40
    }
}

}  // namespace tcx
}  // namespace tk
