// KD query kernels of float64 trees with a float filter (see kd_filter.cuh).
#include <string>

#include "kd_filter.cuh"

namespace tk {

#define TK_FILTER_LIST(X) \
    X(1, 0) X(1, 1) X(1, 2) X(1, 4) X(2, 0) X(2, 1) X(2, 2) X(2, 4) X(3, 0) X(3, 1) X(3, 2) X(3, 4)

const void* kd_filtered_kernel(int D, int R) {
#define TK_FPTR(d, r) \
    if (D == d && R == r) return reinterpret_cast<const void*>(&k_kd_query_filtered<d, r>);
    TK_FILTER_LIST(TK_FPTR)
#undef TK_FPTR
    return nullptr;
}

int kd_filtered_launch(const FilterArgs& a, int D, int R, int grid, cudaStream_t s) {
#define TK_FLAUNCH(d, r) \
    if (D == d && R == r) k_kd_query_filtered<d, r><<<grid, 256, 0, s>>>(a);
    TK_FILTER_LIST(TK_FLAUNCH)
#undef TK_FLAUNCH
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return fail(TK_ECUDA, std::string("filtered KD query launch: ") + cudaGetErrorString(err));
    return TK_OK;
}

}  // namespace tk
