// Tensor-core brute force (declarations; see brute_tc.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace tk {

// Queries per pass of the modes that name the tensor cores: a query's hit lists
// take 4.6 KB a slice, 4.9 GB a pass.
constexpr int64_t kTcPass = int64_t(1) << 20;

size_t brute_tc_workspace_bytes(int64_t n, int64_t nq, int d, int k, int mode, int64_t pass);
int run_brute_tc(const float* ref, int64_t n, const float* q, int64_t nq, int d, int k, int mode, float* dists,
                 int32_t* idx, void* ws, size_t ws_bytes, int64_t pass, cudaStream_t s);

}  // namespace tk
