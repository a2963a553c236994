// Device-wide primitives written for this engine: an exclusive prefix sum and
// a stable radix pass over (8-bit key, uint32 value) pairs, which orders the
// queries of a launch by cost class.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace tk {

// Scratch bytes for exclusive_scan over n ints.
size_t scan_workspace_bytes(int64_t n);
// In-place exclusive prefix sum of data[0..n).  Returns a cudaError_t.
cudaError_t exclusive_scan(int* data, int64_t n, void* ws, cudaStream_t s);

// One stable pass over 8-bit keys (key < 256).  Scratch bytes:
size_t sort_pass8_workspace_bytes(int64_t n);
cudaError_t sort_pass8(const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out, uint32_t* vals_out,
                       int64_t n, void* ws, size_t ws_bytes, cudaStream_t s);

}  // namespace tk
