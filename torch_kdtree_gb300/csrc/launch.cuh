// Launches of a chain of short kernels.
//
// A kernel launched with `after` is set up while the one before it on the
// stream still runs, and its blocks start when that one's last blocks end
// (programmatic dependent launch): some 1.3 us less per link of the chain.
// Such a kernel waits for the one before to have ended and its writes to be
// visible (begin) before it touches memory, so whatever it follows, the order
// is the stream's.  Buffers that the chain writes are not __restrict__ there: a
// load of constant data may be moved above the wait.  Letting the next launch's
// blocks in earlier still was no faster, and slower for small clouds.
#pragma once

#include <cuda_runtime.h>

namespace tk {

__device__ __forceinline__ void begin() { cudaGridDependencySynchronize(); }

template <typename... P, typename... A>
cudaError_t launch(bool after, void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = after ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace tk
