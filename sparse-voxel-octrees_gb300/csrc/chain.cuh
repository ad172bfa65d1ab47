// chain.cuh — launches that overlap the end of the kernel before them.
//
// A chain of short kernels on one stream spends much of its time between
// them.  A kernel that starts with chain_begin() may be launched by
// launch_chained: its CTAs then come up while the kernel before it on the
// stream runs out, and wait in chain_begin() until that kernel has finished
// and its writes are visible.  chain_begin() also lets the next kernel of the
// chain come up, once every CTA of this one is there; the order of the work
// stays that of the stream.  Every thread calls it before any access to
// memory and before any return, so a finished kernel means that those before
// it have finished too.  Launched in the plain way such a kernel runs as any
// other.
//
// Measured on what a caller waits for: an edit of a 200x131x177 volume, its
// octree, table and first view (20 launches) 252 -> 225 us; the octree of a
// 512^3 grid (6) 243 -> 231; a mesh of 327,680 triangles at 1024^3 (17) 867 ->
// 856; a 320x180 frame of a 1024^3 octree (2) 63 -> 58, 1280x720 144.5 -> 143.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace svo {

__device__ __forceinline__ void chain_begin() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}

template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kernel)(Params...), unsigned grid, unsigned block, cudaStream_t st, Args &&...args) {
    cudaLaunchAttribute order{};
    order.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    order.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(block);
    config.stream = st;
    config.attrs = &order;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, kernel, std::forward<Args>(args)...);
}

}  // namespace svo
