// chain.cuh — launches that overlap the end of the kernel before them.
//
// A chain of short kernels on one stream spends much of its time between
// them.  A kernel that starts with chain_begin() may be launched by
// launch_chained: it is then set up while the kernel before it on the stream
// runs, its CTAs come up as soon as the last of that kernel's have left, and
// wait in chain_begin() until its writes are visible.  The order of the work
// stays that of the stream.  Every thread calls it before any access to memory
// and before any return, so a finished kernel means that those before it have
// finished too.  Launched in the plain way such a kernel runs as any other.
//
// What the kernel before may write is not taken as const __restrict__ and not
// read by __ldg: both let the compiler move the read over chain_begin() and
// serve it from the non-coherent cache.  __ldg is for what was complete before
// the chain began (a wait of the host or a plain launch lies between).
//
// chain_next() lets the next kernel's CTAs up earlier, beside this one's last.
// It pays in a kernel of one wave that ends in a few long warps (a frame's
// corners: 320x180 of a 1024^3 octree 59.8 -> 57.8 us).  In a build it costs.
//
// Measured on what a caller waits for, chain_next() in every kernel: an edit of
// a 200x131x177 volume, its octree, table and first view (20 launches) 252 ->
// 225 us; the octree of a 512^3 grid (6) 243 -> 231; a mesh of 327,680
// triangles at 1024^3 (17) 867 -> 856; a 320x180 frame of a 1024^3 octree (2)
// 63 -> 58, 1280x720 144.5 -> 143.  chain_begin() alone against both: the mesh
// 767 against 783 (its kernel of 21,297 short CTAs 16 against 24), the 512^3
// grid 206 against 210, that octree's table 144 against 150.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace svo {

__device__ __forceinline__ void chain_begin() { cudaGridDependencySynchronize(); }

__device__ __forceinline__ void chain_next() { cudaTriggerProgrammaticLaunchCompletion(); }

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
