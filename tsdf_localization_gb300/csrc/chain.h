// Programmatic dependent launch for the kernels that follow one another in a
// stream (the update and resampling chains, the scan reduction).
#pragma once

#include <cuda_runtime.h>

namespace tsdfl {

// Lets launches of `kernel` ask for up to `most` bytes of dynamic shared memory: the
// largest size any call needs, not this call's own.  The limit belongs to the function
// in the process, whatever the context, stream or thread, so a size that follows the
// call would let one thread's small call lower it under another's larger one.
template <typename... Params>
inline cudaError_t allow_smem(void (*kernel)(Params...), size_t most)
{
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e != cudaSuccess) cudaGetLastError();   // the caller reports it
    return e;
}

// First statement of every kernel that launch_chained starts with programmatic
// dependent launch: the grid may be scheduled before the previous kernel in the
// stream has completed, so it waits here until that kernel's writes are visible.
// No kernel lets its successor be scheduled early (griddepcontrol.launch_dependents):
// the successor's waiting blocks then sit beside the running kernel's, and the small
// kernels behind a scoring launch cost it 12 us (a step of 1,000 particles x 2,048
// points 73 us with it, 61 without); the launches overlap all the same.
static __device__ __forceinline__ void chain_enter()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launches a kernel that opens with chain_enter(), so that its launch overlaps
// the end of the previous kernel instead of following it.
template <typename... Params, typename... Args>
inline cudaError_t launch_chained_2d(void (*kernel)(Params...), dim3 grid, unsigned block, size_t smem,
                                     cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// The same with the grid in clusters of `cluster` blocks (of which grid is a multiple).
template <typename... Params, typename... Args>
inline cudaError_t launch_chained_clusters(void (*kernel)(Params...), unsigned grid, unsigned cluster,
                                           unsigned block, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <typename... Params, typename... Args>
inline cudaError_t launch_chained(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem,
                                  cudaStream_t s, Args... args)
{
    return launch_chained_2d(kernel, dim3(grid), block, smem, s, args...);
}

}  // namespace tsdfl
