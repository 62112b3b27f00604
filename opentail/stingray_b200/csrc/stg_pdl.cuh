// Kernels launched behind one another before the one ahead has ended (programmatic dependent launch): the one ahead
// lets its successor start (pdl_release, effective once all of its CTAs have called it or ended) and the successor
// waits for it (pdl_wait: all of the kernel ahead has ended and its writes are seen; returns at once where
// nothing is ahead).  Every CTA of a successor waits, also one without work, so that a kernel's end implies that
// of all before it.
#pragma once
#include <cuda_runtime.h>

namespace stg {

__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... Params, class... Args>
inline cudaError_t launch_behind(void (*fn)(Params...), dim3 grid, int block, size_t smem, cudaStream_t stream, const Args &...args)
{
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, args...);
}

}  // namespace stg
