// pdl.cuh - programmatic dependent launch for the kernels of a step.
//
// A step is a chain of short kernels.  Launched with launch_after(), a kernel's
// blocks are set up while the kernel before it on the stream still runs
// (once all of that one's blocks have called let_next_start()), and wait in
// wait_for_previous() until it has finished and its writes are visible.  Every
// kernel launched this way calls wait_for_previous() before it touches global
// memory, so the chain is as ordered as with plain launches; what goes on
// before that call (shared memory cleared, indices) costs no time.
#pragma once
#include <utility>
#include <cuda_runtime.h>

namespace gcs {

__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}

}  // namespace gcs
