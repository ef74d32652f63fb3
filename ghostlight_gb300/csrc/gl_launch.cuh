// gl_launch.cuh — launches that are set up while the stream's last kernel drains.
//
// A kernel launched by launch_after may be resident before the kernel before it
// in the stream is done; its first instruction is after_previous(), which waits
// for that kernel to be complete and its writes visible.  Every kernel of a chain
// waits so, hence also for the ones before.  The setting up of a short kernel's
// launch (about 2 us) then overlaps the kernel before it.
#pragma once

#include <cuda_runtime.h>

namespace gl {

__device__ __forceinline__ void after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... V>
cudaError_t launch_after(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, const V&... v)
{
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &early;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(v)...);
}

}  // namespace gl
