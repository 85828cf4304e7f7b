// Launch with programmatic stream serialisation, and the wait that goes with
// it: a kernel launched with launch_dep has its CTAs scheduled while its
// predecessor on the stream drains, and waits in pdl_wait, before touching
// memory, until the predecessor has completed and its writes are visible
// (griddepcontrol.wait; a no-op for an ordinary launch).
#pragma once

#include <cuda_runtime.h>

namespace mpm {

#if defined(__CUDACC__)
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

template <typename... P, typename... A>
void launch_dep(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace mpm
