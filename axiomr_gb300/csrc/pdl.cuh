// Programmatic dependent launch (PTX griddepcontrol): a kernel launched with launch_dependent may
// be set up, and its CTAs started, while the kernel before it on the stream still drains; it
// waits at pdl_wait for that kernel's completion (and its writes) before it reads any of them.
// What it reads from kernels of the same chain it loads with plain loads after pdl_wait: a
// read-only (ld.global.nc) load could be moved above the wait. The first kernel of a chain is
// launched in full stream order, so whatever was there before the chain is complete.
#pragma once
#include <cuda_runtime.h>

namespace axr {
namespace {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Lets the next kernel of the chain start once every CTA of this one has called it (or ended).
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_dependent(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t stream, const A&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace
}  // namespace axr
