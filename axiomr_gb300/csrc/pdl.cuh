// Programmatic dependent launch (PTX griddepcontrol): a kernel launched with launch_dependent may
// be set up, and its CTAs started, while the kernel before it on the stream still drains; it
// waits at pdl_wait for that kernel's completion (and its writes) before it touches any of them, and
// only then lets the next one start (pdl_release). So when a kernel starts, all but the kernel
// directly before it are complete: data of those may be read at any point, also by read-only loads
// (ld.global.nc), which could be moved above the wait; data of the kernel directly before it only
// by plain loads after the wait. Behind anything else than such a kernel (a copy, a kernel that never
// releases) the launch is an ordinary one, under capture too.
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
