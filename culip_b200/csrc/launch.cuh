// Launches that overlap their predecessor's end (programmatic dependent
// launch): the kernel's blocks are placed while the kernel before it in the
// stream drains, which hides about 1.5 us of every dependent launch.
//
// Such a kernel waits (wait_previous) before it touches anything that an
// earlier kernel of the stream may have written or still reads, and only then
// lets its own successor start: at once (after_previous does both), for
// successors that load the factor's data meanwhile, or by ending.  A kernel's
// early part may read what was complete before its predecessor began: the
// successor of a kernel that waits starts after everything before that kernel
// is complete and visible.
//
// Such a kernel's life begins before its predecessor has finished writing, so
// what the predecessor may write is read with plain loads through pointers
// without __restrict__: __ldg and const __restrict__ promise that nothing
// writes the memory during the kernel's life, and leave the compiler free to
// move the load above after_previous().
#pragma once

#include "device.h"

namespace culipx {

__device__ __forceinline__ void wait_previous() { cudaGridDependencySynchronize(); }

__device__ __forceinline__ void after_previous()
{
    wait_previous();
    cudaTriggerProgrammaticLaunchCompletion();
}

// overlap = false: an ordinary launch, for the factorization inside the graph
// that the library captures, where the dependent edges cost more than they hide
// (108 against 104 us for the ragged FP32 factor).  In a caller's own capture
// the others keep them: ten products of N = 3000 31 us a replay against 35,
// three stages 10.4 against 14.5.
template <class... P, class... A>
int launch_overlapped(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, bool overlap, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = overlap ? 1 : 0;
    CULIPX_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
    return CULIPX_OK;
}

}  // namespace culipx
