// chain.cuh -- launches of one pass after another without the gap between them (sm_100a
// programmatic dependent launch).
//
// A kernel that starts with chain_trigger() lets the next kernel of its stream start once
// all of its CTAs are resident; a kernel launched by launch_chained(true, ...) may
// therefore run before its predecessor has ended, and touches nothing that earlier work
// writes until chain_wait() returns: that waits for the predecessor's end, and its writes
// are visible then. What a kernel reads before it (its tables in the program blob, kernel
// parameters) was uploaded before the first kernel of the run. What the predecessor wrote is
// read through pointers that are not __restrict__: of those the compiler may take it that
// nothing else writes there, the wait's memory clobber included, and move their loads above it.
// On states whose passes last as long as their setup (10 to 16 us a pass up to 20 qubits) the
// setup and the launch latency of a pass then overlap the pass before it.
#pragma once

#include <cuda_runtime.h>

namespace zxh {

__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// chained: the launch directly follows a kernel of the same run on the stream (no copy or
// memset between), and kern calls chain_wait().
template <typename... P, typename... A>
cudaError_t launch_chained(bool chained, void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                           A... args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

}  // namespace zxh
