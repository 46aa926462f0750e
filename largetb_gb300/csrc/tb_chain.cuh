// tb_chain.cuh -- steps that follow each other in a stream, each launched while
// the one before still runs (programmatic dependent launch): its CTAs take the
// places that the earlier step's CTAs leave, set themselves up and read what no
// step writes, and wait in chain_wait() until the earlier step is complete and
// its results visible.  A launch's latency and a CTA's start, some 4 us of a
// step, then overlap the step before.
#pragma once

#include <cuda_runtime.h>

namespace tb {

// Once a CTA, early: the next step may be launched when every CTA is running.
__device__ __forceinline__ void chain_release() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// Every thread, before it reads a step's results or writes over its inputs.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_chained(void (*fn)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, fn, static_cast<P>(args)...);
}

}  // namespace tb
