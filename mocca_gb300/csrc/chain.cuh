// chain.cuh -- chains of short kernels.
//
// A kernel of a few microseconds costs about as much again to start.  A kernel
// that begins with chain_wait() can be launched while the kernel before it runs
// (launch_early, programmatic dependent launch): its blocks wait there until that
// one has ended and its writes are visible, and let the next one start.  Launched
// in the ordinary way, or behind a kernel without chain_wait(), it runs as any
// other kernel.
#pragma once

#include "mg_internal.cuh"

namespace mg {

__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... V>
int launch_early(mg_ctx* c, void (*kernel)(P...), dim3 grid, int threads, size_t smem, V... args) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = c->stream;
    cfg.attrs = &early;
    cfg.numAttrs = 1;
    MG_CUDA(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
    MG_LAUNCHED(c);
    return MG_OK;
}

}  // namespace mg
