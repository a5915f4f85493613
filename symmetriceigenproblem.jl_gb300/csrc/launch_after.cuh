// launch_after.cuh -- programmatic dependent launch: chains of short kernels on one stream.
//
// A kernel launched with launch_after may start before the memory of the launch ahead has settled;
// wait_previous_launch holds it until that launch has completed and its writes are visible.  Every kernel of a
// chain calls it first, on every path and also where it needs nothing from the launch ahead, so that what
// a kernel reads or overwrites may come from any launch before it.  None lets the next in early
// (griddepcontrol.launch_dependents): blocks that sit and wait cost more than they save (n = 1300 reduction
// 29.6 ms with it ahead of the wait, 28.0 behind it, 27.0 without, 35.3 by ordinary launches).  What the chain
// writes is read through plain pointers: behind a const __restrict__ one the compiler may take the read-only
// loads, which need memory that nothing writes from the kernel's start on.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace symeig {

__device__ __forceinline__ void wait_previous_launch()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... Params, typename... Args>
void launch_after(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t s, Args... args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace symeig
