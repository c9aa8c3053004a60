// pdl.h -- programmatic dependent launches.  A kernel launched by pdl_launch
// may be scheduled while its predecessor's last blocks run; it calls pdl_enter
// before it touches global memory, which waits until the predecessor has
// completed and its writes are visible (no-op in an ordinary launch), and lets
// its own successor be scheduled.  Every block calls it, so a kernel never
// completes before its predecessor, and what follows in the stream by an
// ordinary launch keeps full order.  What it saves is the launch gap, about
// 1 us of the ~60 block-operation launches an iteration has: an FP64 block
// solve of N = 5 48.7 -> 47.8 ms, a mixed N = 6 iteration 3.51 -> 3.48 ms.
#pragma once
#include <cuda_runtime.h>

#include "de_kernels.h"

namespace de {

__device__ __forceinline__ void pdl_enter()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

template <class... P, class... A>
cudaError_t pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = programmatic_launch() ? 1 : 0;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
    count_launch();
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace de
