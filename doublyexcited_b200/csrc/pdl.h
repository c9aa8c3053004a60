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

// Loads of what an earlier kernel wrote.  A kernel that waits inside is resident
// while its predecessor still writes, so the non-coherent path (__ldg, and the
// loads that const __restrict__ parameters allow the compiler), which takes the
// data as constant from the kernel's first instruction to its last, is not for
// them; tables that the handle's creation finished are read with __ldg.
// volatile keeps them behind the wait; no memory clobber, so loads and stores of
// other data may pass.
__device__ __forceinline__ double2 ld_prev(const double2 *p)
{
    double2 v;
    asm volatile("ld.global.v2.f64 {%0,%1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 ld_prev(const float2 *p)
{
    float2 v;
    asm volatile("ld.global.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned long long ld_prev(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.global.b64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
// the same from L2: partial sums that other blocks wrote
__device__ __forceinline__ double2 ld_l2(const double2 *p)
{
    double2 v;
    asm volatile("ld.global.cg.v2.f64 {%0,%1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
    return v;
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
