// launch.cuh — kernel launches that overlap the previous kernel's end
// (programmatic stream serialisation).  A kernel launched with launch_pdl may
// have its CTAs placed on the SMs before the kernel ahead of it in the stream
// has finished; every thread of it calls pdl_enter() before it touches memory,
// which waits until that kernel is complete and its writes are visible.  What
// that kernel may have written is read with plain loads, not through __ldg or a
// const __restrict__ parameter: such loads assume that nothing writes the data
// from the launch on.
// Without it each of a program's short calls pays its launch, about 2 us, after
// the call before has drained.
#pragma once

#include <cuda_runtime.h>
#include <utility>

namespace gbx_launch {

// First statement of a kernel launched with launch_pdl: its work starts when the
// previous kernel is complete, and only then may the next one be placed.  So at
// most one kernel waits on the SMs.  (If a waiting kernel lets in its successor,
// that one the next, and so on, then the SMs fill with CTAs of calls far ahead,
// and several CTAs of one call end up on one SM, whose FP64 pipe they share:
// streams of DGEMM 96 x 128 x 512 took 82 us a call that way, 30 now, 31 without
// overlap.)
__device__ __forceinline__ void pdl_enter()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Hand-over between the warps of a CTA on named barrier id (1-15) of `threads`
// threads: the producing warp arrives without waiting, the others wait and then
// see what it stored.
__device__ __forceinline__ void bar_arrive(int id, int threads)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_wait(int id, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// overlap = false: an ordinary launch (pdl_enter() does nothing then).
template <typename... P, typename... A>
cudaError_t launch_pdl_if(bool overlap, void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t s,
                          A &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(std::forward<A>(args))...);
}
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A &&...args)
{
    return launch_pdl_if(true, kernel, dim3(grid), block, smem, s, std::forward<A>(args)...);
}

// A kernel bound by a pipe or by memory: its CTAs are placed early only if
// there is at most one per SM.  More of them, placed as the previous kernel's
// CTAs leave, end up unevenly on the SMs (a GEMM 756 x 330 x 1710 took 14 %
// longer).
template <typename... P, typename... A>
cudaError_t launch_pdl_short(int sms, void (*kernel)(P...), dim3 grid, unsigned block, cudaStream_t s, A &&...args)
{
    return launch_pdl_if((unsigned long long)grid.x * grid.y <= (unsigned long long)sms, kernel, grid, block, 0, s,
                         std::forward<A>(args)...);
}

}  // namespace gbx_launch
