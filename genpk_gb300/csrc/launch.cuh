// launch.cuh -- kernel launches that overlap the previous kernel's end.
//
// A pass of a small box is a dozen kernels of 5-15 us, and between two plain
// launches of one stream the GPU stands idle for 2-3 us (the first one's last
// block, its memory flush, the second one's launch).  launch_after() lets the
// second kernel's blocks start when the first one's have ended: they set up
// what does not depend on earlier kernels (shared tables, index arithmetic)
// and then wait in wait_previous(), after which everything that earlier kernels
// of the stream wrote is visible.  40 k particles on 64^3: 66 -> 59 us, 2.1 M on
// 128^3: 121 -> 111 us.  (Starting the second kernel's blocks earlier, as soon
// as every block of the first runs, brought small boxes nothing more and cost
// large ones 3-5 %: the waiting blocks hold registers and shared memory.)
//
// Every kernel launched this way calls wait_previous() in every thread before
// it touches global memory that another kernel writes or reads, so that kernels
// complete in stream order, whatever the number of kernels in flight.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace genpk {

__device__ __forceinline__ void wait_previous()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A pointer to what earlier kernels wrote, taken after wait_previous(): loads
// through it cannot be moved before the wait, not even those that go through
// the read-only path (const __restrict__ parameters, __ldg), which the compiler
// may otherwise reorder freely.
template <typename T>
__device__ __forceinline__ T *fresh(T *p)
{
    asm volatile("" : "+l"(p) : : "memory");
    return p;
}

template <typename... Params, typename... Args>
cudaError_t launch_after(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem,
                         cudaStream_t stream, Args &&...args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

}  // namespace genpk
