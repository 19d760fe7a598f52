// pdl.cuh -- launches that overlap their start with the end of the kernel
// before them on the stream (programmatic dependent launch).
//
// A chain of kernels of a few microseconds loses 2.3 us per kernel between the
// last block of one and the first instruction of the next, also inside a CUDA
// graph.  A kernel launched here is set up while the one before it drains, and
// starts with dependency_wait(), which returns when every kernel before it has
// completed and its writes are visible.  Every kernel launched this way waits
// before anything else that reads or writes memory, also on paths that return
// at once, so the order of a chain is that of the stream.  The kernels give no
// early trigger: blocks that come in early and wait hold warps and shared
// memory of the running kernel's last wave (PCG iterations with the coarse
// space, 12 kernels: K = 32768, N = 2, FP64 47.5 ms without these launches,
// 45.2 with, 50.1 with a trigger after the wait; K = 101,246, N = 4, mixed 29.3,
// 28.5 and 29.0).
#pragma once

#include <utility>

#include <cuda_runtime.h>

namespace dgk {

__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t s, A&&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace dgk
