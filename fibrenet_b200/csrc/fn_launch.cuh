/*
 * fn_launch.cuh -- programmatic dependent launch of the step sequence's and
 * the adjoint sweep's kernels.
 */
#pragma once
#include <cuda_runtime.h>

namespace fn {

/* Programmatic dependent launch (launch_next): a kernel of the step sequence
   or of the adjoint sweep waits on the device for the kernel before it, all of
   its blocks and writes, before it touches anything that the kernels of its
   chain write, and says when the next one's blocks may be placed.  The launch
   itself, 1.5 us and more between dependent kernels of a stream, then runs
   beside the kernel before it.  Every thread of every kernel that launch_next
   starts must wait, whatever it does next: one that ended without waiting
   would let its successor run beside its predecessor. */
__device__ __forceinline__ void await_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

/* Launches a kernel that waits (await_previous) so that its blocks
   may be placed while the kernel before it drains. */
template <class... P, class... X>
static void launch_next(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, X... x) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, P(x)...); /* errors are read by the callers' cudaGetLastError */
}

}  // namespace fn
