// Programmatic dependent launches.
#pragma once

#include <cuda_runtime.h>

namespace pdgpu {
namespace {

// Programmatic dependent launch: a kernel launched with launch_dependent
// starts while the one ahead of it in the stream still runs; its CTAs do
// nothing but read constants until pdl_wait, which returns when that kernel has
// finished and its writes are visible.  pdl_start lets the next kernel's CTAs
// come; both are no-ops in a launch without the attribute.  Every CTA of a
// kernel launched this way waits, so that a kernel's end implies the end of all
// those before it.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// launch as a programmatic dependent of the kernel ahead in the stream (see
// pdl_wait); graph captures keep the attribute as a programmatic edge
template <class... P, class... A>
void launch_dependent(void (*k)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                      A... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(grid);
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, k, args...);
}

}  // namespace
}  // namespace pdgpu
