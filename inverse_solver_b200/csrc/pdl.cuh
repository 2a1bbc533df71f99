// Programmatic dependent launch for the passes of a loop: a kernel launched
// through launch_pdl may start while its predecessor in the stream still runs
// (once every block of that one has called pdl_trigger or ended), so its launch
// latency and the loads of its constant tables overlap the predecessor's tail.
// Such a kernel calls pdl_wait before it touches anything that earlier work in
// the stream reads or writes; the wait returns when the predecessor has
// completed and its writes are visible.  What it reads before must have been
// written by work that completed before the predecessor began (the handle's
// tables).  Data written in the stream must not be read through const
// __restrict__ parameters: the compiler may move such loads above the wait.
#pragma once

#include <cuda_runtime.h>

namespace odt {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_pdl(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace odt
