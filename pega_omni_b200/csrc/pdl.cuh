// Programmatic dependent launch. A kernel started with launch_pdl() may begin while the kernel before it in the stream
// (or graph) is still running: everything it does before grid_wait() overlaps that kernel's tail - barrier and TMEM
// set-up, descriptor and weight fetches - and grid_wait() returns once the kernel before it has completed and its writes
// are visible. The rules every kernel launched this way keeps:
//   - before grid_wait() it reads only what no kernel of the same stream writes (weights, tables, staged inputs), and
//     writes nothing to global memory;
//   - every CTA passes grid_wait() in at least one thread before it ends, on every path, so that a kernel's completion
//     implies that of all kernels before it;
//   - grid_trigger() comes first: it lets the next kernel be scheduled as soon as all CTAs of this one have started
//     (what the next kernel reads is ordered by its own grid_wait(), not by the trigger).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace omni {

__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... Params, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace omni
