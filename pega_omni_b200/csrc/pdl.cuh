// Programmatic dependent launch. A kernel started with launch_pdl() may begin while the kernel before it in the stream
// (or graph) is still running: everything it does before grid_wait() overlaps that kernel's tail - barrier and TMEM
// set-up, descriptor and weight fetches - and grid_wait() returns once the kernel before it has completed and its writes
// are visible.
// The rules every kernel launched this way keeps:
//   - before grid_wait() it reads only what no kernel of the same call writes - weights, tables, staged inputs, and what
//     earlier calls left (a call starts behind a copy in its stream, which is ordered behind everything before it) - and
//     writes nothing to global memory;
//   - behind grid_wait(), what an earlier kernel of the call wrote is read past L1 (__ldcg, ld8cg) and through no pointer
//     declared const __restrict__: that tells the compiler that nothing writes the data while the kernel lives, which it does;
//   - behind grid_wait(), TMA and bulk copies of what an earlier kernel of the call wrote come behind fence_async_global()
//     in the thread that issues them (sm100.cuh);
//   - at least one thread of it passes grid_wait() on every path, so that its completion implies that of all kernels
//     before it;
//   - grid_trigger() comes first, or as soon as the CTA holds its TMEM columns: it lets the next kernel be scheduled once
//     all CTAs of this one have started (what the next kernel reads is ordered by its own grid_wait(), not by the trigger).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace omni {

__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// `whole_smem`: the SM's carve-out shall be all of its shared memory, not the smallest that holds this kernel's CTA (the default),
// so that the next kernel's CTAs find room beside it.
template <typename... Params, typename... Args>
inline cudaError_t launch_pdl_smem(bool whole_smem, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                   Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  attr[1].val.sharedMemCarveout = 100;
  cfg.attrs = attr;
  cfg.numAttrs = whole_smem ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
template <typename... Params, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args&&... args) {
  return launch_pdl_smem(false, kernel, grid, block, smem, stream, std::forward<Args>(args)...);
}

}  // namespace omni
