// Launches whose set-up overlaps the end of the kernel before them (programmatic dependent launch).  A kernel launched with
// ``launch_next`` may be placed on SMs while its predecessor in the stream still runs; it calls ``chain_begin`` in every thread
// before it touches global memory, which returns once the predecessor has finished and its writes are visible, and lets its own
// successor be placed in turn.  Every CTA does so before it exits: a kernel is finished only when those before it are.  What is
// saved is the launch latency and the prologue (barriers, tensor memory): 313 launches of a four-block step of width 1024
// 12.38 -> 12.08 ms, four of attention over 128 heads of 640 tokens 197 -> 192 us, the routed layer of 200 tokens 186 -> 169.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace b2 {

__device__ __forceinline__ void chain_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... Params, typename... Args>
static inline cudaError_t launch_next(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                      Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace b2
