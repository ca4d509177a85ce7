// Launches of one step after another (programmatic dependent launch): a step's
// blocks may be placed, and read what no step writes, while the step before
// it still runs; chain_wait holds them until it has finished and its writes
// are visible.  chain_next, after the wait, lets the step after this one be
// placed in turn (after the wait, so that at most one step is ahead).
//
// What the launch before writes is read by ordinary loads (its pointers are
// not __restrict__, no __ldg): the read-only path is for data that stays as it
// is from a launch's first block to its last, and the first blocks may be
// there before the last write.
//
// What it saves is the gap between dependent launches, most of a small step:
// 32 x 32 cloth 6.2 -> 4.1 us a step, 157 x 211 6.2 -> 4.5, 500 x 500 16.4 ->
// 13.6, 1024 x 1024 51.3 -> 47.5, 24 cloths of 16..48 vertices a side (in a
// graph) 6.1 -> 4.5.
#pragma once

#include <cuda_runtime.h>

namespace fgb {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// kernel<<<blocks, threads, smem, s>>>(args...), chained to the launch before
// it when `chained`.
template <class... P, class... A>
cudaError_t chain_launch(void (*kernel)(P...), int blocks, int threads, size_t smem, cudaStream_t s, bool chained,
                         A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(unsigned(blocks));
  cfg.blockDim = dim3(unsigned(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace fgb
