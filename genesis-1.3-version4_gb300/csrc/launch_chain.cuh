// Launches of the step's kernels one behind the other. A run of few slices is a chain of
// kernels of a few microseconds each, and between two of them the chip waits for the first to
// drain, for its writes and for the launch of the second. With chain_launch the second kernel's
// CTAs become resident while the first still runs: every kernel that is launched so calls
// chain_wait before it touches memory that an earlier kernel may write or read (the wait ends
// when the earlier grid has completed and its writes are visible), and chain_next once it no
// longer needs what the next kernel's CTAs could take from it (tensor memory: after its
// allocation). All CTAs of a kernel have started before the next one's appear, so no CTA can
// wait for one that has no room. Kernels launched in the ordinary way wait for all of it.
//
// Used by the mixed form's push and field step: 221 steps of one slice of 151^2 4.50 -> 4.16 ms,
// 48 steps of 150 slices of 117^2 with its copies 4.95 -> 4.66 ms, windows that fill the chip
// unchanged. The FP64 push and segmented ADI wait likewise but never call chain_next: their
// successors appear when the last CTA has ended, without the launch in between (a step without
// records of 1 x 8192 particles, 255^2 67.4 -> 60.5 us, 22 x 2052, 101^2 70.5 -> 66.3). With
// chain_next at their start CTAs placed beside the running kernel's shared an SM's FP64 pipe
// where they would have had one each: 60 steps of 22 slices with records 6.46 -> 8.16 ms.
#pragma once
#include <cuda_runtime.h>

namespace g4 {

__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// cluster: CTAs of a cluster, 0 for none
template <class... P, class... A>
inline void chain_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, int cluster,
                         A... args) {
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim = {(unsigned)(cluster ? cluster : 1), 1, 1};
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = cluster ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace g4
