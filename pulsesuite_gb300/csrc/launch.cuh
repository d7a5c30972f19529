// Launches of the step's kernels.
#pragma once
#include <cuda_runtime.h>

namespace sbe {

// First statement of every kernel that launch() starts: waits until the kernel before has ended
// and its writes are visible.  Every kernel of the chain waits, so a kernel that runs has all
// earlier ones behind it; a plainly launched kernel passes straight through.
__device__ __forceinline__ void pdl_enter() { cudaGridDependencySynchronize(); }

// k<<<grid, block, smem, s>>>(args...) as a programmatic dependent launch: the launch of k is set
// up while the kernel before it runs, and its blocks are placed as that one's last blocks end.
// A step is 41 to 73 launches, most of a few us.  Gain, measured when a step was 40 to 560: 1 x 64
// mixed 647 -> 446 us, FP64 491 -> 386 us, a sweep of 64 mixed wires 5.23 -> 4.09 ms, 32 x 512
// 8.29 -> 8.03 ms.  No kernel triggers its
// dependents before its end: blocks placed in the slots that are left over pile up on the SMs
// that have some (1 x 64 mixed 490 us, 32 x 512 8.19 ms with an early trigger in every kernel of
// at most 152 blocks).
template <class... P, class... A>
inline cudaError_t launch(void (*k)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                          A&&... args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, static_cast<P>(args)...);
}

}  // namespace sbe
