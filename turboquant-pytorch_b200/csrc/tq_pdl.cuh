// Programmatic dependent launch for chains of kernels that one call issues back to back.  The dependent kernel is set up
// while its predecessor still runs and waits (pdl_wait) before it touches what the predecessor wrote; what an earlier
// kernel of the stream wrote is there already, because the first kernel of the chain is an ordinary launch.  The
// predecessor lets it start with pdl_trigger at its own beginning: by then all its CTAs are running, so the dependent
// takes no place from it.  Only a kernel that a launch_after() of the same call follows may trigger: the last kernel of a call
// would let another library's dependent kernel start beside it.  Against ordinary launches of the same kernels, packed
// scores of 131072 keys x 8 heads with softmax took 59.5 instead of 64 us (46 now, the kernels being faster), decode attention of 32640 tokens
// 35 instead of 41 (31 now), three launches each; MSE + QJL: compress and
// scores of 8 x 4096 packed keys 58 instead of 64 (37 now), scores of 16 x 16384 keys 81 instead of 84 (76 now).
#pragma once

#include <cuda_runtime.h>

namespace tq {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch after a kernel of the same call on the same stream.  Under stream capture it is an ordinary launch.
template <typename... P, typename... A>
inline void launch_after(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  const bool plain = cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone;
  if (plain && cap == cudaStreamCaptureStatusNone) cudaGetLastError();      // the query's own error, not the launch's
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = plain ? 0 : 1;
  cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);     // an error is picked up by the caller's check_launch()
}

}  // namespace tq
