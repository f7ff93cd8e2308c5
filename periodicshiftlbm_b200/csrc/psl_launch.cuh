// Programmatic dependent launch: a kernel launched as dependent may have its blocks resident
// before the kernel ahead of it in the stream has finished, so its launch and start-up overlap
// that one's last blocks.
//
// Rules every kernel here follows.  A kernel calls grid_wait before it reads or writes
// anything another kernel writes or reads, in every block (so that its own completion implies
// that of the kernel ahead), and grid_release after it, so that the blocks of the next kernel
// start only once everything before this kernel is complete and visible.  Both are no-ops in a
// kernel launched the ordinary way.
//
// One exception: the training samples, which grad_kernel reads before grid_wait (psl_train.cu).
// Whoever writes them waits for the device before returning to the caller, so no kernel that a
// grad_kernel can overlap writes them.
#pragma once
#include <cuda_runtime.h>

namespace psl {

#if defined(__CUDACC__)
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The same for a kernel whose loads are inline assembly addressed from `index`: the value comes
// out of the wait, so none of them can be scheduled ahead of it.
__device__ __forceinline__ void grid_wait(unsigned int& index) {
  asm volatile("griddepcontrol.wait;" : "+r"(index) : : "memory");
}
__device__ __forceinline__ void grid_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

// Whether work queued on the stream is being recorded into a graph (or that cannot be told):
// launches are then made the ordinary way.
inline bool stream_capturing(cudaStream_t stream) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(stream, &cap) == cudaSuccess) return cap != cudaStreamCaptureStatusNone;
  cudaGetLastError();
  return true;
}

template <typename... P, typename... A>
cudaError_t launch_dependent(bool dependent, void (*kernel)(P...), dim3 blocks, unsigned int threads, size_t smem,
                             cudaStream_t stream, const A&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = blocks;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = dependent ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace psl
