// Kernel launches with attributes.
#pragma once
#include <cuda_runtime.h>

namespace st {

// Streaming kernel of a chain on `stream`: one priority level under the stream's own.  The chain's short kernels run at that, so
// that their CTAs go ahead of those that a streaming kernel of another chain still has to start.
template <typename Args>
inline cudaError_t launch_streaming(void (*kernel)(Args), int grid, int threads, cudaStream_t stream, const Args& args) {
  int own = 0;
  const cudaError_t e = cudaStreamGetPriority(stream, &own);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributePriority;
  attr.val.priority = own < 0 ? own + 1 : own;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args);
}

}  // namespace st
