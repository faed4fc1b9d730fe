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

// Kernel behind whatever the stream holds.
template <typename... Params, typename... Args>
inline cudaError_t launch_first(void (*kernel)(Params...), dim3 grid, int threads, cudaStream_t stream, const Args&... args) {
  kernel<<<grid, threads, 0, stream>>>(args...);
  return cudaGetLastError();
}

// Kernel directly behind another kernel of the stream, with no event in between: it may begin while that one ends, see
// behind_previous().  Worth 0.1 to 0.6 % of a captured step; not for emission to peers, see launch_select_one_pass.
template <typename... Params, typename... Args>
inline cudaError_t launch_behind(void (*kernel)(Params...), dim3 grid, int threads, cudaStream_t stream, const Args&... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace st
