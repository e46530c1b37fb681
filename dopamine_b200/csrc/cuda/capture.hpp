// A sequence of launches as an executable graph.
#pragma once
#include <cuda_runtime_api.h>

namespace dpm {
namespace gpu {

// What enqueue() launches on st, captured and instantiated; null when that fails at any step, with the
// error cleared, so that the caller can enqueue the launches themselves.
template <class F>
cudaGraphExec_t capture_graph(cudaStream_t st, F enqueue) {
  cudaGraph_t g = nullptr;
  cudaGraphExec_t exec = nullptr;
  bool ok = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal) == cudaSuccess;
  if (ok) {
    enqueue();
    ok = cudaStreamEndCapture(st, &g) == cudaSuccess && g;
  }
  if (ok) ok = cudaGraphInstantiate(&exec, g, 0) == cudaSuccess;
  if (g) cudaGraphDestroy(g);
  if (ok) return exec;
  cudaGetLastError();
  return nullptr;
}

}  // namespace gpu
}  // namespace dpm
