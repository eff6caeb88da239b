// Stream capture and replay of a recorded pass (ops/graph.py).
//
// A pass of a small model is a few hundred kernels of 3 - 15 us, and launching one from Python costs about 25 us of host
// time (wrapper, tensor maps, cudaLaunchKernelEx); replaying the recording costs the host one call.  Capture is in
// relaxed mode, so that what other threads do meanwhile (a data loader pinning memory) neither fails nor ends it.
#include <cuda_runtime.h>

extern "C" int grb_capture_begin(void* stream) {
  return cudaStreamBeginCapture(reinterpret_cast<cudaStream_t>(stream), cudaStreamCaptureModeRelaxed) == cudaSuccess ? 0 : -60;
}

// Ends the capture on `stream`; *exec receives the executable graph (null if the capture was invalidated).
extern "C" int grb_capture_end(void* stream, void** exec) {
  *exec = nullptr;
  cudaGraph_t graph = nullptr;
  if (cudaStreamEndCapture(reinterpret_cast<cudaStream_t>(stream), &graph) != cudaSuccess || !graph) {
    cudaGetLastError();
    return -61;
  }
  cudaGraphExec_t ex = nullptr;
  const cudaError_t rc = cudaGraphInstantiate(&ex, graph, 0);
  cudaGraphDestroy(graph);
  if (rc != cudaSuccess) {
    cudaGetLastError();
    return -62;
  }
  *exec = ex;
  return 0;
}

extern "C" int grb_graph_launch(void* exec, void* stream) {
  return cudaGraphLaunch(reinterpret_cast<cudaGraphExec_t>(exec), reinterpret_cast<cudaStream_t>(stream)) == cudaSuccess ? 0 : -63;
}

// A launch still in flight keeps the graph alive until it has finished.
extern "C" int grb_graph_destroy(void* exec) {
  return !exec || cudaGraphExecDestroy(reinterpret_cast<cudaGraphExec_t>(exec)) == cudaSuccess ? 0 : -64;
}

extern "C" int grb_is_capturing(void* stream) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(reinterpret_cast<cudaStream_t>(stream), &st) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return st != cudaStreamCaptureStatusNone;
}
