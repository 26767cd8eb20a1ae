// CUDA graphs of a solver's steps (host code; no counterpart in manapy).
//
// A capture runs on a stream made for it: one from a pool that the program's other threads draw from
// too could be theirs at the same time, and what they launch would become part of the graph.  The
// mode is relaxed, so what other threads do meanwhile (allocate, free another graph) does not
// invalidate the capture.  Nothing here is shared between captures, so threads need no lock.
#include "fv_common.cuh"

using namespace mb;

namespace {
// While it lives, this thread's calls neither fail for nor invalidate a capture that another thread, or the
// program around a garbage collection that frees a graph, has begun in the global mode.
struct Relaxed {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
}  // namespace

extern "C" {

int mb_graph_begin(void **stream) {
  MB_NVTX();
  if (!stream) return MB_EINVAL;
  const Relaxed relaxed;
  cudaStream_t s = nullptr;
  if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return MB_ECUDA;
  if (cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed) != cudaSuccess) {
    cudaStreamDestroy(s);
    return MB_ECUDA;
  }
  *stream = s;
  return MB_OK;
}

int mb_graph_end(void *stream, void **graph) {
  MB_NVTX();
  if (!stream) return MB_EINVAL;
  const Relaxed relaxed;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  cudaGraph_t g = nullptr;
  cudaGraphExec_t x = nullptr;
  cudaError_t e = cudaStreamEndCapture(s, &g);
  if (e == cudaSuccess && graph) e = cudaGraphInstantiate(&x, g, 0);
  if (g) cudaGraphDestroy(g);
  cudaStreamDestroy(s);
  if (graph) *graph = e == cudaSuccess ? x : nullptr;
  return e == cudaSuccess ? MB_OK : MB_ECUDA;
}

int mb_graph_launch(void *graph, void *stream) {
  MB_NVTX();
  if (!graph) return MB_EINVAL;
  return cudaGraphLaunch(reinterpret_cast<cudaGraphExec_t>(graph), reinterpret_cast<cudaStream_t>(stream)) == cudaSuccess
             ? MB_OK
             : MB_ECUDA;
}

int mb_graph_free(void *graph) {
  if (!graph) return MB_EINVAL;
  const Relaxed relaxed;
  return cudaGraphExecDestroy(reinterpret_cast<cudaGraphExec_t>(graph)) == cudaSuccess ? MB_OK : MB_ECUDA;
}

}  // extern "C"
