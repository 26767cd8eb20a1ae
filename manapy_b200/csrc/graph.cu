// CUDA graphs of a solver's steps (host code; no counterpart in manapy).
//
// A capture has a stream to itself while it runs: one from a pool that the program's other threads
// draw from too could be theirs at the same time, and what they launch would become part of the
// graph.  Streams are kept for later captures, as many a device as ever ran at once.  The mode is
// relaxed, so what other threads do meanwhile (allocate, free another graph) does not invalidate
// the capture.
#include <mutex>
#include <vector>

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

struct Kept {
  int device;
  cudaStream_t stream;
};
std::mutex kept_lock;
std::vector<Kept> &kept() {      // never destroyed: a thread may end its capture while the process exits
  static auto *v = new std::vector<Kept>;
  return *v;
}
cudaError_t take_stream(cudaStream_t *s) {
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  {
    const std::lock_guard<std::mutex> hold(kept_lock);
    for (size_t k = 0; k < kept().size(); ++k)
      if (kept()[k].device == device) {
        *s = kept()[k].stream;
        kept()[k] = kept().back();
        kept().pop_back();
        return cudaSuccess;
      }
  }
  return cudaStreamCreateWithFlags(s, cudaStreamNonBlocking);
}
void keep_stream(cudaStream_t s) {
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return;
  const std::lock_guard<std::mutex> hold(kept_lock);
  kept().push_back(Kept{device, s});
}
}  // namespace

extern "C" {

int mb_graph_begin(void **stream) {
  MB_NVTX();
  if (!stream) return MB_EINVAL;
  const Relaxed relaxed;
  cudaStream_t s = nullptr;
  if (take_stream(&s) != cudaSuccess) return MB_ECUDA;
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
  if (e == cudaSuccess) keep_stream(s); else cudaStreamDestroy(s);
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
