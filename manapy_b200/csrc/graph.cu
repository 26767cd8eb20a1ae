// CUDA graphs of a solver's steps (host code; no counterpart in manapy).
//
// A capture has a stream to itself while it runs: one from a pool that the program's other threads
// draw from too could be theirs at the same time, and what they launch would become part of the
// graph.  Streams are kept for later captures (making one is a tenth of a short capture).  The mode
// is relaxed, so what other threads do meanwhile (allocate, free another graph) does not
// invalidate the capture.
#include <mutex>

#include "fv_common.cuh"

using namespace mb;

namespace {
// an error is reported by the call that met it, not again by the next one that asks for the last error
int done(cudaError_t e) {
  if (e == cudaSuccess) return MB_OK;
  cudaGetLastError();
  return MB_ECUDA;
}

// While it lives, this thread's calls neither fail for nor invalidate a capture that another thread, or the
// program around a garbage collection that frees a graph, has begun in the global mode.
struct Relaxed {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~Relaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// streams kept for later captures, a few at most (nothing here allocates: no exception at a C entry)
struct Kept {
  int device;
  cudaStream_t stream;
};
constexpr int kMostKept = 16;
Kept kept[kMostKept];
int kept_count = 0;
std::mutex kept_lock;

cudaError_t take_stream(cudaStream_t *s) {
  int device = 0;
  const cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  {
    const std::lock_guard<std::mutex> hold(kept_lock);
    for (int k = 0; k < kept_count; ++k)
      if (kept[k].device == device) {
        *s = kept[k].stream;
        kept[k] = kept[--kept_count];
        return cudaSuccess;
      }
  }
  return cudaStreamCreateWithFlags(s, cudaStreamNonBlocking);
}
void give_stream(cudaStream_t s, bool good) {
  int device = 0;
  if (good && cudaGetDevice(&device) == cudaSuccess) {
    const std::lock_guard<std::mutex> hold(kept_lock);
    if (kept_count < kMostKept) {
      kept[kept_count++] = Kept{device, s};
      return;
    }
  }
  cudaStreamDestroy(s);
}
}  // namespace

extern "C" {

int mb_graph_begin(void **stream) {
  MB_NVTX();
  if (!stream) return MB_EINVAL;
  const Relaxed relaxed;
  cudaStream_t s = nullptr;
  cudaError_t e = take_stream(&s);
  if (e != cudaSuccess) return done(e);
  e = cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed);
  if (e == cudaSuccess) *stream = s;
  else give_stream(s, false);
  return done(e);
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
  give_stream(s, e == cudaSuccess);
  if (graph) *graph = e == cudaSuccess ? x : nullptr;
  return done(e);
}

int mb_graph_launch(void *graph, void *stream) {
  MB_NVTX();
  if (!graph) return MB_EINVAL;
  return done(cudaGraphLaunch(reinterpret_cast<cudaGraphExec_t>(graph), reinterpret_cast<cudaStream_t>(stream)));
}

int mb_graph_free(void *graph) {
  if (!graph) return MB_EINVAL;
  const Relaxed relaxed;
  return done(cudaGraphExecDestroy(reinterpret_cast<cudaGraphExec_t>(graph)));
}

}  // extern "C"
