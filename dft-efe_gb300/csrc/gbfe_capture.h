// gbfe_capture.h -- capture of a stream's launches into a graph that an exception
// cannot leave open.
#pragma once
#include <cuda_runtime_api.h>

namespace gbfe {

// Captures `stream` from begin() to end(), with `flag` set meanwhile.  Left without
// end() (an exception on the way), the destructor ends the capture and drops the graph,
// so that the stream takes launches again.
class CaptureScope {
 public:
  CaptureScope(cudaStream_t stream, bool &flag) : stream_(stream), flag_(flag) {}
  ~CaptureScope() {
    cudaGraph_t graph = nullptr;
    if (!open_) return;
    (void)end(&graph);
    if (graph) cudaGraphDestroy(graph);
    (void)cudaGetLastError();
  }
  CaptureScope(const CaptureScope &) = delete;
  CaptureScope &operator=(const CaptureScope &) = delete;
  cudaError_t begin() {
    const cudaError_t e = cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal);
    open_ = flag_ = e == cudaSuccess;
    return e;
  }
  cudaError_t end(cudaGraph_t *graph) {
    open_ = flag_ = false;
    return cudaStreamEndCapture(stream_, graph);
  }

 private:
  cudaStream_t stream_;
  bool &flag_;
  bool open_ = false;
};

// a value that is put back on every way out
template <class T>
class Restore {
 public:
  Restore(T &ref, T value) : ref_(ref), old_(ref) { ref = value; }
  ~Restore() { ref_ = old_; }
  Restore(const Restore &) = delete;
  Restore &operator=(const Restore &) = delete;

 private:
  T &ref_;
  T old_;
};

}  // namespace gbfe
