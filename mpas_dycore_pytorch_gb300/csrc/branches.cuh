// Independent kernels of a captured step as branches of its graph.
//
// While the stream is being captured, next() sends the launches that follow back to the point
// where the object was made, so that they do not wait for the ones before, and join()
// makes the launches after it wait for all branches.  The dependencies of the capture are
// edited in place: no further stream or event exists.  Outside a capture nothing happens
// and the launches run in the order they are issued.  Kernels of two branches must not write
// what the other reads or writes.
#pragma once

#include <cuda_runtime.h>

#include <vector>

class GraphBranches {
 public:
  // wanted = false: the launches keep the order they are issued in
  explicit GraphBranches(cudaStream_t s, bool wanted = true) : s_(s) {
    on_ = wanted && current(base_) && !base_.empty();
  }
  bool active() const { return on_; }
  int next() { return on_ && !(collect() && set(base_)) ? MPASG_E_CUDA : MPASG_OK; }
  int join() {
    if (!on_) return MPASG_OK;
    on_ = false;
    return collect() && set(ends_) ? MPASG_OK : MPASG_E_CUDA;
  }

 private:
  // the nodes the next launch waits for; false when nothing is being captured
  bool current(std::vector<cudaGraphNode_t>& out) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    const cudaGraphNode_t* d = nullptr;
    size_t n = 0;
    if (cudaStreamGetCaptureInfo(s_, &st, nullptr, nullptr, &d, nullptr, &n) != cudaSuccess) {
      cudaGetLastError();
      return false;
    }
    if (st != cudaStreamCaptureStatusActive) return false;
    out.assign(d, d + n);
    return true;
  }
  bool collect() {
    std::vector<cudaGraphNode_t> now;
    if (!current(now)) return false;
    for (cudaGraphNode_t x : now) {
      bool known = false;
      for (cudaGraphNode_t y : ends_) known = known || x == y;
      if (!known) ends_.push_back(x);
    }
    return true;
  }
  bool set(std::vector<cudaGraphNode_t>& nodes) {
    return cudaStreamUpdateCaptureDependencies(s_, nodes.data(), nullptr, nodes.size(),
                                               cudaStreamSetCaptureDependencies) == cudaSuccess;
  }

  cudaStream_t s_;
  bool on_ = false;
  std::vector<cudaGraphNode_t> base_, ends_;
};
