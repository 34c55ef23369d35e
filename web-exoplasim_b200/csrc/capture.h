// Graphs and stream capture that an exception leaves in order.
#pragma once
#include <cuda_runtime_api.h>

#include "error.h"

namespace exogcm {

// A graph destroyed with its owner unless released.
class Graph {
 public:
  Graph() = default;
  Graph(const Graph&) = delete;
  Graph& operator=(const Graph&) = delete;
  ~Graph() {
    if (graph_) cudaGraphDestroy(graph_);
  }
  cudaGraph_t get() const { return graph_; }
  cudaGraph_t* out() { return &graph_; }
  cudaGraph_t release() {
    const cudaGraph_t g = graph_;
    graph_ = nullptr;
    return g;
  }

 private:
  cudaGraph_t graph_ = nullptr;
};

// The capture of what is launched on a stream. If the work being captured
// throws, the capture is ended and its graph dropped, so that the stream
// takes work again and the engine's next call fails or succeeds by itself.
class Capture {
 public:
  explicit Capture(cudaStream_t stream) : stream_(stream) {
    check(cudaStreamBeginCapture(stream, cudaStreamCaptureModeRelaxed), "capture");
    open_ = true;
  }
  Capture(const Capture&) = delete;
  Capture& operator=(const Capture&) = delete;
  ~Capture() {
    if (!open_) return;
    Graph dropped;
    cudaStreamEndCapture(stream_, dropped.out());
    cudaGetLastError();
  }
  // Ends the capture; `graph` owns what was captured.
  void end(Graph& graph) {
    open_ = false;
    check(cudaStreamEndCapture(stream_, graph.out()), "capture end");
  }

 private:
  const cudaStream_t stream_;
  bool open_ = false;
};

}  // namespace exogcm
