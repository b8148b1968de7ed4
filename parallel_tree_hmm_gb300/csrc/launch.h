// Where a kernel launch goes: to a stream, or into a graph under construction.
//
// A workspace replays its device step from a CUDA graph (runtime.cc). The graph
// is built node by node from the step's own launches and not by capturing them:
// while a stream of the device is being captured, a device-wide synchronisation
// by any other thread fails and invalidates the capture, whatever its mode.
#ifndef THMM_LAUNCH_H_
#define THMM_LAUNCH_H_

#include <cstddef>

#include <cuda_runtime.h>

namespace thmm {

// A graph of nodes that run one after the other.
struct GraphChain {
  cudaGraph_t graph = nullptr;
  cudaGraphNode_t last = nullptr;
  GraphChain() = default;
  GraphChain(const GraphChain &) = delete;
  GraphChain &operator=(const GraphChain &) = delete;
  ~GraphChain() {
    if (graph != nullptr)
      static_cast<void>(cudaGraphDestroy(graph));
  }
  std::size_t Dependencies() const { return last != nullptr ? 1 : 0; }
};

struct LaunchStream {
  LaunchStream(cudaStream_t launch_stream) : stream(launch_stream) {}
  explicit LaunchStream(GraphChain *launch_chain) : chain(launch_chain) {}
  cudaStream_t stream = nullptr;
  GraphChain *chain = nullptr; // null: launches go to `stream`
};

#if defined(__CUDACC__)
// Launches `kernel` with `threads` threads a block on `to`, or appends it.
template <class Args>
cudaError_t LaunchOn(const LaunchStream &to, void (*kernel)(Args), unsigned grid,
                     unsigned threads, std::size_t smem, const Args &args) {
  if (to.chain == nullptr) {
    kernel<<<grid, threads, smem, to.stream>>>(args);
    return cudaGetLastError();
  }
  void *parameters[] = {const_cast<Args *>(&args)}; // copied into the node
  cudaKernelNodeParams node{};
  node.func = reinterpret_cast<void *>(kernel);
  node.gridDim = dim3(grid);
  node.blockDim = dim3(threads);
  node.sharedMemBytes = static_cast<unsigned>(smem);
  node.kernelParams = parameters;
  cudaGraphNode_t previous = to.chain->last;
  return cudaGraphAddKernelNode(&to.chain->last, to.chain->graph, &previous,
                                to.chain->Dependencies(), &node);
}
#endif

// Zeroes `words` 4-byte words at `p`.
inline cudaError_t ClearOn(const LaunchStream &to, void *p, std::size_t words) {
  if (to.chain == nullptr)
    return cudaMemsetAsync(p, 0, words * 4, to.stream);
  cudaMemsetParams node{};
  node.dst = p;
  node.elementSize = 4;
  node.width = words;
  node.height = 1;
  cudaGraphNode_t previous = to.chain->last;
  return cudaGraphAddMemsetNode(&to.chain->last, to.chain->graph, &previous,
                                to.chain->Dependencies(), &node);
}

} // namespace thmm

#endif // THMM_LAUNCH_H_
