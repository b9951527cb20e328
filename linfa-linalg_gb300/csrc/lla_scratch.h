// lla_scratch.h -- device scratch of one launch sequence.
//
// Device entry points may be called by one thread on several streams, and be
// captured in CUDA graphs: scratch that is shared through the thread's context
// would be written by two streams at once.  A StreamScratch is allocated and
// freed in stream order, so every launch sequence has its own.  The memory comes
// from one pool per device that keeps at most kScratchKeepBytes while idle and
// gives the rest back at the next synchronisation, so a repeated call costs no
// cudaMalloc.
//
// In a capture, stream order would put allocation nodes into the caller's graph,
// which could then be neither cloned nor instantiated twice nor used as a child
// graph.  There the memory is allocated beside the capture, and the graph keeps it:
// a user object of the graph hands it back once the graph, its clones and its
// executable instances are gone (to the pool, at the next call on that device: the
// hand-back itself must not call CUDA).  Instances of one captured call share its
// scratch, as they share its operands.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace lla {

constexpr size_t kScratchKeepBytes = 256u << 20;

class StreamScratch {
  public:
    explicit StreamScratch(cudaStream_t st) : st_(st) {}
    ~StreamScratch() {
        if (p_ && !kept_by_graph_) cudaFreeAsync(p_, st_);  // in stream order: after the launches that use it
    }
    StreamScratch(const StreamScratch &) = delete;
    StreamScratch &operator=(const StreamScratch &) = delete;
    cudaError_t alloc(size_t bytes);
    void *get() const { return p_; }

  private:
    cudaStream_t st_;
    void *p_ = nullptr;
    bool kept_by_graph_ = false;
};

}  // namespace lla
