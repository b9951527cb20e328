// lla_scratch.h -- stream-ordered device scratch of one launch sequence.
//
// Device entry points may be called by one thread on several streams, and be
// captured in CUDA graphs: scratch that is shared through the thread's context
// would be written by two streams at once.  A StreamScratch is allocated and
// freed in stream order (in a capture: by nodes of the graph), so every launch
// sequence has its own.  The memory comes from one pool per device that keeps
// at most kScratchKeepBytes while idle and gives the rest back at the next
// synchronisation, so a repeated call costs no cudaMalloc.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace lla {

constexpr size_t kScratchKeepBytes = 256u << 20;

class StreamScratch {
  public:
    explicit StreamScratch(cudaStream_t st) : st_(st) {}
    ~StreamScratch() {
        if (p_) cudaFreeAsync(p_, st_);  // in stream order: after the launches that use it
    }
    StreamScratch(const StreamScratch &) = delete;
    StreamScratch &operator=(const StreamScratch &) = delete;
    cudaError_t alloc(size_t bytes);
    void *get() const { return p_; }

  private:
    cudaStream_t st_;
    void *p_ = nullptr;
};

}  // namespace lla
