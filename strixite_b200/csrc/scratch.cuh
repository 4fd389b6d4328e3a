// Stream-ordered scratch memory for the entry points whose callers hand over activations in a form that a kernel cannot
// read at speed (row-major BF16 into the tcgen05 kernels): the operand form is written once per call into memory that lives
// until the work enqueued before its release has run.
//
// The memory comes from a pool of this library's own, one per device, through the runtime's stream-ordered allocator: an
// allocation is ordered on the stream it is made on, so calls from several threads and streams never share live memory.
// A captured call gets none (scratch.cu).  The pool keeps at most kKeepBytes between calls; what lies above that goes back to the
// device at the next synchronization, all of it with sxb_release_scratch.
#pragma once

#include "common.cuh"

namespace sxb {

class StreamScratch {
  public:
    StreamScratch() = default;
    StreamScratch(const StreamScratch &) = delete;
    StreamScratch &operator=(const StreamScratch &) = delete;
    ~StreamScratch();  // enqueues the release on the stream of the allocation
    // False when there is none to be had (out of memory, a capturing stream, inside a NoScratch): no error is left behind.
    bool get(size_t bytes, cudaStream_t stream);
    void *ptr() const { return p_; }

  private:
    void *p_ = nullptr;
    cudaStream_t stream_ = nullptr;
};

// While one of these lives, StreamScratch::get of this thread returns false (the allocation-free entry points).
class NoScratch {
  public:
    NoScratch();
    ~NoScratch();
};

}  // namespace sxb
