// Scratch that one call needs from its first kernel to its last (stream_scratch.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace q4k {

struct CapturedBlock;

// acquire() before the call's first kernel, release() after its last launch: in between p() is the call's own memory,
// whatever other streams, threads and graphs do.  Nothing about its contents may be assumed.
class StreamScratch {
 public:
  // alternate: for calls whose first kernel may run beside the call before it on the stream.  Where alternates() then says
  // so, p() shares nothing with what that call was given.  A call that ends without release(), because a launch failed,
  // makes the next one not alternate.
  cudaError_t acquire(cudaStream_t stream, uint64_t bytes, bool alternate = false);
  bool alternates() const { return alternates_; }
  cudaError_t release();
  void* p() const { return p_; }
  ~StreamScratch() { (void)give_back(); }
  StreamScratch() = default;
  StreamScratch(StreamScratch const&) = delete;
  StreamScratch& operator=(StreamScratch const&) = delete;

 private:
  cudaError_t give_back();
  void* p_ = nullptr;
  cudaStream_t stream_ = nullptr;
  CapturedBlock* block_ = nullptr;
  bool owned_ = false;  // to be freed in stream order
  bool alternate_ = false, alternates_ = false;
};

}  // namespace q4k
