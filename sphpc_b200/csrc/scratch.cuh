// scratch.cuh -- device memory for the length of one call (scratch.cu).
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace sphpc {

// One buffer of device memory in stream order: taken on a stream, given back on
// the same stream when the object ends, so work enqueued on it in between may
// use it.
class CallScratch {
 public:
  CallScratch() = default;
  CallScratch(const CallScratch&) = delete;
  CallScratch& operator=(const CallScratch&) = delete;
  ~CallScratch();
  cudaError_t take(size_t bytes, cudaStream_t stream);
  template <class T>
  T* at(size_t offset) const {
    return reinterpret_cast<T*>(static_cast<char*>(p_) + offset);
  }

 private:
  void* p_ = nullptr;
  cudaStream_t stream_ = nullptr;
  bool pooled_ = false;
};

// Offsets of the parts of one buffer, each aligned to 256 bytes.
class ScratchLayout {
 public:
  size_t part(size_t bytes) {
    const size_t at = used_;
    used_ += (bytes + 255) & ~(size_t)255;
    return at;
  }
  size_t bytes() const { return used_; }

 private:
  size_t used_ = 0;
};

}  // namespace sphpc
