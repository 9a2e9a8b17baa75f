// One device allocation for the buffers of a call.
#pragma once
#include <cuda_runtime.h>
#include <string.h>

#include <vector>

#include "qg_internal.h"

namespace qg {

// Buffers are declared first (add, upload), then allocated together: a
// cudaMalloc and cudaFree per buffer and a copy per small input were a third of
// the smallest scatters.  Inputs given to upload() lie at the front and go to
// the device in one copy.  The memory is the call's own and freed with the
// arena.
class DevArena {
 public:
  ~DevArena() {
    if (base_) cudaFree(base_);
  }
  // Reserves `bytes`; returns the buffer's offset.
  size_t add(size_t bytes) {
    const size_t at = size_;
    size_ += (bytes + 255) / 256 * 256;
    return at;
  }
  // Reserves a copy of `bytes` bytes at p; before any add().
  size_t upload(const void *p, size_t bytes) {
    const size_t at = add(bytes);
    host_.resize(size_, 0);
    if (bytes) memcpy(host_.data() + at, p, bytes);
    return at;
  }
  int alloc(cudaStream_t st) {
    QG_CUDA_TRY(cudaMalloc(&base_, size_ ? size_ : 16));
    if (!host_.empty()) QG_CUDA_TRY(cudaMemcpyAsync(base_, host_.data(), host_.size(), cudaMemcpyHostToDevice, st));
    return QPMS_SUCCESS;
  }
  template <typename T>
  T *at(size_t offset) const {
    return reinterpret_cast<T *>(static_cast<char *>(base_) + offset);
  }

 private:
  void *base_ = nullptr;
  size_t size_ = 0;
  std::vector<char> host_;
};

}  // namespace qg
