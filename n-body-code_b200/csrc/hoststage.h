// Pinned staging buffer of one engine: small host transfers go through it as
// one copy, since a copy from or to pageable memory costs several microseconds
// however small it is.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

namespace nbody {

class HostStage {
 public:
  HostStage() = default;
  HostStage(const HostStage&) = delete;
  HostStage& operator=(const HostStage&) = delete;
  ~HostStage() { cudaFreeHost(p_); }
  // At least `bytes` of pinned memory; the contents do not survive a growth.
  cudaError_t need(size_t bytes) {
    if (bytes <= bytes_) return cudaSuccess;
    cudaFreeHost(p_);
    p_ = nullptr;
    bytes_ = 0;
    const cudaError_t e = cudaMallocHost(&p_, bytes);
    if (e == cudaSuccess) bytes_ = bytes;
    return e;
  }
  double* doubles() const { return static_cast<double*>(p_); }

 private:
  void* p_ = nullptr;
  size_t bytes_ = 0;
};

}  // namespace nbody
