// Whether a kernel may read and write an array that a caller names by address.
#pragma once
#include <cuda_runtime_api.h>

namespace nbody {

// p is memory of device `dev` itself, or managed memory.  A kernel that touches
// another device's memory or the host's, where no mapping was set up, faults;
// the runtime's copies check.  get: cudaPointerGetAttributes.
template <class Get>
inline bool local_to(const void* p, int dev, Get&& get) {
  cudaPointerAttributes at{};
  if (get(&at, p) != cudaSuccess) {
    cudaGetLastError();  // not a failure of the calls that follow
    return false;
  }
  return at.type == cudaMemoryTypeManaged || (at.type == cudaMemoryTypeDevice && at.device == dev);
}

}  // namespace nbody
