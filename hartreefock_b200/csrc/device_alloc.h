// Device memory of the library's own buffers.
#pragma once

#include <cuda_runtime_api.h>

namespace hfg {

// cudaMalloc that, where memory is short, first gives back the idle workspaces
// of the MO transforms on the current device (mo_transform.cu) and tries again.
cudaError_t device_alloc(void **p, size_t bytes);
template <class T>
cudaError_t device_alloc(T **p, size_t bytes) {
  return device_alloc(reinterpret_cast<void **>(p), bytes);
}

}  // namespace hfg
