// user_buffer.h -- what a caller's pointer is, and so how its values travel.
#pragma once
#include <cuda_runtime_api.h>

namespace opfc {

// Kernels of `device` read and write only that device's own memory directly:
// another GPU's needs peer access, which nobody promised, and host or managed
// memory is slower that way than a copy.
inline bool own_device_memory(const cudaPointerAttributes &a, int device) {
  return a.type == cudaMemoryTypeDevice && a.device == device;
}

// page-locked host memory: one asynchronous copy moves it at the link's rate
inline bool pinned_host_memory(const cudaPointerAttributes &a) { return a.type == cudaMemoryTypeHost; }

// attributes of p; an unregistered host pointer where CUDA does not know it
inline cudaPointerAttributes pointer_attributes(const void *p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    a = cudaPointerAttributes{};
    a.type = cudaMemoryTypeUnregistered;
  }
  return a;
}

}  // namespace opfc
