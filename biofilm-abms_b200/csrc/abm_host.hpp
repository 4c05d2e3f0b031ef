// Device-to-host copies of frames and tables (abm_host.cpp)
#pragma once
#include <cstddef>
#include <cuda_runtime.h>

namespace abm {

// `height` rows of `width` bytes from device memory to host memory of any kind, after what
// `st` holds; returns when they have arrived
cudaError_t copy_to_host(int dev, void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
                         size_t height, cudaStream_t st);
// the contexts of the process: the last to go gives the shared pinned memory back
void host_copy_retain();
void host_copy_release();

}   // namespace abm
