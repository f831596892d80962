// s2d_readback.h -- device fields into the caller's pageable memory.
#pragma once
#include <cstddef>
#include <cuda_runtime.h>

namespace s2d {

// Every solver and ensemble holds one reference to its device's staging for its lifetime; the
// staging is made once its holders have read 16 MB and given back with the last reference.
void readback_retain(int dev);
void readback_release(int dev);

// bytes from device memory src to host memory dst, behind the work `stream` holds now; returns
// when dst is complete.  The current device is `dev`.
cudaError_t read_back(int dev, void* dst, const void* src, size_t bytes, cudaStream_t stream);

}  // namespace s2d
