// Device and page-locked memory of the library's pools (gm_pool.cpp).
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace gm {

// Ready on stream s; on another stream after s has been waited for.
cudaError_t device_alloc(void **out, size_t bytes, int device, cudaStream_t s);
// After every stream that used the block has been waited for.
void device_free(void *p, cudaStream_t s);
cudaError_t host_alloc(void **out, size_t bytes);
void host_free(void *p, size_t bytes);

}  // namespace gm
