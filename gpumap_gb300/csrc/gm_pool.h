// Device and page-locked memory of the library's pools (gm_pool.cpp).
#pragma once

#include <cstddef>
#include <cuda_runtime.h>

namespace gm {

// Ready on stream s; on another stream after s has been waited for.
cudaError_t device_alloc(void **out, size_t bytes, int device, cudaStream_t s);
// The n-th device_alloc from here on in the calling thread fails with
// cudaErrorMemoryAllocation (n < 0: the next -n do, 0: none; tests).
void device_fail_in(int n);
// After every stream that used the block has been waited for.
void device_free(void *p, cudaStream_t s);
// After a session's `bytes` were freed and its stream waited for: gives back
// what the pool holds beyond what it keeps for the next session.
void device_closed(int device, size_t bytes);
// After an operator freed `bytes` of scratch: gives back what is above the most
// that a pool may keep (small operators take what is there and are not worth
// the question).
void device_bound(int device, size_t bytes);
// Bytes the device's pool holds, and those of them in use.
cudaError_t device_held(int device, size_t *reserved, size_t *used);
cudaError_t host_alloc(void **out, size_t bytes);
void host_free(void *p, size_t bytes);
// Waits for the devices and gives back everything unused, on the host too.
cudaError_t memory_release();

}  // namespace gm
