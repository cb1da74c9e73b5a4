// Memory that sessions and operators come and go in: a device pool of the
// library's own (stream-ordered allocations of the CUDA runtime) and a short
// list of page-locked blocks.  A session takes about sixty buffers; allocating
// and freeing them, and mapping and unmapping the gigabytes of an exact one,
// cost 0.6 ms (600 x 24) to 6 ms (160,000 x 128, precision 1) of every session
// where the same memory had just been freed.
//
// Bounds: at most kDeviceKeep bytes of freed device memory stay with the pool
// (what is above goes back at the next synchronisation), and kHostKeep bytes
// of page-locked memory.  An allocation that fails gives everything unused
// back and tries once more.  Both lists are safe with several threads; a block
// is only freed after its streams have been waited for, so the next owner may
// use it on any stream once its allocation's stream has been waited for.
#include <mutex>
#include <vector>

#include "gm_pool.h"

namespace gm {

namespace {

constexpr unsigned long long kDeviceKeep = 16ull << 30;
constexpr size_t kHostKeep = (size_t)64 << 20;
constexpr int kMaxDevices = 64;

std::mutex g_mu;
cudaMemPool_t g_pools[kMaxDevices] = {};

cudaError_t pool_of(int device, cudaMemPool_t *out) {
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> g(g_mu);
  if (!g_pools[device]) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t p = nullptr;
    cudaError_t e = cudaMemPoolCreate(&p, &props);
    if (e != cudaSuccess) return e;
    unsigned long long keep = kDeviceKeep;
    e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
      cudaMemPoolDestroy(p);
      return e;
    }
    g_pools[device] = p;
  }
  *out = g_pools[device];
  return cudaSuccess;
}

struct HostBlock {
  void *p;
  size_t bytes;
};
std::mutex g_host_mu;
std::vector<HostBlock> g_host;
size_t g_host_bytes = 0;

size_t host_size(size_t bytes) {  // whole 64 KB pages
  return (bytes + 65535) / 65536 * 65536;
}

}  // namespace

cudaError_t device_alloc(void **out, size_t bytes, int device, cudaStream_t s) {
  *out = nullptr;
  cudaMemPool_t p = nullptr;
  cudaError_t e = pool_of(device, &p);
  if (e != cudaSuccess) return e;
  e = cudaMallocFromPoolAsync(out, bytes, p, s);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    cudaMemPoolTrimTo(p, 0);
    e = cudaMallocFromPoolAsync(out, bytes, p, s);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    *out = nullptr;
  }
  return e;
}

void device_free(void *p, cudaStream_t s) {
  if (p) cudaFreeAsync(p, s);
}

cudaError_t host_alloc(void **out, size_t bytes) {
  const size_t want = host_size(bytes);
  {
    std::lock_guard<std::mutex> g(g_host_mu);
    for (size_t i = 0; i < g_host.size(); ++i)
      if (g_host[i].bytes == want) {
        *out = g_host[i].p;
        g_host_bytes -= want;
        g_host.erase(g_host.begin() + (long)i);
        return cudaSuccess;
      }
  }
  const cudaError_t e = cudaHostAlloc(out, want, cudaHostAllocPortable);
  if (e != cudaSuccess) {
    cudaGetLastError();
    *out = nullptr;
  }
  return e;
}

void host_free(void *p, size_t bytes) {
  if (!p) return;
  const size_t size = host_size(bytes);
  {
    std::lock_guard<std::mutex> g(g_host_mu);
    if (g_host_bytes + size <= kHostKeep) {
      g_host.push_back({p, size});
      g_host_bytes += size;
      return;
    }
  }
  cudaFreeHost(p);
}

}  // namespace gm
