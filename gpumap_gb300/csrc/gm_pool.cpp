// Memory that sessions and operators come and go in: a device pool of the
// library's own (stream-ordered allocations of the CUDA runtime) and a short
// list of page-locked blocks.  A session takes about sixty buffers; allocating
// and freeing them, and mapping and unmapping the gigabytes of an exact one,
// cost 0.6 ms (600 x 24) to 6 ms (160,000 x 128, precision 1) of every session
// where the same memory had just been freed.
//
// Unused device memory that stays with a pool: as much as brings it back to the
// most that was in use at any of the last kCloses closes (a program that drops
// several sessions together, as a garbage collection does, opens as many again),
// and never more than a 16th of the device's memory: sessions beyond that take
// long to fill, and their memory is not worth keeping from others.  Each close
// gives back what is above.  With what the last session held as the rule, the
// 160,000 x 128 builds mapped a session again after every collection: 31.6 ms
// each instead of 30.4.  kHostKeep bounds the page-locked blocks.
// An allocation that fails, and memory_release(), give everything unused back.
//
// Both lists are safe with several threads; a block is only freed after its
// streams have been waited for, so the next owner may use it on any stream once
// its allocation's stream has been waited for.
#include <algorithm>
#include <mutex>
#include <vector>

#include "gm_pool.h"

namespace gm {

namespace {

constexpr size_t kHostKeep = (size_t)64 << 20;
constexpr size_t kDeviceShare = 16;
constexpr int kCloses = 16;
constexpr size_t kPoolSlack = (size_t)64 << 20;
constexpr int kMaxDevices = 64;

struct DevicePool {
  cudaMemPool_t pool = nullptr;
  size_t most = 0;              // a 16th of the device's memory
  size_t in_use[kCloses] = {};  // bytes in use before each of the last closes
  int next = 0;
};
std::mutex g_mu;
DevicePool g_pools[kMaxDevices];

// The device's pool, made on first use (g_mu held).
cudaError_t pool_of(int device, DevicePool **out) {
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  DevicePool &d = g_pools[device];
  if (!d.pool) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t p = nullptr;
    cudaError_t e = cudaMemPoolCreate(&p, &props);
    if (e != cudaSuccess) return e;
    // (the runtime gives nothing back by itself: its threshold counts the memory
    // in use as well)
    unsigned long long never = ~0ull;
    e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &never);
    size_t free_b = 0, total = 0;
    if (e == cudaSuccess) e = cudaMemGetInfo(&free_b, &total);
    if (e != cudaSuccess) {
      cudaMemPoolDestroy(p);
      return e;
    }
    d.pool = p;
    d.most = total / kDeviceShare;
  }
  *out = &d;
  return cudaSuccess;
}

void held(cudaMemPool_t p, size_t *reserved, size_t *used) {
  unsigned long long r = 0, u = 0;
  cudaMemPoolGetAttribute(p, cudaMemPoolAttrReservedMemCurrent, &r);
  cudaMemPoolGetAttribute(p, cudaMemPoolAttrUsedMemCurrent, &u);
  *reserved = (size_t)r;
  *used = (size_t)u;
}

// At most `keep` unused bytes stay.
void trim(cudaMemPool_t p, size_t keep) {
  size_t reserved = 0, used = 0;
  held(p, &reserved, &used);
  if (reserved > used + keep) cudaMemPoolTrimTo(p, used + keep);
}

struct HostBlock {
  void *p;
  size_t bytes;
};
std::mutex g_host_mu;
size_t g_host_bytes = 0;
std::vector<HostBlock> &host_blocks() {  // (never destroyed: a session may go after the statics)
  static std::vector<HostBlock> *v = new std::vector<HostBlock>;
  return *v;
}

void host_release() {
  std::lock_guard<std::mutex> g(g_host_mu);
  for (const HostBlock &b : host_blocks()) cudaFreeHost(b.p);
  host_blocks().clear();
  g_host_bytes = 0;
}

size_t host_size(size_t bytes) {  // whole 64 KB pages
  return (bytes + 65535) / 65536 * 65536;
}

}  // namespace

namespace {
thread_local int g_fail_in = 0;
}
void device_fail_in(int n) { g_fail_in = n; }

cudaError_t device_alloc(void **out, size_t bytes, int device, cudaStream_t s) {
  *out = nullptr;
  if (g_fail_in > 0 && --g_fail_in == 0) return cudaErrorMemoryAllocation;
  if (g_fail_in < 0) {
    ++g_fail_in;
    return cudaErrorMemoryAllocation;
  }
  cudaMemPool_t p = nullptr;
  {
    std::lock_guard<std::mutex> g(g_mu);
    DevicePool *d = nullptr;
    const cudaError_t e = pool_of(device, &d);
    if (e != cudaSuccess) return e;
    p = d->pool;
  }
  cudaError_t e = cudaMallocFromPoolAsync(out, bytes, p, s);
  if (e == cudaErrorMemoryAllocation) {
    // a freed block goes back to the device once its free has been waited for
    cudaGetLastError();
    cudaDeviceSynchronize();
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

void device_closed(int device, size_t bytes) {
  std::lock_guard<std::mutex> g(g_mu);
  if (device < 0 || device >= kMaxDevices || !g_pools[device].pool) return;
  DevicePool &d = g_pools[device];
  size_t reserved = 0, used = 0;
  held(d.pool, &reserved, &used);
  d.in_use[d.next] = used + bytes;
  d.next = (d.next + 1) % kCloses;
  size_t peak = *std::max_element(d.in_use, d.in_use + kCloses);
  // (the pool's blocks are somewhat larger than what lies in them)
  peak += peak / 8 + kPoolSlack;
  trim(d.pool, std::min(d.most, peak > used ? peak - used : 0));
}

void device_bound(int device, size_t bytes) {
  if (bytes < kPoolSlack) return;
  std::lock_guard<std::mutex> g(g_mu);
  if (device < 0 || device >= kMaxDevices || !g_pools[device].pool) return;
  trim(g_pools[device].pool, g_pools[device].most);
}

cudaError_t device_held(int device, size_t *reserved, size_t *used) {
  std::lock_guard<std::mutex> g(g_mu);
  *reserved = *used = 0;
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  if (g_pools[device].pool) held(g_pools[device].pool, reserved, used);
  return cudaSuccess;
}

cudaError_t memory_release() {
  cudaError_t first = cudaSuccess;
  {
    std::lock_guard<std::mutex> g(g_mu);
    int current = 0;
    const bool back = cudaGetDevice(&current) == cudaSuccess;
    for (int dev = 0; dev < kMaxDevices; ++dev) {
      if (!g_pools[dev].pool) continue;
      cudaError_t e = cudaSetDevice(dev);
      if (e == cudaSuccess) e = cudaDeviceSynchronize();
      if (e == cudaSuccess) e = cudaMemPoolTrimTo(g_pools[dev].pool, 0);
      if (first == cudaSuccess) first = e;
    }
    if (back) cudaSetDevice(current);
  }
  host_release();
  return first;
}

cudaError_t host_alloc(void **out, size_t bytes) {
  const size_t want = host_size(bytes);
  {
    std::lock_guard<std::mutex> g(g_host_mu);
    std::vector<HostBlock> &v = host_blocks();
    for (size_t i = 0; i < v.size(); ++i)
      if (v[i].bytes == want) {
        *out = v[i].p;
        g_host_bytes -= want;
        v.erase(v.begin() + (long)i);
        return cudaSuccess;
      }
  }
  cudaError_t e = cudaHostAlloc(out, want, cudaHostAllocPortable);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    host_release();
    e = cudaHostAlloc(out, want, cudaHostAllocPortable);
  }
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
      host_blocks().push_back({p, size});
      g_host_bytes += size;
      return;
    }
  }
  cudaFreeHost(p);
}

}  // namespace gm
