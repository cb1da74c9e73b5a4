// Order-preserving compaction.  Three passes (per-block totals, a single-block
// scan of the totals, per-block write); results are deterministic and keep
// ascending index order.
#include "gm_common.cuh"
#include "gm_kernels.h"

#include <algorithm>
#include <atomic>

namespace gm {

namespace {
std::atomic<uint64_t> g_launches{0};
}  // namespace

void note_launch(int n) { g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed); }
uint64_t launch_counter() { return g_launches.load(std::memory_order_relaxed); }
void launch_counter_reset() { g_launches.store(0, std::memory_order_relaxed); }

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;
constexpr int kScanBlock = kScanThreads * kScanItems;  // 1024 items per block

// Inclusive scan of one int per thread across a 256-thread block.
__device__ __forceinline__ int block_inclusive_scan(int v, int *warp_tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  if (lane == 31) warp_tot[warp] = v;
  __syncthreads();
  if (warp == 0) {
    int w = (lane < kScanThreads / 32) ? warp_tot[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < kScanThreads / 32) warp_tot[lane] = w;
  }
  __syncthreads();
  if (warp > 0) v += warp_tot[warp - 1];
  __syncthreads();
  return v;
}

// Item i stays when its flag is not 0, or is `select` when that is >= 0.
struct Pred {
  const int *vals;
  int n, select;
  __device__ __forceinline__ int len() const { return n; }
  __device__ __forceinline__ int at(int i) const { return (select < 0 ? vals[i] != 0 : vals[i] == select) ? 1 : 0; }
};

// Item i stays when its value is at least *max_val / parts (none does when the
// maximum is not positive).
struct PredAtLeast {
  const float *vals, *max_val;
  const int *n_dev;
  int n_host, parts;
  __device__ __forceinline__ int len() const { return min(*n_dev, n_host); }
  __device__ __forceinline__ int at(int i) const {
    const float mw = *max_val;
    return mw > 0.0f && vals[i] >= __fdiv_rn(mw, (float)parts) ? 1 : 0;
  }
};

template <typename P>
__global__ void __launch_bounds__(kScanThreads) k_block_totals(P p, int *tot) {
  pdl_enter();
  __shared__ int wt[kScanThreads / 32];
  const int n = p.len();
  const int base = blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
  int s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i)
    if (base + i < n) s += p.at(base + i);
  s = block_inclusive_scan(s, wt);
  if (threadIdx.x == kScanThreads - 1) tot[blockIdx.x] = s;
}

// Exclusive scan of tot[0..nb) in place; tot[nb] = grand total.  One block.
__global__ void __launch_bounds__(kScanThreads) k_scan_totals(int *tot, int nb,
                                                              int *total_out) {
  pdl_enter();
  __shared__ int wt[kScanThreads / 32];
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int c0 = 0; c0 < nb; c0 += kScanBlock) {
    const int base = c0 + threadIdx.x * kScanItems;
    int v[kScanItems];
    int s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
      v[i] = (base + i < nb) ? tot[base + i] : 0;
      s += v[i];
    }
    const int incl = block_inclusive_scan(s, wt);
    int run = carry + incl - s;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
      if (base + i < nb) tot[base + i] = run;
      run += v[i];
    }
    __syncthreads();
    if (threadIdx.x == kScanThreads - 1) carry = run;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    tot[nb] = carry;
    if (total_out) *total_out = carry;
  }
}

template <typename P>
__global__ void __launch_bounds__(kScanThreads) k_block_write(P p, const int *tot, int *out,
                                                              int n_cap_out) {
  pdl_enter();
  __shared__ int wt[kScanThreads / 32];
  const int n = p.len();
  const int base = blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
  int v[kScanItems];
  int s = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    v[i] = (base + i < n) ? p.at(base + i) : 0;
    s += v[i];
  }
  const int incl = block_inclusive_scan(s, wt);
  int run = tot[blockIdx.x] + incl - s;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (v[i] && run < n_cap_out) out[run] = base + i;
    run += v[i];
  }
}

inline int nblocks(int n) { return n <= 0 ? 1 : (n + kScanBlock - 1) / kScanBlock; }

template <typename P>
void compact(const P &p, int n_max, int *out, int *count, int *tmp, cudaStream_t s) {
  const int nb = nblocks(n_max);
  launch(k_block_totals<P>, nb, kScanThreads, 0, s, p, tmp);
  note_launch();
  launch(k_scan_totals, 1, kScanThreads, 0, s, tmp, nb, count);
  note_launch();
  launch(k_block_write<P>, nb, kScanThreads, 0, s, p, tmp, out, n_max);
  note_launch();
}

}  // namespace

namespace {
__global__ void k_fill_u32(uint32_t *p, uint32_t v, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    p[i] = v;
}
__global__ void k_fill_u64(unsigned long long *p, unsigned long long v, size_t n) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    p[i] = v;
}
}  // namespace

// Rows from host memory into the feature matrix (row stride ld >= d; the
// padding keeps its zeros), read in place over the coherent link to the CPU:
// pageable memory too, where the GPU uses the host's page tables.  The copy
// into pinned staging that a transfer needs instead ran at 16 GB/s on one
// core and the staging had to be allocated for every session; 500 rows x 784
// (1.57 MB): 122 us with it, 18 us so; 10,000 x 128 (5.1 MB): 394 and 36 us.
namespace {
constexpr int kRowCopyThreads = 256;
__global__ void __launch_bounds__(kRowCopyThreads)
    k_copy_rows(const float *src, float *dst, int d, int ld, size_t total) {
  const size_t stride = (size_t)gridDim.x * kRowCopyThreads;
  const size_t first = (size_t)blockIdx.x * kRowCopyThreads + threadIdx.x;
  if (d == ld && ((uintptr_t)src & 15) == 0) {  // (ld is a multiple of 4)
    const float4 *s4 = reinterpret_cast<const float4 *>(src);
    float4 *d4 = reinterpret_cast<float4 *>(dst);
    for (size_t i = first; i < total / 4; i += stride) d4[i] = __ldcs(s4 + i);
    return;
  }
  for (size_t i = first; i < total; i += stride) {
    const size_t r = i / (size_t)d;
    dst[r * (size_t)ld + (i - r * (size_t)d)] = __ldcs(src + i);
  }
}
}  // namespace

void launch_copy_rows(const float *src, float *dst, size_t rows, int d, int ld, int sms, cudaStream_t s) {
  const size_t total = rows * (size_t)d;
  if (total == 0) return;
  const size_t blocks = std::min<size_t>((total + kRowCopyThreads * 4 - 1) / (kRowCopyThreads * 4),
                                         (size_t)std::max(sms, 1) * 4);
  k_copy_rows<<<(unsigned)blocks, kRowCopyThreads, 0, s>>>(src, dst, d, ld, total);
  note_launch();
}

void fill_u64(void *p, unsigned long long v, size_t n, cudaStream_t s) {
  if (n == 0) return;
  const size_t blocks = std::min<size_t>((n + 255) / 256, 4096);
  k_fill_u64<<<(unsigned)blocks, 256, 0, s>>>((unsigned long long *)p, v, n);
  note_launch();
}

void fill_u32(void *p, uint32_t v, size_t n, cudaStream_t s) {
  if (n == 0) return;
  const size_t blocks = std::min<size_t>((n + 255) / 256, 4096);
  k_fill_u32<<<(unsigned)blocks, 256, 0, s>>>((uint32_t *)p, v, n);
  note_launch();
}

size_t compact_tmp_ints(int n) { return (size_t)nblocks(n) + 2; }

void compact_flags(const int *flag, int n, int select, int *out, int *count,
                   int *tmp, cudaStream_t s) {
  compact(Pred{flag, n, select}, n, out, count, tmp, s);
}

void compact_at_least(const float *vals, const float *max_val, int parts, const int *n_dev, int n_max,
                      int *out, int *count, int *tmp, cudaStream_t s) {
  compact(PredAtLeast{vals, max_val, n_dev, n_max, parts}, n_max, out, count, tmp, s);
}

}  // namespace gm
