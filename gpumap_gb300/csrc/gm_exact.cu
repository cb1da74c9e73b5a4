// Exact insertion (precision = 1): each insertion batch is compared with
// every inserted row.  Distances are first formed on the 5th-generation tensor
// cores (split-BF16 operands staged by TMA, FP32 accumulators in TMEM), then
// every pair that a rigorous error bound cannot rule out is re-scored with the
// canonical FP32 distance.  Resulting lists are the exact 32 nearest rows
// under the canonical distance, identical to a brute-force CPU computation.
//
// Split BF16: each FP32 value x is stored as hi = bf16(x) and lo = bf16(x - hi)
// (x - hi is exact in FP32), and a.b is formed as hi.hi + hi.lo + lo.hi in one
// FP32 accumulator: three BF16 products per element, relative operand error
// about 3 * 2^-16 instead of 2^-7 for plain BF16.
//
//  k_to_bf16     batch rows -> [hi | lo] shadow rows (each zero padded to dh, a multiple of 64)
//  k_exact_dist  approx D[m][j] = |x_m|^2 + |x_j|^2 - 2 (x_m . x_j)_split
//                (tcgen05.mma kind::f16, M=128 x N=256 x K=16 per instruction),
//                screened as the accumulators are drained (the tile is not
//                stored): per batch row, the columns that may be among its
//                32 nearest; per existing row, the batch rows that may enter
//                its list
//  k_seed_select, k_pre_select  per batch row: its seed, then its exact
//                threshold and candidates from the stored columns
//  k_row_threshold  the same from the CTAs' heaps (after an overflow)
//  k_rescore     canonical FP32 re-score of the survivors
//  k_row_select / k_merge_offers   exact top-32 merges
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <atomic>
#include <mutex>

#include "gm_common.cuh"
#include "gm_kernels.h"
#include "gm_rowdot.cuh"

namespace gm {

namespace {

constexpr int kTM = 128;                       // batch rows per tile (MMA M)
constexpr int kTN = 256;                       // columns per tile (MMA N)
constexpr int kTK = 64;                        // bf16 per K chunk = one 128-byte swizzle row
// A stage holds one K chunk of all four operand halves (A hi | A lo | B hi |
// B lo) and feeds all three products of the split (12 MMAs of K = 16), so a
// byte in flight carries 1.5x the work of one product per stage and B's hi
// half is fetched once instead of twice.
constexpr int kStages = 2;
constexpr int kABytes = kTM * kTK * 2;         // 16 KB
constexpr int kBBytes = kTN * kTK * 2;         // 32 KB
constexpr int kStageBytes = 2 * kABytes + 2 * kBBytes; // 96 KB
// Warp 0 TMA, warp 1 MMA, then the epilogue: one warp group (four warps, one
// per 32-row quarter of the tile) per column share of the tile.  The heap
// pass keeps one group (its per-row heaps cannot be shared); the others run
// four, each on 64 of the tile's 256 columns, so that every scheduler has
// four epilogue warps to hide their latencies with.
__host__ __device__ constexpr int exact_groups(int pass) { return pass == 1 ? 1 : 4; }
__host__ __device__ constexpr int exact_threads(int pass) { return 64 + 128 * exact_groups(pass); }
constexpr int kTmemCols = 512;                 // two 128 x 256 FP32 accumulators
constexpr uint32_t kWaitLimit = 1u << 24;      // bounded mbarrier waits
// epilogue column buffer: the 256 columns' squared norms, bound factors and
// list bars of a tile, double buffered (two tiles), then per buffer sixteen
// per-warp maxima of the norms and bound factors (float bits: both >= 0)
constexpr size_t kEpiBytes = (size_t)2 * 3 * kTN * sizeof(float) + (size_t)2 * 2 * 16 * sizeof(float);
constexpr uint32_t kInfBits = 0x7f800000u;     // floats >= 0 below it are finite
constexpr int kListTop = 32;                   // list width the screen keeps exact
constexpr size_t kHeapBytes = (size_t)kListTop * kTM * sizeof(float);
constexpr size_t kExactSmem = (size_t)kStages * kStageBytes + 1024 + 256 + kEpiBytes + kHeapBytes;
static_assert(kExactSmem <= 232448, "k_exact_dist shared memory above the 227 KB per-CTA limit");

// Instruction descriptor, kind::f16: D=F32 (bits 4-5), A=B=BF16 (7-9, 10-12),
// both K-major (15, 16 = 0), N>>3 at 17-22, M>>4 at 24-28.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) |
                            ((uint32_t)(kTN >> 3) << 17) | ((uint32_t)(kTM >> 4) << 24);

GM_D uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

GM_D void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
GM_D void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
GM_D void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Waits (bounded) until the phase with the given parity has completed.
GM_D bool mbar_wait(uint64_t *bar, uint32_t parity) {
  const uint32_t a = smem_u32(bar);
  for (uint32_t it = 0; it < kWaitLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

GM_D void tma_load_2d(const CUtensorMap *map, uint64_t *bar, void *dst, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
      "l"((uint64_t)map), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}
// The same with an L2 cache policy (createpolicy) for the lines it reads: the
// column tiles stream through L2 once per row tile while other kernels of the
// session (the embedding's SGD) work out of L2, so their lines go first.
GM_D void tma_load_2d_hint(const CUtensorMap *map, uint64_t *bar, void *dst, int x, int y,
                           uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1, {%2, %3}], [%4], %5;" ::"r"(smem_u32(dst)),
      "l"((uint64_t)map), "r"(x), "r"(y), "r"(smem_u32(bar)), "l"(policy)
      : "memory");
}
// Shared-memory matrix descriptor: K-major operand, 128-byte swizzle,
// 8-row groups 1024 bytes apart (stride byte offset), descriptor version 1.
GM_D uint64_t sw128_desc(uint32_t addr) {
  uint64_t d = (uint64_t)((addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;            // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;  // stride byte offset
  d |= (uint64_t)1 << 46;            // version
  d |= (uint64_t)2 << 61;            // 128-byte swizzle
  return d;
}

GM_D void umma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(kIdesc), "r"(acc));
}
GM_D void umma_commit(uint64_t *bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}
GM_D void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
GM_D void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 consecutive columns of this thread's lane; the registers are valid after
// tmem_ld_wait (which names them, so that no read of them moves above it)
GM_D void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
GM_D void tmem_ld_wait(uint32_t (&r)[16]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]),
                 "+r"(r[6]), "+r"(r[7]), "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]),
                 "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
               :
               : "memory");
}

// Batch rows to split BF16 (both halves round to nearest): shadow row =
// hi[0..dh) | lo[0..dh), zero padded past d.
__global__ void k_to_bf16(const float *X, int ld, int d, int dh, int row0, int nrows,
                          __nv_bfloat16 *Xh) {
  pdl_enter();
  const long total = (long)nrows * dh;
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long)gridDim.x * blockDim.x) {
    const int r = (int)(i / dh), c = (int)(i - (long)r * dh);
    const size_t row = (size_t)(row0 + r);
    const float v = c < d ? X[row * ld + c] : 0.0f;
    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
    const __nv_bfloat16 lo = __float2bfloat16_rn(__fsub_rn(v, __bfloat162float(hi)));
    Xh[row * 2 * dh + c] = hi;
    Xh[row * 2 * dh + dh + c] = lo;
  }
}

// Rigorous bound on |approx - canonical| for one pair, as coef * sqrt(na nb)
// + 2^-21 (na + nb), with coef from exact_bound_coef.  Both distances share
// fl(na + nb); they differ by 2 |v - dot_c| plus the final subtraction's
// rounding (2^-24 of |s - 2v| and of |s - 2 dot_c|, each below 2 (na + nb)
// for any pair within the bound).  sa, sb: sqrt(na), sqrt(nb) rounded up, so
// sa * sb (rounded up) >= sqrt(na nb).
GM_D float pair_bound(float coef, float sa, float sb, float na, float nb) {
  return __fadd_ru(__fmul_ru(coef, __fmul_ru(sa, sb)),
                   __fadd_ru(__fmul_ru(4.8e-7f, __fadd_ru(na, nb)), 1e-30f));
}


// A tile's distance |a|^2 + |b|^2 - 2 a.b from the sum of the norms, rounded,
// and the accumulator (doubling it is exact, so one rounding remains).
GM_D float tile_dist(float na, float nb, float acc) {
  return __fmaf_rn(-2.0f, acc, __fadd_rn(na, nb));
}

// Max-heap of the 32 smallest upper bounds of one row, in shared memory with
// stride kTM (element i of row r at h[i * kTM]).  Pushes x (the caller has
// checked x < the current threshold) and returns the new threshold: the
// largest of the 32 once the heap is full, +inf before.
GM_D float heap_push(float *h, int &cnt, float x) {
  if (cnt < kListTop) {
    int pos = cnt++;
    while (pos > 0) {
      const int up = (pos - 1) >> 1;
      const float pv = h[up * kTM];
      if (pv >= x) break;
      h[pos * kTM] = pv;
      pos = up;
    }
    h[pos * kTM] = x;
    return cnt < kListTop ? __int_as_float(0x7f800000) : h[0];
  }
  int pos = 0;
  for (;;) {
    int c = 2 * pos + 1;
    if (c >= kListTop) break;
    if (c + 1 < kListTop && h[(c + 1) * kTM] > h[c * kTM]) ++c;
    const float cv = h[c * kTM];
    if (cv <= x) break;
    h[pos * kTM] = cv;
    pos = c;
  }
  h[pos * kTM] = x;
  return h[0];
}

// Screen state of one block of batch rows (batch-local row m).
struct TileScreen {
  int tile_count;     // column tiles this pass visits: tile t is column tile t * tile_stride
  int tile_stride;
  float *heaps;       // (m * gridDim.x + CTA) * 32: each CTA's 32 smallest upper bounds of row m
  const float *seed;  // passes 1 and 3: per-row upper bounds from pass 0 (or null)
  float *mins;        // pass 0: m * mins_ld + 8 * t + c: smallest upper bound of row m over
  int mins_ld;        //   the 32 columns of chunk c of sampled tile t
  const float *row_t; // exact per-row thresholds (pass 2)
  int *cand;          // m * cand_ld + i: candidate columns of row m (pass 2)
  long cand_ld;
  int *row_cnt;       // candidates per row (zeroed before pass 2)
  int *pool_j, *pool_m;  // (existing row, batch row) pairs that may enter j's list
  int *pool_counter;
  long pool_cap;
  const Key *g_key;   // working lists (the 32nd entry of an existing row is its bar)
  int n_exist;        // rows [0, n_exist) are the existing rows
  float coef;
  // pass 3: the stored columns of row m seen by CTA c, packed (lower bound
  // bits << 32 | column) with their upper bounds in pre_ub, in segment
  // (m * gridDim.x + c) of pre_cap entries; pre_cnt holds each segment's
  // length and pre_over is set when one would exceed pre_cap
  unsigned long long *pre;
  float *pre_ub;
  int *pre_cnt;
  int pre_cap;
  int *pre_over;
  int col_test;       // pass 1: run the column test (off when pass 3 already did)
  const int *run_if;  // when set, the launch does nothing unless *run_if != 0
};

// Distances of a block of batch rows against all columns, screened as they
// leave the tensor memory (the tile itself is not stored).  grid.y: 128-row
// tiles of the batch; grid.x: CTAs sharing the column tiles.  For every pair
// (batch row m, column j) the epilogue forms D and the bound B (pair_bound);
// its upper bound is D + B and its lower bound D - B.
//  Pass 0 (kPass == 0), on an evenly spaced sample of column tiles: per row
//    and 32-column chunk, the smallest upper bound (sc.mins).  The 32nd
//    smallest of a row's chunk minima (k_seed_select) is the largest upper
//    bound of 32 distinct columns, so it bounds the row's 32nd smallest
//    upper bound over all columns from above: the seed.
//  Pass 3 (kPass == 3), all column tiles: every column whose lower bound is
//    at most the seed is stored with its bounds.  Every column whose upper
//    bound is at most the row's exact threshold T (its 32nd smallest upper
//    bound) is among them, so k_pre_select finds T exactly from the stored
//    upper bounds, then keeps the stored columns with lower bound <= T.
//    Column side, for an existing row j: (j, m) goes to the pair pool when
//    D - B is at most the 32nd distance of j's list.
// Up to four column tiles there is no pass 0 and the seed is infinite.  For a
// block whose stored columns overflowed, or have no room:
//  Pass 1 (kPass == 1), all column tiles: every CTA keeps, per row, a
//    max-heap of the 32 smallest upper bounds it sees (at or below the seed
//    when there is one) and stores it to sc.heaps; the 32nd smallest of
//    their union (k_row_threshold) is T, or the seed when smaller.  The
//    column test as in pass 3 (sc.col_test; off after a pass 3).
//  Pass 2 (kPass == 2): the same tiles again; j becomes a candidate of row m
//    when D - B <= T.
// Either way the candidates hold every column whose canonical distance can
// be among m's 32 smallest.  With kKeepD the tile is also written to D (ldD
// columns per row), for tests.
template <int kPass, bool kKeepD>
__global__ void __launch_bounds__(exact_threads(kPass), 1)
    k_exact_dist(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                 int arow0, int nb, int n, int kchunks, int dh, const float *norms,
                 const float *snorms, TileScreen sc, float *D, long ldD, unsigned *err) {
  pdl_enter();
  // a gated launch (the fallback after a pass 3 whose stored columns did
  // not overflow) does nothing: the flag is read before any barrier or
  // tensor memory is set up, by every thread alike
  if (sc.run_if && *sc.run_if == 0) return;
  extern __shared__ __align__(1024) unsigned char raw[];
  unsigned char *base = (unsigned char *)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
  uint64_t *full = (uint64_t *)(base + (size_t)kStages * kStageBytes);
  uint64_t *empty = full + kStages;
  uint64_t *tmem_full = empty + kStages;  // [2]: accumulator b holds a finished tile
  uint64_t *tmem_empty = tmem_full + 2;   // [2]: accumulator b has been drained
  uint32_t *tmem_slot = (uint32_t *)(tmem_empty + 2);
  float *epi = (float *)(base + (size_t)kStages * kStageBytes + 256);
  float *heaps = (float *)((unsigned char *)epi + kEpiBytes);

  constexpr int kGroups = exact_groups(kPass);
  constexpr int kEpi = 128 * kGroups;    // epilogue threads
  constexpr int kGroupCols = kTN / kGroups;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mt = blockIdx.y;
  const int m0 = mt * kTM;  // batch-local first row of this tile

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], kEpi);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  bool ok = true;

  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;
      uint64_t pol;
      asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
      for (int t = blockIdx.x; t < sc.tile_count && ok; t += gridDim.x) {
        const int ct = t * sc.tile_stride;
        // kchunks K chunks, each with the hi and lo halves of both operands
        // (x offsets are multiples of 64; lo halves start at x = dh)
        for (int kc = 0; kc < kchunks; ++kc, ++it) {
          const uint32_t s = it % kStages, use = it / kStages;
          if (use > 0 && !mbar_wait(&empty[s], (use - 1) & 1)) {
            ok = false;
            break;
          }
          const int kx = kc * kTK;
          unsigned char *a = base + (size_t)s * kStageBytes;
          mbar_expect_tx(&full[s], kStageBytes);
          tma_load_2d(&tm_a, &full[s], a, kx, arow0 + m0);
          tma_load_2d(&tm_a, &full[s], a + kABytes, dh + kx, arow0 + m0);
          tma_load_2d_hint(&tm_b, &full[s], a + 2 * kABytes, kx, ct * kTN, pol);
          tma_load_2d_hint(&tm_b, &full[s], a + 2 * kABytes + kBBytes, dh + kx, ct * kTN, pol);
        }
      }
      if (!ok) atomicOr(err, kDevErrSpin);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // tile tc accumulates in TMEM columns [256 (tc & 1), +256): the MMAs of
      // the next tile run while the epilogue drains this one
      uint32_t it = 0, tc = 0;
      for (int t = blockIdx.x; t < sc.tile_count && ok; t += gridDim.x, ++tc) {
        const uint32_t b = tc & 1u, use = tc >> 1;
        if (use > 0 && !mbar_wait(&tmem_empty[b], (use - 1) & 1)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t acc = tmem + b * (uint32_t)kTN;
        for (int kc = 0; kc < kchunks; ++kc, ++it) {
          const uint32_t s = it % kStages, u2 = it / kStages;
          if (!mbar_wait(&full[s], u2 & 1)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t ahi = smem_u32(base + (size_t)s * kStageBytes);
          const uint32_t alo = ahi + kABytes, bhi = ahi + 2 * kABytes, blo = bhi + kBBytes;
          // a.b = hi.hi + hi.lo + lo.hi, K = 16 at a time
#pragma unroll
          for (int k = 0; k < kTK / 16; ++k) {
            umma_bf16(acc, sw128_desc(ahi + k * 32), sw128_desc(bhi + k * 32), (kc | k) != 0 ? 1u : 0u);
            umma_bf16(acc, sw128_desc(ahi + k * 32), sw128_desc(blo + k * 32), 1u);
            umma_bf16(acc, sw128_desc(alo + k * 32), sw128_desc(bhi + k * 32), 1u);
          }
          umma_commit(&empty[s]);
        }
        if (!ok) break;
        umma_commit(&tmem_full[b]);
      }
      if (!ok) atomicOr(err, kDevErrSpin);
    }
    __syncwarp();
  } else {
    // epilogue: warp w reads TMEM lanes 32*(w%4) .. +31 (tile rows), one row
    // per thread, 16 columns per tcgen05.ld; warp group g = (w - 2) / 4
    // takes columns [g * kGroupCols, +kGroupCols) of each tile.  Each group
    // loads its columns' data (squared norms, bound factors, list bars) one
    // tile ahead into a double-buffered shared array that its lanes read by
    // broadcast; each tile begins with a barrier of the group's 128 threads
    // (named barrier 1 + g), executed the same number of times by each of
    // them, so that groups run on without waiting for one another.  Named
    // barrier 5 spans the whole epilogue (before the first tile and, in pass
    // 3, after the last).
    const int quarter = warp & 3;
    const int group = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;
    const int m = m0 + r;
    const bool live = m < nb;
    const int row = arow0 + m;
    const int gt = threadIdx.x - 64 - 128 * group;  // 0..127 within the group
    const float inf = __int_as_float(0x7f800000);
    // rows past the block's last have an infinite norm and no limit: no
    // column passes their tests (with a limit of +inf every column did, and
    // a warp with such a row took all of them through the exact tests)
    const float nm = live ? norms[row] : inf;
    const float sm = live ? snorms[row] : 0.0f;
    float *heap = heaps + r;
    int hcnt = 0;
    float t_loc = inf;  // passes 0 and 1: the heap's largest once it holds 32
    const float t_row = (kPass == 2 && live) ? sc.row_t[m] : -inf;
    const float seed = (kPass == 1 || kPass == 3) ? (!live ? -inf : sc.seed ? sc.seed[m] : inf) : -inf;
    int *cand_m = sc.cand + (long)m * sc.cand_ld;
    // pass 3: the segment of stored columns of (row m, this CTA), filled by
    // the row's threads of every group through a shared-memory counter
    // (in the heap space, which pass 3 does not use)
    const size_t seg = ((size_t)m * gridDim.x + blockIdx.x) * (size_t)sc.pre_cap;
    int *scnt = reinterpret_cast<int *>(heaps);
    if (kPass == 3 && group == 0) scnt[r] = 0;
    asm volatile("bar.sync 5, %0;" ::"n"(kEpi) : "memory");
    const bool col_test = kPass == 3 || (kPass == 1 && sc.col_test);
    // this thread's columns of a tile: group * kGroupCols + gt + 128 h
    constexpr int kColsPer = (kGroupCols + 127) / 128;
    float cv[3 * kColsPer];
    auto load_cols = [&](int t) {
      const int c0 = t * sc.tile_stride * kTN;
#pragma unroll
      for (int h = 0; h < kColsPer; ++h) {
        const int gi = gt + h * 128;
        const int jj = group * kGroupCols + gi;
        const int j = c0 + jj;
        const bool in = gi < kGroupCols && j < n;
        cv[3 * h] = in ? norms[j] : 0.0f;
        cv[3 * h + 1] = in ? snorms[j] : 0.0f;
        cv[3 * h + 2] = ((kPass == 1 || kPass == 3) && gi < kGroupCols && j < sc.n_exist)
                            ? key_dist(sc.g_key[(size_t)j * kListW + kListW - 1])
                            : -inf;
      }
    };
    if ((int)blockIdx.x < sc.tile_count) load_cols(blockIdx.x);
    bool eok = true;
    uint32_t tc = 0;
    for (int t = blockIdx.x; t < sc.tile_count; t += gridDim.x, ++tc) {
      const uint32_t b = tc & 1u;
      float *cn = epi + (size_t)b * 3 * kTN;  // norms | bound factors | list bars
      // per-warp maxima of the column norms and factors: slot 4 g + q for
      // warp q of group g (0 where the warp has no columns)
      unsigned *mx = reinterpret_cast<unsigned *>(epi + 2 * 3 * kTN) + b * 2 * 16;
      {
        unsigned mn = 0, ms = 0;
#pragma unroll
        for (int h = 0; h < kColsPer; ++h) {
          const int gi = gt + h * 128;
          if (gi < kGroupCols) {
            const int jj = group * kGroupCols + gi;
            cn[jj] = cv[3 * h];
            cn[kTN + jj] = cv[3 * h + 1];
            cn[2 * kTN + jj] = cv[3 * h + 2];
            // a column whose norm is infinite or NaN (its row has such a
            // feature, or overflows) passes no test: D - B is NaN for every
            // row.  Its norm would make the filter's slack NaN for the whole
            // group
            const unsigned un = __float_as_uint(cv[3 * h]), us = __float_as_uint(cv[3 * h + 1]);
            mn = max(mn, un < kInfBits ? un : 0u);
            ms = max(ms, us < kInfBits ? us : 0u);
          }
        }
        mn = __reduce_max_sync(0xffffffffu, mn);
        ms = __reduce_max_sync(0xffffffffu, ms);
        if (lane == 0) {
          mx[4 * group + quarter] = mn;
          mx[16 + 4 * group + quarter] = ms;
        }
      }
      switch (group) {  // the barrier id is an immediate
        case 0: asm volatile("bar.sync 1, 128;" ::: "memory"); break;
        case 1: asm volatile("bar.sync 2, 128;" ::: "memory"); break;
        case 2: asm volatile("bar.sync 3, 128;" ::: "memory"); break;
        default: asm volatile("bar.sync 4, 128;" ::: "memory"); break;
      }
      // the largest pair bound of the row over this group's finite columns
      // (pair_bound is nondecreasing in the column's norm and factor)
      float bmax, nmax;
      {
        unsigned mn = 0, ms = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          mn = max(mn, mx[4 * group + q]);
          ms = max(ms, mx[16 + 4 * group + q]);
        }
        nmax = __uint_as_float(mn);
        bmax = pair_bound(sc.coef, sm, __uint_as_float(ms), nm, nmax);
      }
      if (t + (int)gridDim.x < sc.tile_count) load_cols(t + gridDim.x);
      if (eok && !mbar_wait(&tmem_full[b], (tc >> 1) & 1)) {
        if (lane == 0) atomicOr(err, kDevErrSpin);
        eok = false;
      }
      if (!eok) continue;
      tc_fence_after();
      const int ctile = t * sc.tile_stride * kTN;
      // passes 2 and 3: a column needs no exact test unless its nj - 2 a is
      // at most L + slack, L the larger of the row's limit and the
      // column's list bar, both 0 or more, or -inf.  With M = nm + nmax and
      // u = 2^-24, |2 a| below 1.1 M: for L > 4 M it always is.  For L below
      // that, a test that passes has RD(D - B) <= L, hence D <= L + bmax +
      // 8 u M, and D = fl(fl(nm + nj) - 2 a) is at least nm + nj - 2 a -
      // 3.1 u M; the slack adds 1e-6 M = 16.8 u M to bmax - nm, and the two
      // per-column roundings are directed to the safe side.
      const float lim = kPass == 3 ? seed : t_row;
      const float slack = __fadd_ru(__fsub_ru(bmax, nm), __fmul_ru(1e-6f, __fadd_ru(nm, nmax)));
      float cmin = inf;    // pass 0: the 32-column chunk's smallest D over other columns
      unsigned hmask = 0;  // column test: the chunk's hit columns (bit i)
      // the exact tests of column c + i of the tile (chunk bit (c & 16) + i),
      // whose D is dv
      auto slow = [&](int i, float dv, int c) {
        const float nj = cn[c + i];
        const int j = ctile + c + i;
        const bool other = live && j < n && j != row;
        const float wj = (kPass == 1 || kPass == 3) ? cn[2 * kTN + c + i] : -inf;
        const float sj = cn[kTN + c + i];
        const float bnd = pair_bound(sc.coef, sm, sj, nm, nj);
        if (kPass == 1 && other) {
          // (the clamp keeps a NaN, which fails the test; fmaxf would make it 0)
          const float sum = __fadd_ru(dv, bnd), ub = sum <= 0.0f ? 0.0f : sum;
          if (ub < t_loc && ub <= seed) t_loc = heap_push(heap, hcnt, ub);
        }
        if (kPass == 3 && other) {
          const float lb = __fsub_rd(dv, bnd);
          if (lb <= seed) {
            const int q = atomicAdd(&scnt[r], 1);
            if (q < sc.pre_cap) {
              sc.pre[seg + q] = ((unsigned long long)__float_as_uint(lb) << 32) | (unsigned)j;
              sc.pre_ub[seg + q] = fmaxf(__fadd_ru(dv, bnd), 0.0f);
            }
          }
        }
        if (col_test) {
          if (live && j < sc.n_exist && __fsub_rd(dv, bnd) <= wj) hmask |= 1u << ((c & 16) + i);
        } else if (kPass == 2 && other && __fsub_rd(dv, bnd) <= t_row) {
          cand_m[atomicAdd(&sc.row_cnt[m], 1)] = j;
        }
      };
      // 16 columns from c (a half of a 32-column chunk), their accumulators
      // in v
      auto half = [&](uint32_t(&v)[16], int c) {
        const int col0 = ctile + c;
        // fast phase: D of the 16 columns or, for passes 2 and 3, a mask of
        // the columns where this row may pass a test; 16 independent chains
        // without branches
        unsigned may = 0u;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          const float acc = __uint_as_float(v[i]);
          if (kPass == 2 || kPass == 3) {
            const float wj = kPass == 3 ? cn[2 * kTN + c + i] : -inf;
            const float part = __fmaf_rd(-2.0f, acc, cn[c + i]);
            if (part <= __fadd_ru(fmaxf(lim, wj), slack)) may |= 1u << i;
          }
          if (kPass < 2 || kKeepD) {
            const float dv = tile_dist(nm, cn[c + i], acc);
            if (kPass == 1) v[i] = __float_as_uint(dv);
            if (kKeepD && live && col0 + i < n) D[(long)m * ldD + col0 + i] = dv;
            if (kPass == 0 && live && col0 + i < n && col0 + i != row) cmin = fminf(cmin, dv);
          }
        }
        // slow phase: every column for the heap pass, in order; for passes 2
        // and 3 each lane its own flagged columns, the lanes' side by side
        // (about one pair in 250 is flagged, so 16 columns of 32 rows have two
        // or three, rarely two in one row; a column of the warp at a time
        // they were two thirds of the kernel's instructions)
        if constexpr (kPass == 1) {
#pragma unroll
          for (int i = 0; i < 16; ++i) slow(i, __uint_as_float(v[i]), c);
        } else if constexpr (kPass == 2 || kPass == 3) {
          while (may) {
            const int i = __ffs(may) - 1;
            may &= may - 1;
            // v[i]
            unsigned w8[8], w4[4];
#pragma unroll
            for (int q = 0; q < 8; ++q) w8[q] = (i & 1) ? v[2 * q + 1] : v[2 * q];
#pragma unroll
            for (int q = 0; q < 4; ++q) w4[q] = (i & 2) ? w8[2 * q + 1] : w8[2 * q];
            const unsigned w = (i & 8) ? ((i & 4) ? w4[3] : w4[2]) : ((i & 4) ? w4[1] : w4[0]);
            slow(i, tile_dist(nm, cn[c + i], __uint_as_float(w)), c);
          }
          __syncwarp();
        }
      };
      // after both halves of the 32-column chunk at c
      auto chunk_end = [&](int c) {
        const int col0 = ctile + c;
        if (kPass == 0 && live)
          sc.mins[(size_t)m * sc.mins_ld + t * (kTN / 32) + c / 32] =
              cmin == inf ? inf : fmaxf(__fadd_ru(cmin, bmax), 0.0f);
        cmin = inf;
        if (col_test) {
          // the chunk's (existing row j, batch row m) pairs: one pool
          // reservation per warp, lanes in order
          const int cnt = __popc(hmask);
          int incl = cnt;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
          }
          const int total = __shfl_sync(0xffffffffu, incl, 31);
          if (total) {
            int base = 0;
            if (lane == 31) base = atomicAdd(sc.pool_counter, total);
            base = __shfl_sync(0xffffffffu, base, 31);
            long q = (long)base + incl - cnt;
            while (hmask) {
              const int i = __ffs(hmask) - 1;
              hmask &= hmask - 1;
              if (q < sc.pool_cap) {
                sc.pool_j[q] = col0 + i;
                sc.pool_m[q] = m;
              } else {
                atomicOr(err, kDevErrOverflow);
              }
              ++q;
            }
          }
          hmask = 0;
        }
      };
      // the group's columns 16 at a time, the next half's tensor-memory load
      // in flight while this half is screened
      constexpr int kHalves = kGroupCols / 16;
      const uint32_t ta = tmem + ((uint32_t)(quarter * 32) << 16) + b * (uint32_t)kTN +
                          (uint32_t)(group * kGroupCols);
      uint32_t va[16], vb[16];
      tmem_ld16(ta, va);
#pragma unroll 1
      for (int h = 0; h < kHalves; h += 2) {
        tmem_ld_wait(va);
        tmem_ld16(ta + (uint32_t)(h + 1) * 16, vb);
        half(va, group * kGroupCols + h * 16);
        tmem_ld_wait(vb);
        if (h + 2 < kHalves) tmem_ld16(ta + (uint32_t)(h + 2) * 16, va);
        half(vb, group * kGroupCols + (h + 1) * 16);
        chunk_end(group * kGroupCols + h * 16);
      }
      tc_fence_before();
      mbar_arrive(&tmem_empty[b]);
    }
    if (kPass == 1 && live) {
      float *out = sc.heaps + ((size_t)m * gridDim.x + blockIdx.x) * kListTop;
      for (int i = 0; i < kListTop; ++i) out[i] = i < hcnt ? heap[i * kTM] : inf;
    }
    if (kPass == 3) {
      // every group's stores to the row's counter are done
      asm volatile("bar.sync 5, %0;" ::"n"(kEpi) : "memory");
      if (group == 0 && live) {
        const int pcnt = scnt[r];
        sc.pre_cnt[(size_t)m * gridDim.x + blockIdx.x] = min(pcnt, sc.pre_cap);
        if (pcnt > sc.pre_cap) atomicOr(sc.pre_over, 1);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols));
  }
}

// ---- screen: exact threshold, FP32 re-score, exact top-32 -----------------
//
// Around and after k_exact_dist, per block of batch rows (brow0 .. +nrows):
//  k_row_threshold  warp per batch row: T = 32nd smallest upper bound over all
//                columns, from the union of the CTAs' heaps (pass 1), for the
//                candidate test of pass 2
//  k_pool_count / k_pool_place   groups the column pairs by batch row
//                (counting sort; order inside a group is free)
//  k_rescore     canonical distances of the row candidates and of the column
//                pairs, whose offers go on the existing rows' chains
//  k_row_select  warp per batch row: exact top-32 keys of its candidates
//  k_merge_offers (gm_kernels_insert.cu)  warp per existing row: merges its
//                chains into its list
// Both merges are order independent: a list ends as the 32 smallest keys of
// its old entries and every candidate, and keys are unique (distinct ids).
//
// fmaf(a, b, c) = fmaf(b, a, c) exactly, so d(x, y) = d(y, x) bit for bit.

constexpr int kFinalWarps = 4;

// Merges each lane's value u into the warp's ascending top 32 (lane l holds
// the l-th smallest); values not below the current 32nd change nothing.
GM_D void top32_merge(float &top, float u, int lane) {
  unsigned pend = __ballot_sync(0xffffffffu, u < __shfl_sync(0xffffffffu, top, 31));
  while (pend) {
    const int src = __ffs(pend) - 1;
    pend &= pend - 1;
    const float x = __shfl_sync(0xffffffffu, u, src);
    const unsigned pos_mask = __ballot_sync(0xffffffffu, x < top);
    if (!pos_mask) continue;
    const int pos = __ffs(pos_mask) - 1;
    const float prev = __shfl_up_sync(0xffffffffu, top, 1);
    if (lane > pos) top = prev;
    else if (lane == pos) top = x;
  }
}

// The 32nd smallest of values >= 0 (inf included), by a search over its bits:
// the smallest x that `count` (the warp's number of values <= x) puts at 32 or
// more; inf when there are fewer.
template <typename F>
GM_D float bits_32nd(F &&count) {
  unsigned x = 0;
#pragma unroll 1
  for (int b = 30; b >= 0; --b)
    if (count(__uint_as_float(x | ((1u << b) - 1u))) < kListTop) x |= 1u << b;
  return __uint_as_float(min(x, 0x7f800000u));
}

// The 32nd smallest of cnt values >= 0 at v (inf when there are fewer), one
// warp.  Up to 512 are held in registers and searched by bits (31 counts);
// inserting them one at a time took 10 us a launch for 128 values, this 3 us.
// Past that, eight 32-value chunks are loaded together, then inserted.
GM_D float warp_32nd(const float *v, int cnt, int lane) {
  const float inf = __int_as_float(0x7f800000);
  constexpr int kHeld = 16;
  if (cnt <= kHeld * 32) {
    float u[kHeld];
#pragma unroll
    for (int q = 0; q < kHeld; ++q) u[q] = q * 32 + lane < cnt ? v[q * 32 + lane] : inf;
    const int used = (cnt + 31) / 32;
    return bits_32nd([&](float x) {
      int c = 0;
#pragma unroll
      for (int q = 0; q < kHeld; ++q)
        if (q < used) c += u[q] <= x;
      return (int)__reduce_add_sync(0xffffffffu, (unsigned)c);
    });
  }
  float top = inf;
  for (int c0 = 0; c0 < cnt; c0 += 8 * 32) {
    float u[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int idx = c0 + q * 32 + lane;
      u[q] = idx < cnt ? v[idx] : inf;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) top32_merge(top, u[q], lane);
  }
  return __shfl_sync(0xffffffffu, top, 31);
}

// The 32nd smallest of cnt values >= 0 (inf included), value i at get(i), by a
// whole CTA: inf when there are fewer.  The values' bits are counted in up to
// 256 equal bins of their range, then of the bin that holds the 32nd, and so
// on until it is alone in its bin: at most four rounds of two barriers, where
// a search by bits takes 31 rounds and compares every value in each.  Every
// thread returns it.
struct Select32 {
  int4 bins[2][64];
  unsigned lo, hi;
};
template <int kThreads, typename F>
GM_D float cta_32nd(int cnt, F &&get, Select32 &sh) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  if (cnt < kListTop) return __int_as_float(0x7f800000);  // (the same for every thread)
  unsigned lo = full, hi = 0u;
  for (int i = threadIdx.x; i < cnt; i += kThreads) {
    const unsigned v = __float_as_uint(get(i));
    lo = min(lo, v);
    hi = max(hi, v);
  }
  if (threadIdx.x == 0) {
    sh.lo = full;
    sh.hi = 0u;
  }
  if (threadIdx.x < 64) sh.bins[0][threadIdx.x] = make_int4(0, 0, 0, 0);
  __syncthreads();
  lo = __reduce_min_sync(full, lo);
  hi = __reduce_max_sync(full, hi);
  if (lane == 0) {
    atomicMin(&sh.lo, lo);
    atomicMax(&sh.hi, hi);
  }
  __syncthreads();
  lo = sh.lo;
  hi = sh.hi;
  int want = kListTop;  // the rank of the value among those in [lo, hi]
  for (int buf = 0; lo < hi; buf ^= 1) {
    const int shift = max(0, 24 - __clz((int)(hi - lo)));  // (hi - lo) >> shift < 256
    for (int i = threadIdx.x; i < cnt; i += kThreads) {
      const unsigned v = __float_as_uint(get(i));
      if (v >= lo && v <= hi) atomicAdd(reinterpret_cast<int *>(sh.bins[buf]) + ((v - lo) >> shift), 1);
    }
    if (threadIdx.x < 64) sh.bins[buf ^ 1][threadIdx.x] = make_int4(0, 0, 0, 0);
    __syncthreads();
    // each warp finds the bin: eight of them a lane
    const int4 b0 = sh.bins[buf][lane * 2], b1 = sh.bins[buf][lane * 2 + 1];
    const int c[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
    const int sum = ((b0.x + b0.y) + (b0.z + b0.w)) + ((b1.x + b1.y) + (b1.z + b1.w));
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(full, incl, o);
      if (lane >= o) incl += y;
    }
    const int src = __ffs(__ballot_sync(full, incl >= want)) - 1;
    int rank = want - (incl - sum), bin = 0, in_bin = c[0];
#pragma unroll
    for (int q = 0; q < 7; ++q)
      if (bin == q && rank > c[q]) {
        rank -= c[q];
        ++bin;
        in_bin = c[q + 1];
      }
    want = __shfl_sync(full, rank, src);
    in_bin = __shfl_sync(full, in_bin, src);
    lo += (unsigned)__shfl_sync(full, lane * 8 + bin, src) << shift;
    hi = min(hi, lo + ((1u << shift) - 1u));
    if (in_bin == 1) {  // (the same for every thread)
      for (int i = threadIdx.x; i < cnt; i += kThreads) {
        const unsigned v = __float_as_uint(get(i));
        if (v >= lo && v <= hi) sh.lo = v;
      }
      __syncthreads();
      return __uint_as_float(sh.lo);
    }
    __syncthreads();
  }
  return __uint_as_float(lo);
}

// Warp per batch row: T = the 32nd smallest of the union of the CTAs' heaps
// (pass 1), capped by the seed; both bound the row's 32nd smallest upper
// bound from above.  With run_if, only when *run_if != 0.
__global__ void __launch_bounds__(kFinalWarps * 32)
    k_row_threshold(const float *heaps, int ncta, int nrows, int n, const float *seed, float *row_t,
                    const int *run_if, unsigned long long *stat) {
  pdl_enter();
  if (run_if && *run_if == 0) return;
  const int lane = threadIdx.x & 31;
  const int ml = blockIdx.x * kFinalWarps + (threadIdx.x >> 5);
  if (ml >= nrows) return;
  const float inf = __int_as_float(0x7f800000);
  const float T = fminf(warp_32nd(heaps + (size_t)ml * ncta * kListTop, ncta * kListTop, lane),
                        seed ? seed[ml] : inf);
  if (lane == 0) {
    // fewer than 32 other rows: every column is a candidate
    row_t[ml] = n - 1 < kListTop ? inf : T;
    if (stat) atomicAdd(&stat[5], (unsigned long long)n);
  }
}

// CTA per batch row: the seed, the 32nd smallest of the row's chunk minima
// from pass 0 (the largest upper bound of 32 distinct columns).  Clears the
// counters of the passes after it.  1,000 rows of 600 minima: 25 us by a warp
// per row (insertion above 512 values), 8.0 us.
constexpr int kSeedThreads = 128, kSeedStage = 4096;
__global__ void __launch_bounds__(kSeedThreads)
    k_seed_select(const float *mins, int mins_ld, float *seed, int *row_cnt, int *pcnt, int *counter,
                  int *pre_over) {
  pdl_enter();
  extern __shared__ float s_min[];
  __shared__ Select32 sh;
  const int m = blockIdx.x;
  const float *v = mins + (size_t)m * mins_ld;
  const int staged = min(mins_ld, kSeedStage);
  for (int i = threadIdx.x; i < staged; i += kSeedThreads) s_min[i] = v[i];
  // (each thread reads back what it wrote)
  const float T = cta_32nd<kSeedThreads>(mins_ld, [&](int i) { return i < kSeedStage ? s_min[i] : v[i]; }, sh);
  if (threadIdx.x == 0) {
    seed[m] = T;
    row_cnt[m] = pcnt[m] = 0;
    if (m == 0) *counter = *pre_over = 0;
  }
}

// CTA per batch row, after pass 3: T = the 32nd smallest stored upper
// bound (exact: every column whose upper bound is at most T was stored),
// then the row's candidates, the stored columns with lower bound <= T.  Does
// nothing when a segment overflowed (the heap passes then run instead).
// The entries (about 0.4 % of the columns: the seed is a 32 / 8192 quantile)
// are gathered from the row's segments into shared memory, each by its own
// thread (a warp per segment waited for one segment after another).
// A warp per row that inserted the bounds one at a time was bound by latency: 33
// us for 500 rows of ~600 entries, a CTA that searched them by bits 24 us in a
// run (31 rounds over all values, bound by issue), this form 11 us.  A row with
// more than kPreStage entries (data far from the origin, whose bounds are wide) is
// worked through where they lie, by the same search: by one warp a bit at a time
// 9,600 such rows x 8 in cycles of 300 took 38.2 ms (31.8 with the insertion before
// that), 24.7 so.
constexpr int kPreThreads = 128;
constexpr int kPreStage = 2048, kPreSegs = 512;
__global__ void __launch_bounds__(kPreThreads)
    k_pre_select(const unsigned long long *pre, const float *pre_ub, const int *pre_cnt, int gx,
                 int cap, const int *pre_over, int n, float *row_t, int *cand, long cand_ld,
                 int *row_cnt, unsigned long long *stat) {
  pdl_enter();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, m = blockIdx.x;
  if (*pre_over) {
    if (stat && m == 0 && threadIdx.x == 0) atomicAdd(&stat[9], 1ull);
    return;
  }
  __shared__ float s_ub[kPreStage];
  __shared__ unsigned long long s_ent[kPreStage];
  __shared__ int s_off[kPreSegs + 1], s_kept;
  __shared__ Select32 sel;
  const unsigned full = 0xffffffffu;
  const int *cnts = pre_cnt + (size_t)m * gx;
  const size_t seg0 = (size_t)m * gx * (size_t)cap;
  if (warp == 0) {
    int run = 0;
    for (int c0 = 0; c0 < gx; c0 += 32) {
      const int v = c0 + lane < gx ? cnts[c0 + lane] : 0;
      int incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += y;
      }
      if (c0 + lane < gx) s_off[c0 + lane] = run + incl - v;
      run += __shfl_sync(full, incl, 31);
    }
    if (lane == 0) {
      s_off[kPreSegs] = run;
      s_kept = 0;
    }
  }
  __syncthreads();
  const int total = s_off[kPreSegs];
  int *out = cand + (long)m * cand_ld;
  auto keep = [&](bool in, unsigned long long e, float T) {
    const bool ok = in && __uint_as_float((unsigned)(e >> 32)) <= T;
    const unsigned bal = __ballot_sync(full, ok);
    int base = 0;
    if (lane == 0 && bal) base = atomicAdd(&s_kept, __popc(bal));
    base = __shfl_sync(full, base, 0);
    if (ok) out[base + __popc(bal & ((1u << lane) - 1u))] = (int)(unsigned)e;
  };
  // entry i is in the last segment that begins at or before it
  auto place = [&](int i) {
    int c = 0;
    for (int step = kPreSegs / 2; step > 0; step >>= 1)
      if (c + step < gx && s_off[c + step] <= i) c += step;
    return seg0 + (size_t)c * cap + (i - s_off[c]);
  };
  auto select = [&](auto &&ub, auto &&entry) {
    // fewer than 32 other rows: every column is a candidate
    float T = cta_32nd<kPreThreads>(total, ub, sel);
    if (n - 1 < kListTop) T = __int_as_float(0x7f800000);
    for (int i = warp * 32; i < total; i += kPreThreads)
      keep(i + lane < total, i + lane < total ? entry(i + lane) : 0ull, T);
    return T;
  };
  float T;
  if (total <= kPreStage) {
#pragma unroll 4
    for (int i = threadIdx.x; i < total; i += kPreThreads) {
      const size_t from = place(i);
      s_ub[i] = pre_ub[from];
      s_ent[i] = pre[from];
    }
    __syncthreads();
    T = select([&](int i) { return s_ub[i]; }, [&](int i) { return s_ent[i]; });
  } else {
    T = select([&](int i) { return pre_ub[place(i)]; }, [&](int i) { return pre[place(i)]; });
    if (stat && threadIdx.x == 0) atomicAdd(&stat[10], 1ull);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    row_t[m] = T;
    row_cnt[m] = s_kept;
    if (stat) atomicAdd(&stat[5], (unsigned long long)n);
  }
}

// Pairs per batch row (at most 1,024 rows a block, counted in shared memory
// first), then, in one CTA, the groups' offsets and fill cursors.
constexpr int kMaxBlockRows = 1024;
__global__ void __launch_bounds__(256)
    k_pool_count(const int *pool_m, const int *counter, long pool_cap, int nrows, int *cnt,
                 unsigned long long *stat) {
  pdl_enter();
  __shared__ int s_cnt[kMaxBlockRows];
  const long total = min((long)*counter, pool_cap);
  for (int i = threadIdx.x; i < nrows; i += blockDim.x) s_cnt[i] = 0;
  __syncthreads();
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x)
    atomicAdd(&s_cnt[pool_m[e]], 1);
  __syncthreads();
  for (int i = threadIdx.x; i < nrows; i += blockDim.x)
    if (s_cnt[i]) atomicAdd(&cnt[i], s_cnt[i]);
  if (stat && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&stat[6], (unsigned long long)total);
}
// off: the groups' offsets, fill: the same, as cursors; task: prefix of the
// groups of 32 chains (candidates, then pairs) that each row takes.
__global__ void __launch_bounds__(kMaxBlockRows)
    k_pool_offsets(int nrows, const int *cnt, const int *row_cnt, int *off, int *fill, int *task) {
  pdl_enter();
  __shared__ int s_tot[2][32];
  const int i = threadIdx.x, lane = i & 31, warp = i >> 5;
  const int c = i < nrows ? cnt[i] : 0;
  const int g = i < nrows ? (row_cnt[i] + 31) / 32 + (c + 31) / 32 : 0;
  int v = c, w = g;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o), z = __shfl_up_sync(0xffffffffu, w, o);
    if (lane >= o) {
      v += y;
      w += z;
    }
  }
  if (lane == 31) {
    s_tot[0][warp] = v;
    s_tot[1][warp] = w;
  }
  __syncthreads();
  for (int q = 0; q < warp; ++q) {
    v += s_tot[0][q];
    w += s_tot[1][q];
  }
  if (i < nrows) {
    off[i] = fill[i] = v - c;
    task[i] = w - g;
    if (i == nrows - 1) {
      off[nrows] = v;
      task[nrows] = w;
    }
  }
}
__global__ void k_pool_place(const int *pool_j, const int *pool_m, const int *counter, long pool_cap,
                             int *fill, int *pair_j, int *pair_m) {
  pdl_enter();
  const long total = min((long)*counter, pool_cap);
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const int m = pool_m[e], q = atomicAdd(&fill[m], 1);
    pair_j[q] = pool_j[e];
    pair_m[q] = m;
  }
}

// Canonical distances, 32 chains per warp against one batch row
// (gm_rowdot.cuh): a warp takes groups of 32 of a row's candidates or column
// pairs in a grid stride, found in the groups' prefix by two 32-way steps.  A
// pair's offer goes on one of its existing row's chains, as in the NN-Descent
// insertion (its entry is its place in pair_j).
// Pairs are spread very unevenly: a row near the middle of its cluster enters
// thousands of lists, so a fixed number of warps per row waits for such rows.
// 500 rows x 784 features against 70,000 (60 candidates and 60 pairs a row on
// average): candidates by a CTA of four warps per row and pairs with both rows
// gathered 130 us, four warps per row and kind 79 us, groups 33 us.
__global__ void __launch_bounds__(32)
    k_rescore(const float *X, int ld, const float *norms, int brow0, int nrows, const int *cand,
              long cand_ld, const int *row_cnt, float *cand_d, const int *pair_j, const int *pair_off,
              float *pair_d, const int *task, const Key *g_key, OfferChains chains) {
  pdl_enter();
  __shared__ __align__(16) RowDotTiles tiles;
  const int lane = threadIdx.x;
  const unsigned full = 0xffffffffu;
  const int total = task[nrows];
  const int step = (nrows + 31) / 32;  // (at most 32: kMaxBlockRows)
  for (int t = blockIdx.x; t < total; t += gridDim.x) {
    // the last row whose groups begin at or before t
    int at = lane * step;
    unsigned le = __ballot_sync(full, at < nrows && task[at] <= t);
    const int base = (31 - __clz(le)) * step;
    at = base + lane;
    le = __ballot_sync(full, lane < step && at < nrows && task[at] <= t);
    const int ml = base + 31 - __clz(le), row = brow0 + ml;
    const int n_cand = row_cnt[ml], g = t - task[ml], gc = (n_cand + 31) / 32;
    const bool pairs = g >= gc;
    const int begin = pairs ? pair_off[ml] : 0;
    const int cnt = pairs ? pair_off[ml + 1] - begin : n_cand;
    const int *ids = pairs ? pair_j + begin : cand + (long)ml * cand_ld;
    float *out = pairs ? pair_d + begin : cand_d + (long)ml * cand_ld;
    const int i = (pairs ? g - gc : g) * 32 + lane;
    const int j = i < cnt ? ids[i] : row;
    const float dv = canon_dist(norms[row], norms[j], warp_row_dot(X, ld, X + (size_t)row * ld, j, tiles));
    if (i < cnt) {
      out[i] = dv;
      if (pairs && make_key(dv, row) < g_key[(size_t)j * kListW + kListW - 1])
        chains.next[begin + i] = atomicExch(&chains.heads[(size_t)j * 32 + (row & 31)], begin + i);
    }
  }
}

// Exact top 32 of a row's candidates, a warp per row: chunks of 32 keys are
// sorted by a bitonic network and merged with the 32 smallest so far (the
// elementwise minimum of one list and the other reversed is bitonic and holds
// the 32 smallest of both).  Inserting one key at a time took 10.3 us for 500
// rows of ~100 candidates, this 4.9 us.
GM_D Key bitonic_step(Key k, int partner, bool up) {
  const Key o = __shfl_xor_sync(0xffffffffu, k, partner);
  return ((threadIdx.x & partner) == 0) == up ? (k < o ? k : o) : (k < o ? o : k);
}
GM_D Key warp_sort32(Key k) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int size = 2; size <= 32; size *= 2)
#pragma unroll
    for (int j = size / 2; j > 0; j /= 2) k = bitonic_step(k, j, (lane & size) == 0);
  return k;
}
constexpr int kRowWarps = 4;
__global__ void k_row_select(const float *cand_d, int brow0, int nrows, const int *cand,
                             long cand_ld, const int *row_cnt, Key *g_key,
                             unsigned long long *stat) {
  pdl_enter();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ml = blockIdx.x * kRowWarps + warp;
  if (ml >= nrows) return;
  const int cnt = row_cnt[ml];
  const int *cl = cand + (long)ml * cand_ld;
  const float *dr = cand_d + (long)ml * cand_ld;
  Key mine = kEmptyKey;
  for (int c0 = 0; c0 < cnt; c0 += 32) {
    const int c = c0 + lane;
    Key ck = c < cnt ? make_key(dr[c], cl[c]) : ~(Key)0;
    if (!__any_sync(0xffffffffu, ck < __shfl_sync(0xffffffffu, mine, 31))) continue;
    ck = warp_sort32(ck);
    ck = __shfl_sync(0xffffffffu, ck, 31 - lane);
    mine = ck < mine ? ck : mine;
#pragma unroll
    for (int j = 16; j > 0; j /= 2) mine = bitonic_step(mine, j, true);
  }
  g_key[(size_t)(brow0 + ml) * kListW + lane] = mine;
  if (stat && lane == 0) atomicAdd(&stat[6], (unsigned long long)cnt);
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                         &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  });
  return fn;
}

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

}  // namespace

int exact_dh(int d) { return (d + kTK - 1) / kTK * kTK; }

// coef of pair_bound for d features (dh padded).  With S = sum |a_i b_i| <=
// |a||b| (Cauchy-Schwarz) and u = 2^-8 the BF16 unit roundoff:
//  * operands: a_i b_i - (hi hi + hi lo + lo hi) = lo lo + hi r + lo r + r hi + ...
//    with |lo| <= u|a_i|, |r| = |a_i - hi - lo| <= u^2 |a_i|: below 3.1 u^2 S;
//  * tensor-core accumulation of m = 3 dh exact products: every operand of
//    every internal addition (the products, and the running sum once per
//    K=16 instruction; m/4 allows for up to four internal stages each) is cut
//    by at most 2^-23 of the largest magnitude involved, itself at most the
//    products' magnitude sum (1 + u)^2 S + 2 u (1 + u) S < 1.02 S: below
//    (1.25 m + 1) 2^-23 * 1.02 S;
//  * canonical FP32 chain of d fused multiply-adds (round to nearest):
//    below d 2^-24 S (1 + d 2^-24);
//  times 2 for -2 dot, and 1 + d 2^-23 because sqrt(na nb) is formed from FP32
//  norms that may fall short of |a|^2 |b|^2 by that factor.
float exact_bound_coef(int d, int dh) {
  const double u = std::ldexp(1.0, -8);
  const double m = 3.0 * dh;
  const double op = 3.1 * u * u;
  const double acc = (1.25 * m + 1.0) * std::ldexp(1.0, -23) * 1.02;
  const double canon = d * std::ldexp(1.0, -24) * (1.0 + d * std::ldexp(1.0, -24));
  const double c = 2.0 * (op + acc + canon) * (1.0 + d * std::ldexp(1.0, -23)) * 1.001;
  return (float)(c * (1.0 + 1e-6));
}

bool make_row_maps(void *xh, int n_cap, int dh, ExactMaps *out) {
  auto enc = get_encode();
  if (!enc) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)dh * 2, (cuuint64_t)std::max(n_cap, 1)};
  const cuuint64_t strides[1] = {(cuuint64_t)dh * 4};
  const cuuint32_t estr[2] = {1, 1};
  const cuuint32_t box_a[2] = {(cuuint32_t)kTK, (cuuint32_t)kTM};
  const cuuint32_t box_b[2] = {(cuuint32_t)kTK, (cuuint32_t)kTN};
  CUresult r1 = enc(reinterpret_cast<CUtensorMap *>(out->a), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, xh,
                    dims, strides, box_a, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  CUresult r2 = enc(reinterpret_cast<CUtensorMap *>(out->b), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, xh,
                    dims, strides, box_b, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r1 == CUDA_SUCCESS && r2 == CUDA_SUCCESS;
}

void launch_to_bf16(const DevState &st, void *xh, int dh, int row0, int nrows, cudaStream_t s) {
  if (nrows <= 0) return;
  const long total = (long)nrows * dh;
  launch(k_to_bf16, std::min(cdiv(total, 256), 4096), 256, 0, s, st.X, st.ld, st.d, dh, row0, nrows,
         (__nv_bfloat16 *)xh);
  note_launch();
}

template <int kPass, bool kKeepD>
static void launch_tile(const DevState &st, const ExactMaps &maps, int dh, int row0, int blk0,
                        int nrows, int n, const ExactScreen &x, long ldD, int gx, int m_tiles,
                        int tile_count, int tile_stride, const float *seed, int pre_cap,
                        int mins_ld, int col_test, const int *run_if, cudaStream_t s) {
  // once per device (sessions on several host threads may launch at once)
  static std::atomic<unsigned> configured{0u};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 32 && !(configured.load() & (1u << dev))) {
    cudaFuncSetAttribute(k_exact_dist<kPass, kKeepD>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kExactSmem);
    configured.fetch_or(1u << dev);
  }
  CUtensorMap ta, tb;
  memcpy(&ta, maps.a, sizeof(ta));
  memcpy(&tb, maps.b, sizeof(tb));
  TileScreen sc;
  sc.tile_count = tile_count;
  sc.tile_stride = tile_stride;
  sc.heaps = x.heaps;
  sc.seed = seed;
  sc.mins = x.mins;
  sc.mins_ld = mins_ld;
  sc.pre = x.pre;
  sc.pre_ub = x.pre_ub;
  sc.pre_cnt = x.pre_cnt;
  sc.pre_cap = pre_cap;
  sc.pre_over = x.pre_over;
  sc.col_test = col_test;
  sc.run_if = run_if;
  sc.row_t = x.row_t;
  sc.cand = x.cand;
  sc.cand_ld = ldD;
  sc.row_cnt = x.row_cnt;
  sc.pool_j = x.pool_j;
  sc.pool_m = x.pool_m;
  sc.pool_counter = x.counter;
  sc.pool_cap = x.pool_cap;
  sc.g_key = st.g_key;
  sc.n_exist = row0;
  sc.coef = exact_bound_coef(st.d, dh);
  launch(k_exact_dist<kPass, kKeepD>, dim3(gx, m_tiles), exact_threads(kPass), kExactSmem, s, ta, tb,
         row0 + blk0, nrows, n, dh / kTK, dh, st.norms, st.snorms, sc, x.D, ldD, st.err);
  note_launch();
}

// Up to kExactRoomTiles column tiles the segments hold every column.  Rows that
// come ordered, by cluster say, need it: a row's neighbours then lie in few
// chunks, its seed in another cluster, and the store pass admits whole tiles.
// With segments of 64 entries 13 of the 16 blocks of 4,999 rows x 131 in ten
// ordered clusters overflowed and ran the heap passes as well: a build of cycles
// of 333 took 4.4 ms, 2.7 with the room (shuffled rows 2.3 and 2.1).  Twelve bytes
// for each of 8,448 columns and 1,024 block rows are 104 MB; from 132 tiles on the
// segments of 64 entries take as much.
// Column tiles of the seed pass (evenly spaced over the columns): at least
// 16, and one in 8 of the block's tiles, so that the seed stays a low
// quantile of the row's upper bounds at any column count; all of them up to 32.
// One in 16, 8, 4 (the seed and store passes of 1,000 rows x 128 against
// 160,000, on average over an insertion): 120, 107, 103 us; of 500 rows x 784
// against 70,000: 88, 87, 92 us.
// It needs 32 chunks of 32 columns, and some more to be low (from kSeedMin
// tiles, 40 chunks: it then admits about 65 of 1,280 columns).  Below that
// there is no seed and every column is stored, where the segments have room for
// them all.  The heap and candidate passes, which need no room: a thread's heap
// of a row and one group of epilogue warps make them 170 us a block where the
// seed and store passes and their selections take 43 us (333 rows x 131 against
// 4,000), and 147 us where the store of every column takes 34 (333 rows against
// 333 to 999).
constexpr int kSeedTiles = 16;
constexpr int kSeedEvery = 8;
constexpr int kSeedMin = 5;

int exact_seed_tiles(int n_tiles) {
  return n_tiles <= 2 * kSeedTiles ? std::max(n_tiles, 1) : std::max(kSeedTiles, n_tiles / kSeedEvery);
}

void launch_exact_dist(const DevState &st, const ExactMaps &maps, int dh, int row0, int blk0,
                       int nrows, int n, const ExactScreen &x, long ldD, bool keep_d, int sms,
                       cudaStream_t s) {
  const int n_tiles = cdiv(n, kTN);
  const int m_tiles = cdiv(nrows, kTM);
  // CTAs per row tile so that the grid covers the SMs once; where the segments
  // are to hold every column, no more than the column tiles per CTA call for
  // (the longest CTA stays, and the segments are as long as those tiles)
  int gx = std::max(1, std::min(n_tiles, std::max(1, sms / m_tiles)));
  if (n_tiles <= kExactRoomTiles) gx = cdiv(n_tiles, cdiv(n_tiles, gx));
  const bool kd = keep_d && x.D;
  const int tiles = exact_seed_tiles(n_tiles);
  // entries per stored segment: the row's whole allocation shared by its
  // tile's CTAs (fewer CTAs per row tile, longer segments)
  const int cap = x.pre_fixed || gx > x.pre_gx ? x.pre_cap : (int)((long)x.pre_gx * x.pre_cap / gx);
  // columns of a CTA: with room for all of them no segment overflows
  const int cta_cols = cdiv(n_tiles, gx) * kTN;
  const bool seeded = n_tiles >= kSeedMin;
  if (x.pre && cap > 0 && gx <= x.pre_gx && gx <= kPreSegs &&
      (seeded ? tiles * (kTN / 32) <= x.mins_ld : cap >= cta_cols)) {
    // seed pass over a spread sample of tiles (or no seed: every column is
    // stored), then the store pass
    const int mins_ld = seeded ? tiles * (kTN / 32) : 0;
    if (seeded)
      launch_tile<0, false>(st, maps, dh, row0, blk0, nrows, n, x, ldD,
                            std::max(1, std::min(tiles, std::max(1, sms / m_tiles))), m_tiles, tiles,
                            n_tiles / tiles, nullptr, 0, mins_ld, 0, nullptr, s);
    launch(k_seed_select, nrows, kSeedThreads, std::min(mins_ld, kSeedStage) * sizeof(float), s, x.mins, mins_ld,
           x.seed, x.row_cnt, x.pcnt, x.counter, x.pre_over);
    if (kd)
      launch_tile<3, true>(st, maps, dh, row0, blk0, nrows, n, x, ldD, gx, m_tiles, n_tiles, 1, x.seed,
                           cap, 0, 0, nullptr, s);
    else
      launch_tile<3, false>(st, maps, dh, row0, blk0, nrows, n, x, ldD, gx, m_tiles, n_tiles, 1, x.seed,
                            cap, 0, 0, nullptr, s);
    launch(k_pre_select, nrows, kPreThreads, 0, s, x.pre, x.pre_ub, x.pre_cnt, gx, cap, x.pre_over, n,
           x.row_t, x.cand, ldD, x.row_cnt, st.stat);
    note_launch(2);
    if (cap >= cta_cols) return;
    // after an overflow only: the heap pass (seed-capped; its pairs were
    // already pooled), the threshold and the candidate pass
    launch_tile<1, false>(st, maps, dh, row0, blk0, nrows, n, x, ldD, gx, m_tiles, n_tiles, 1, x.seed, 0,
                          0, 0, x.pre_over, s);
    launch(k_row_threshold, cdiv(nrows, kFinalWarps), kFinalWarps * 32, 0, s, x.heaps, gx, nrows, n, x.seed,
           x.row_t, x.pre_over, st.stat);
    note_launch();
    launch_tile<2, false>(st, maps, dh, row0, blk0, nrows, n, x, ldD, gx, m_tiles, n_tiles, 1, nullptr, 0,
                          0, 0, x.pre_over, s);
    return;
  }
  cudaMemsetAsync(x.row_cnt, 0, (size_t)nrows * sizeof(int), s);
  cudaMemsetAsync(x.pcnt, 0, (size_t)nrows * sizeof(int), s);
  cudaMemsetAsync(x.counter, 0, sizeof(int), s);
  if (kd)
    launch_tile<1, true>(st, maps, dh, row0, blk0, nrows, n, x, ldD, gx, m_tiles, n_tiles, 1, nullptr, 0,
                         0, 1, nullptr, s);
  else
    launch_tile<1, false>(st, maps, dh, row0, blk0, nrows, n, x, ldD, gx, m_tiles, n_tiles, 1, nullptr, 0,
                          0, 1, nullptr, s);
  launch(k_row_threshold, cdiv(nrows, kFinalWarps), kFinalWarps * 32, 0, s, x.heaps, gx, nrows, n, nullptr,
         x.row_t, nullptr, st.stat);
  note_launch();
  launch_tile<2, false>(st, maps, dh, row0, blk0, nrows, n, x, ldD, gx, m_tiles, n_tiles, 1, nullptr, 0,
                        0, 0, nullptr, s);
}

void launch_exact_screen(const DevState &st, int row0, int blk0, int nrows, int n,
                         const ExactScreen &x, long ldD, int sms, cudaStream_t s) {
  if (nrows <= 0 || n <= 0) return;
  const int brow0 = row0 + blk0;  // global first row of the block
  const int grid = 4 * std::max(sms, 1);
  // the pairs as found are done with once placed: pool_m holds the chains
  const OfferChains chains{x.heads, x.pool_m};
  if (row0 > 0) {
    launch(k_pool_count, grid, 256, 0, s, x.pool_m, x.counter, x.pool_cap, nrows, x.pcnt, st.stat);
    note_launch();
  }
  launch(k_pool_offsets, 1, kMaxBlockRows, 0, s, nrows, x.pcnt, x.row_cnt, x.poff, x.pfill, x.ptask);
  if (row0 > 0) {
    launch(k_pool_place, grid, 256, 0, s, x.pool_j, x.pool_m, x.counter, x.pool_cap, x.pfill, x.pair_j,
           x.pair_m);
    note_launch();
  }
  // (twelve CTAs fit an SM)
  launch(k_rescore, 12 * std::max(sms, 1), 32, 0, s, st.X, st.ld, st.norms, brow0, nrows, x.cand, ldD,
         x.row_cnt, x.cand_d, x.pair_j, x.poff, x.pool_d, x.ptask, st.g_key, chains);
  launch(k_row_select, cdiv(nrows, kRowWarps), kRowWarps * 32, 0, s, x.cand_d, brow0, nrows, x.cand, ldD,
         x.row_cnt, st.g_key, st.stat);
  note_launch(2);
  if (row0 > 0) launch_merge_offers(st, row0, brow0, chains, x.pool_d, x.pair_m, nullptr, nullptr, s);
}

}  // namespace gm
