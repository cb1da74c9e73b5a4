// Canonical FP32 dot products against gathered feature rows, one chain per
// lane: shared by the NN-Descent insertion and the exact re-score.
//
// A warp forms 32 sequential fused multiply-add chains at once.  The 32 rows
// are brought in 32 features at a time by 16-byte cp.async (eight lanes per
// row, four rows per instruction) into a ring of kDotRing warp-private
// shared-memory slots, kDotRing - 1 chunks ahead of the chains; a row takes 36
// words in a slot, so the eight lanes of a quarter-warp's 16-byte read fall on
// distinct banks.  Rows must start on 16-byte boundaries (ld a multiple of 4)
// with zeros from d to ld: fma(0, 0, x) = x keeps the chain's value.
#pragma once

#include "gm_common.cuh"

namespace gm {

constexpr int kDotRing = 4;
constexpr int kDotChunk = 32;           // features per chunk
constexpr int kDotLd = kDotChunk + 4;   // words per row in a slot

// Slots of one warp: the lanes' rows, and one row common to the warp.
struct RowDotTiles {
  float b[kDotRing][32][kDotLd];
  float a[kDotRing][kDotChunk];
};
GM_D void dot_cp16(float *dst, const float *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
GM_D void dot_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// All but the newest kDotRing - 1 groups have landed.
GM_D void dot_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kDotRing - 1) : "memory"); }

GM_D float dot_fma4(float4 a, float4 b, float acc) {
  acc = __fmaf_rn(a.x, b.x, acc);
  acc = __fmaf_rn(a.y, b.y, acc);
  acc = __fmaf_rn(a.z, b.z, acc);
  return __fmaf_rn(a.w, b.w, acc);
}

// Lane l: dot of row xa (common to the warp) and row rb (lane l's own).
// Every lane takes part; lanes without work pass any valid row.
GM_D float warp_row_dot(const float *X, int ld, const float *xa, int rb, RowDotTiles &t) {
  const int lane = threadIdx.x & 31, q = lane & 7, r0 = lane >> 3;
  const float *src[8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
    src[i] = X + (size_t)__shfl_sync(0xffffffffu, rb, r0 + 4 * i) * ld + 4 * q;
  const int nch = (ld + kDotChunk - 1) / kDotChunk;
  // one commit group per chunk index (empty past the last chunk)
  auto issue = [&](int c) {
    const int col = c * kDotChunk + 4 * q;
    if (col < ld) {
      const int slot = c % kDotRing;
      if (r0 == 0) dot_cp16(&t.a[slot][4 * q], xa + col);
#pragma unroll
      for (int i = 0; i < 8; ++i) dot_cp16(&t.b[slot][r0 + 4 * i][4 * q], src[i] + c * kDotChunk);
    }
    dot_commit();
  };
  for (int c = 0; c < kDotRing - 1; ++c) issue(c);
  float dot = 0.0f;
  for (int c = 0; c < nch; ++c) {
    issue(c + kDotRing - 1);  // refills the slot the previous iteration consumed
    dot_wait();
    __syncwarp();
    const int slot = c % kDotRing, nq = min(kDotChunk, ld - c * kDotChunk) >> 2;
    const float4 *av = reinterpret_cast<const float4 *>(t.a[slot]);
    const float4 *bv = reinterpret_cast<const float4 *>(t.b[slot][lane]);
    if (nq == 8) {
#pragma unroll
      for (int i = 0; i < 8; ++i) dot = dot_fma4(av[i], bv[i], dot);
    } else {
      for (int i = 0; i < nq; ++i) dot = dot_fma4(av[i], bv[i], dot);
    }
    __syncwarp();
  }
  return dot;
}

}  // namespace gm
