// Embedding phase: fuzzy simplicial set over the published k-NN (self
// prepended), edge scheduling and negative-sampling SGD.  Restates the
// reference's embedding_kernel.cuh and Impl::embed (impl.cuh:335-500) with
// every count and threshold kept on the device (no host round trips).
#include <algorithm>

#include <mutex>

#include "gm_common.cuh"
#include "gm_kernels.h"

namespace gm {

// Scalar slots in EmbedScratch.
//   fscal: 0 mean_dist, 1 max_w, 2 rounding, 3 x_min, 4 x_max
//   iscal: 0 nnz (directed + extras), 1 extras, 2 nnz after trim, 3 max degree,
//          4 rows n (read by the SGD epochs so a captured graph stays valid),
//          5 rows left for k_fix_sigma
enum { FS_MEAN = 0, FS_MAXW = 1, FS_ROUND = 2, FS_XMIN = 3, FS_XMAX = 4 };
enum { IS_NNZ = 0, IS_EXTRA = 1, IS_NNZ2 = 2, IS_MAXDEG = 3, IS_N = 4, IS_MARKED = 5 };

namespace {

constexpr float kSmoothTol = 1e-5f;  // SMOOTH_K_TOLERANCE
constexpr float kMinKDistScale = 1e-3f;

// Embed-time k-NN (reference prepend_self_knn_kernel, embedding_kernel.cuh:599-631):
// column 0 is the row itself at distance 0; column c >= 1 is published
// neighbour c-1 (the k-th is dropped); euclidean distances are square-rooted.
GM_D uint32_t eidx(const uint32_t *pub_idx, int k, int row, int c) {
  return c == 0 ? (uint32_t)row : pub_idx[(size_t)row * (k + 1) + (c - 1)];
}
GM_D float edist(const float *pub_dist, int k, int row, int c, int euclid) {
  if (c == 0) return 0.0f;
  const float v = pub_dist[(size_t)row * (k + 1) + (c - 1)];
  return euclid ? __fsqrt_rn(v > 0.0f ? v : 0.0f) : v;
}
GM_D bool valid_d(float v) { return isfinite(v) && v >= 0.0f && v < FLT_MAX / 2.0f; }

GM_D float membership(float dist, float rho, float sigma) {
  const float dr = __fsub_rn(dist, rho);
  if (dr <= 0.0f || sigma == 0.0f) return 1.0f;
  const float v = gm_expf(-__fdiv_rn(dr, sigma));
  return v < FLT_MIN ? FLT_MIN : v;
}

// Block sums of the embed-time distances (256 per block, FP32 tree).  Clears
// what the kernels after it count into: the head degrees, their maximum, the
// largest weight, the rows left for k_fix_sigma.
__global__ void __launch_bounds__(256)
    k_mean_partial(const float *pub_dist, int n, int k, int euclid, float *part, int *ipart, int *deg,
                   int *iscal, float *fscal) {
  pdl_enter();
  __shared__ float ss[256];
  const int t = threadIdx.x;
  const long g = (long)blockIdx.x * 256 + t;
  if (g < n) deg[g] = 0;
  if (g == 0) {
    iscal[IS_MAXDEG] = iscal[IS_MARKED] = 0;
    fscal[FS_MAXW] = 0.0f;
  }
  float v = 0.0f;
  bool ok = false;
  if (g < (long)n * k) {
    const int row0 = (int)((long)blockIdx.x * 256 / k);
    const int in = (int)((long)blockIdx.x * 256 - (long)row0 * k) + t;
    const float raw = edist(pub_dist, k, row0 + in / k, in % k, euclid);
    if (raw >= 0.0f && raw < FLT_MAX / 2.0f) {
      v = raw;
      ok = true;
    }
  }
  ss[t] = v;
  const int c = __syncthreads_count(ok);
#pragma unroll
  for (int s = 128; s >= 32; s >>= 1) {
    if (t < s) ss[t] = __fadd_rn(ss[t], ss[t + s]);
    __syncthreads();
  }
  if (t >= 32) return;
  v = ss[t];
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) v = __fadd_rn(v, __shfl_down_sync(0xffffffffu, v, s));
  if (t == 0) {
    part[blockIdx.x] = v;
    ipart[blockIdx.x] = c;
  }
}

// The mean of the partials, added in index order by one thread (each addition
// waits for the one before it; the partials come through shared memory, four
// per read).  The whole block calls it.
constexpr int kMeanStage = 2048;
GM_D void mean_final(const float *part, const int *ipart, int nb, float *fscal, float *stage) {
  float s = 0.0f;
  int c = 0;
  for (int i0 = 0; i0 < nb; i0 += kMeanStage) {
    const int m = min(kMeanStage, nb - i0);
    __syncthreads();
    for (int i = threadIdx.x; i < (m + 3) / 4 * 4; i += blockDim.x) {
      stage[i] = i < m ? part[i0 + i] : 0.0f;
      c += i < m ? ipart[i0 + i] : 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      // (the partials are not negative: adding a +0 of the padding is exact)
#pragma unroll 8
      for (int i = 0; i < m; i += 4) {
        const float4 v = *reinterpret_cast<const float4 *>(stage + i);
        s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, v.x), v.y), v.z), v.w);
      }
    }
  }
  __shared__ unsigned long long s_c;
  if (threadIdx.x == 0) s_c = 0ull;
  __syncthreads();
  if (c) atomicAdd(&s_c, (unsigned long long)c);
  __syncthreads();
  if (threadIdx.x == 0)
    fscal[FS_MEAN] = (s_c > 0ull && isfinite(s) && s > 0.0f) ? __fdiv_rn(s, (float)(long)s_c) : 1.0f;
}

// Exact sum of two floats: s + e (Knuth, The Art of Computer Programming,
// vol. 2, 4.2.2, theorem B).
GM_D void two_sum(float a, float b, float &s, float &e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// Where the bisection's sum is known to lie outside the tolerance: at sigma <=
// .x below the target, at sigma >= .y above it (-1 and infinity: nowhere).  The
// sum over sigma rises, so one value decides for all beyond it.  Newton's
// method on the logarithm of g(l) = sum exp(-d l), l = 1 / sigma, which is
// convex in l, from l = 0 (g = the number of terms); then g at both sides of
// where it stopped, about kAside from the target.
// Rounding: __expf is good to 2 + 1.17 |x| units in the last place, so with up
// to 31 terms g, near a target of at most 5, is off by less than 3e-6 for that,
// 1.5e-6 for the additions and 1.5e-6 for the roundings of l d and 1 / l; the
// bisection's own sum (gm_expf, a rounded quotient) by 2e-6 there and by 8e-6
// at the largest sums.  With g kSure from the target the bisection's sum is more
// than twice the tolerance from it, on the same side, there and beyond.
constexpr float kSure = 4e-5f, kAside = 8e-5f;
constexpr int kNewtonSteps = 8;
template <int L>
GM_D float2 sigma_bracket(const float (&dj)[4], const bool (&contrib)[4], float target) {
  const unsigned full = 0xffffffffu;
  auto row_sum = [&](float v) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(full, v, o));
    return v;
  };
  float d[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) d[j] = fmaxf(dj[j], 0.0f);
  auto terms = [&](float l, float &g, float &slope) {
    float e[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) e[j] = contrib[j] ? __expf(__fmul_rn(-d[j], l)) : 0.0f;
    g = row_sum(__fadd_rn(__fadd_rn(e[0], e[1]), __fadd_rn(e[2], e[3])));
    slope = __fadd_rn(__fadd_rn(__fmul_rn(d[0], e[0]), __fmul_rn(d[1], e[1])),
                      __fadd_rn(__fmul_rn(d[2], e[2]), __fmul_rn(d[3], e[3])));
  };
  float ones = 0.0f;
#pragma unroll
  for (int j = 0; j < 4; ++j) ones = __fadd_rn(ones, contrib[j] && !(dj[j] > 0.0f) ? 1.0f : 0.0f);
  ones = row_sum(ones);
  float l = 0.0f, slope = 0.0f;
  for (int i = 0; i < kNewtonSteps; ++i) {
    float g;
    terms(l, g, slope);
    slope = row_sum(slope);
    const bool near = fabsf(__fsub_rn(g, target)) < 0.1f * kAside;
    if (!near) l = __fadd_rn(l, __fmul_rn(__fdividef(g, slope), __logf(__fdividef(g, target))));
    if (__all_sync(full, near || !(l > 0.0f) || ones > target)) break;
  }
  const float aside = __fdividef(kAside, slope);
  const float la = __fadd_rn(l, aside), lb = __fsub_rn(l, aside);
  float ga, gb, unused;
  terms(la, ga, unused);
  terms(lb, gb, unused);
  float2 r = make_float2(-1.0f, __int_as_float(0x7f800000));
  if (lb > 0.0f && isfinite(la) && target <= 5.0f) {
    if (ga <= target - kSure) r.x = __fdiv_rn(1.0f, la);
    if (gb >= target + kSure) r.y = __fdiv_rn(1.0f, lb);
  }
  if (ones >= target + kSure) r.y = 0.0f;  // (at every sigma)
  return r;
}

// sigma / rho by bisection (reference smooth_knn_dist_kernel,
// embedding_kernel.cuh:135-207), L lanes per row (4 for k <= 16, 8 for k <=
// 32), terms q, q + L, q + 2L, q + 3L on lane q.  The bisection's target sum is
// defined in FP64, by the xor butterfly of 32 lanes with term c on lane c (the
// terms of lanes >= k are +0, adding them is exact).  Its only use is two
// comparisons (within the tolerance of the target; above it), so it is formed
// in FP32 with exact error terms, to within 1e-12, and FP64 additions run only
// where that cannot decide (within kUnsure of the tolerance's edge): FP64 has
// 1/64 of the FP32 rate here and bound the kernel.  The other terms of the
// FP64 tree: (t0 + t2) + (t1 + t3) on each lane, then xor L/2 .. 1.
// Most of the bisection's steps are decided by where its sum is known to lie
// (sigma_bracket), and take no sum: three or four of about twenty do.
// 70,000 rows at k = 15: 151 us in FP64, 56 with FP32 sums, 33 so; 100,000 at k = 30:
// 1508 (a warp per row), 187, 70.
// The first CTA takes the global mean meanwhile, which only rows without a
// positive distance need: those are left marked (sigma < 0, *marked set) for
// k_fix_sigma.
constexpr float kUnsure = 1e-10f;
constexpr int kSmoothThreads = 256;
template <int L>
__global__ void __launch_bounds__(kSmoothThreads)
    k_smooth_knn(const float *pub_dist, int n, int k, int euclid, double target, float t_hi,
                 float t_lo, float *sigma, float *rho, const float *part, const int *ipart, int nb,
                 float *fscal, int *marked) {
  pdl_enter();
  __shared__ __align__(16) float stage[kMeanStage];
  if (blockIdx.x == 0) {
    mean_final(part, ipart, nb, fscal, stage);
    return;
  }
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int q = lane & (L - 1), base = lane - q;
  const long gid = ((long)(blockIdx.x - 1) * kSmoothThreads + threadIdx.x) / L;
  const bool live = gid < n;
  const int row = live ? (int)gid : 0;
  float raw[4], san[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = q + L * j;
    raw[j] = (live && c < k) ? edist(pub_dist, k, row, c, euclid) : 0.0f;
    san[j] = (live && c < k && valid_d(raw[j])) ? raw[j] : 0.0f;
  }
  // row sum in column order, first nonzero column
  float sum = 0.0f, r = 0.0f;
  bool found = false;
#pragma unroll
  for (int c = 0; c < 4 * L; ++c) {
    const float v = __shfl_sync(full, san[c / L], base + (c & (L - 1)));
    if (c < k) {
      sum = __fadd_rn(sum, v);
      if (!found && v > 0.0f) {
        found = true;
        r = v;
      }
    }
  }
  const float row_mean = __fdiv_rn(sum, (float)k);
  float lo = 0.0f, hi = FLT_MAX, mid = 1.0f;
  float dj[4];
  bool contrib[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int c = q + L * j;
    contrib[j] = c >= 2 && c < k;
    dj[j] = __fsub_rn(san[j], r);
  }
  bool done = !live || !found;
  const float2 known = sigma_bracket<L>(dj, contrib, t_hi);
  // one bisection step, when the sum at mid is not within the tolerance
  auto step = [&](bool above) {
    if (above) {
      hi = mid;
      mid = __fmul_rn(__fadd_rn(lo, hi), 0.5f);
    } else {
      lo = mid;
      mid = (hi == FLT_MAX) ? __fmul_rn(mid, 2.0f) : __fmul_rn(__fadd_rn(lo, hi), 0.5f);
    }
  };
  for (int it = 0;; ++it) {
    while (!done && it < 64 && (mid <= known.x || mid >= known.y)) {
      step(mid >= known.y);
      ++it;
    }
    if (it >= 64) done = true;
    if (__all_sync(full, done)) break;
    float t[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      t[j] = 0.0f;
      if (contrib[j] && !done) t[j] = (dj[j] > 0.0f) ? gm_expf(__fdiv_rn(-dj[j], mid)) : 1.0f;
    }
    float s0, e0, s1, e1, s, e;
    two_sum(t[0], t[2], s0, e0);
    two_sum(t[1], t[3], s1, e1);
    two_sum(s0, s1, s, e);
    e = __fadd_rn(e, __fadd_rn(e0, e1));
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
      const float so = __shfl_xor_sync(full, s, o), eo = __shfl_xor_sync(full, e, o);
      float sn, en;
      two_sum(s, so, sn, en);
      s = sn;
      e = __fadd_rn(en, __fadd_rn(e, eo));
    }
    const float off = __fadd_rn(__fsub_rn(s, t_hi), __fsub_rn(e, t_lo));
    bool within = fabsf(off) < kSmoothTol, above = off > 0.0f;
    const bool unsure = !done && fabsf(__fsub_rn(fabsf(off), kSmoothTol)) <= kUnsure;
    if (__any_sync(full, unsure)) {
      double term = ((double)t[0] + (double)t[2]) + ((double)t[1] + (double)t[3]);
#pragma unroll
      for (int o = L / 2; o > 0; o >>= 1) term += __shfl_xor_sync(full, term, o);
      if (unsure) {
        within = fabs(term - target) < (double)kSmoothTol;
        above = term > target;
      }
    }
    if (done) continue;
    if (within) done = true;
    else step(above);
  }
  if (!live || q != 0) return;
  if (!found) {
    rho[row] = 0.0f;
    sigma[row] = -1.0f;
    *marked = 1;
    return;
  }
  if (!isfinite(mid) || mid <= 0.0f) mid = 1.0f;
  // (r > 0: the row's own mean is the scale, never the global one)
  const float min_scale = __fmul_rn(kMinKDistScale, row_mean);
  rho[row] = r;
  sigma[row] = mid < min_scale ? min_scale : mid;
}

// Rows without a positive distance: a share of the global mean.
__global__ void k_fix_sigma(int n, const float *fscal, float *sigma, const int *marked) {
  pdl_enter();
  if (!*marked) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && sigma[i] < 0.0f) sigma[i] = __fmul_rn(kMinKDistScale, fscal[FS_MEAN]);
}

// The block's largest m into *to (both >= 0); the whole block calls it.
GM_D void block_max(int m, int *to) {
  __shared__ int s_max;
  if (threadIdx.x == 0) s_max = 0;
  __syncthreads();
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(&s_max, m);
  __syncthreads();
  // (most blocks find a value that is no smaller)
  if (threadIdx.x == 0 && s_max > *(volatile int *)to) atomicMax(to, s_max);
}

// Directed membership p_ij for batch rows and the fuzzy union
// w = p_ij + p_ji - p_ij p_ji; flag marks edges whose reverse is absent
// (reference: embedding_kernel.cuh:214-320).  Their largest w goes to
// fscal[FS_MAXW] by the order of the bits (w >= 0; an extra edge has the w of
// the edge it reverses).
// Bound by the reads of the other rows' lists out of L2 (120 bytes an edge at k
// = 30: 128 us for 3 million edges; 16 or 32 lanes that read a list in one
// request take as long, and 8.5 us instead of 5.6 for 15,000 edges).
__global__ void __launch_bounds__(256)
    k_memb_sym(const uint32_t *pub_idx, const float *pub_dist, int n, int k, int euclid,
               const float *sigma, const float *rho, const int *batch, int nb, int *coo_row,
               int *coo_col, float *coo_val, int *flag, float *fscal) {
  pdl_enter();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  float w = 0.0f;
  if (tid < nb * k) {
    const int bi = tid / k, ki = tid - bi * k;
    const int row = batch[bi];
    const uint32_t raw_col = eidx(pub_idx, k, row, ki);
    const bool valid_col = raw_col < (uint32_t)n;
    const int col = valid_col ? (int)raw_col : row;
    const float dist = edist(pub_dist, k, row, ki, euclid);
    float pij = 0.0f;
    if (valid_col && col != row && valid_d(dist)) pij = membership(dist, rho[row], sigma[row]);
    float pji = 0.0f;
    for (int kj = 0; kj < k; ++kj) {
      if ((int)eidx(pub_idx, k, col, kj) == row) {
        const float dji = edist(pub_dist, k, col, kj, euclid);
        if (!valid_d(dji)) break;
        pji = membership(dji, rho[col], sigma[col]);
        break;
      }
    }
    w = __fmaf_rn(-pij, pji, __fadd_rn(pij, pji));
    coo_row[tid] = row;
    coo_col[tid] = col;
    coo_val[tid] = w;
    flag[tid] = (pji == 0.0f) ? 1 : 0;
  }
  block_max(w > 0.0f ? __float_as_int(w) : 0, reinterpret_cast<int *>(&fscal[FS_MAXW]));
}

__global__ void k_write_extras(const int *idx, const int *cnt, int ndir, int *coo_row,
                               int *coo_col, float *coo_val, int *iscal) {
  pdl_enter();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = *cnt;
  if (q == 0) {
    iscal[IS_NNZ] = ndir + c;
    iscal[IS_EXTRA] = c;
  }
  if (q >= c) return;
  const int src = idx[q];
  coo_row[ndir + q] = coo_col[src];
  coo_col[ndir + q] = coo_row[src];
  coo_val[ndir + q] = coo_val[src];
}

// Gather survivors; epochs_per_sample; head degrees and their maximum; epoch
// state (reference: :469-495, :405-460).  A row's edges stand together but
// for the extras: the first of each run in a warp adds the run's length (one
// atomic for up to 32 edges).  Bound by the chain of loads from an edge's index
// to its degree: kGatherAhead edges a thread, their loads together.
// 4.3 million edges: 67 us with one a thread and an atomic each, 43 us so.
constexpr int kGatherAhead = 4;
__global__ void __launch_bounds__(256)
    k_gather_sched(const int *idx, int *iscal, const int *crow, const int *ccol, const float *cval,
                   const float *fscal, int n_epochs, float nsr_inv, int *trow, int *tcol, float *eps,
                   float *next_s, float *next_n, int *deg) {
  pdl_enter();
  const int nnz = iscal[IS_NNZ2], q0 = blockIdx.x * 256 * kGatherAhead;
  if (q0 >= nnz) return;
  const int lane = threadIdx.x & 31;
  const float mw = fscal[FS_MAXW];
  int src[kGatherAhead], head[kGatherAhead], tail[kGatherAhead], dmax = 0;
  float w[kGatherAhead];
#pragma unroll
  for (int u = 0; u < kGatherAhead; ++u) {
    const int q = q0 + u * 256 + threadIdx.x;
    src[u] = q < nnz ? idx[q] : -1;
  }
#pragma unroll
  for (int u = 0; u < kGatherAhead; ++u) {
    head[u] = src[u] >= 0 ? crow[src[u]] : -1;
    tail[u] = src[u] >= 0 ? ccol[src[u]] : 0;
    w[u] = src[u] >= 0 ? cval[src[u]] : 0.0f;
  }
#pragma unroll
  for (int u = 0; u < kGatherAhead; ++u) {
    const int prev = __shfl_up_sync(0xffffffffu, head[u], 1);
    const bool first = lane == 0 || head[u] != prev;
    const unsigned starts = __ballot_sync(0xffffffffu, first);
    if (head[u] < 0) continue;
    const int q = q0 + u * 256 + threadIdx.x;
    const float ns = __fmul_rn((float)n_epochs, __fdiv_rn(w[u], mw));
    const float e = (ns > 0.0f) ? __fdiv_rn((float)n_epochs, ns) : -1.0f;
    trow[q] = head[u];
    tcol[q] = tail[u];
    eps[q] = e;
    next_s[q] = e;
    next_n[q] = __fmul_rn(e, nsr_inv);
    if (first) {
      const unsigned later = lane == 31 ? 0u : starts >> (lane + 1);
      const int run = later ? __ffs(later) : 32 - lane;
      dmax = max(dmax, atomicAdd(&deg[head[u]], run) + run);
    }
  }
  block_max(dmax, &iscal[IS_MAXDEG]);
}

// Gradient rounding factor 2^ceil-ish via frexp (reference :433-460), and the
// SGD's row count.
__global__ void k_rounding(int *iscal, float *fscal, float alpha, int n) {
  pdl_enter();
  const int nnz = iscal[IS_NNZ2];
  const int md = iscal[IS_MAXDEG];
  float r = 1.0f;
  if (nnz > 0 && md > 0) {
    const float max_abs = __fmul_rn(__fmul_rn((float)md, 4.0f), fabsf(alpha));
    const float denom = __fsub_rn(1.0f, __fmul_rn(__fmul_rn(2.0f, (float)md), FLT_EPSILON));
    const float delta = __fdiv_rn(max_abs, denom);
    int ex;
    frexpf(delta, &ex);
    r = ldexpf(1.0f, ex);
  }
  fscal[FS_ROUND] = r;
  iscal[IS_N] = n;
}

GM_D float fclip(float v) {
  if (!isfinite(v)) return 0.0f;
  return fmaxf(fminf(v, 4.0f), -4.0f);
}
GM_D float trunc_grad(float rounding, float x) {
  return __fsub_rn(__fadd_rn(rounding, x), rounding);
}

// One edge of one SGD epoch (reference optimize_batch_kernel, :509-589;
// Hogwild updates, tail moved by rounded atomics, head accumulated then
// added).  Embedding positions are read through L2 (ld.global.cg): in the
// persistent kernel other SMs update them between epochs.  The positions of
// the head, the tail and the first kNegAhead negative samples (rows drawn in
// the same Philox order) are fetched together; a sample that is this edge's
// own tail is advanced by this thread's tail update, which in sequential
// order precedes the read.  powf(d2, b - 1) and powf(d2, b) share one log.
constexpr int kNegAhead = 8;

// 8-byte embedding row read through L2, issued where it stands (volatile, a
// memory clobber): the sample positions are fetched ahead of their use.
GM_D float2 ld_pos(const float *p) {
  float2 v;
  asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
  return v;
}

// x mod n by a precomputed 64-bit reciprocal, exact for every 32-bit x and
// n >= 1 (Lemire, Kaser and Kurz, "Faster remainder by direct computation",
// 2019): M = floor((2^64 - 1) / n) + 1, x mod n = high64((M * x mod 2^64) * n).
GM_D uint32_t fastmod(uint32_t x, uint64_t M, uint32_t n) {
  return (uint32_t)__umul64hi(M * (uint64_t)x, (uint64_t)n);
}

// Number of negative samples of an active edge at epoch fe.
GM_D int sgd_n_neg(float fe, float nn, float ep_neg) {
  return (int)__fdiv_rn(__fsub_rn(fe, nn), ep_neg);
}

// One edge of one epoch.  The head and tail positions are read first; the
// first kNegAhead negative samples (rows from this edge's Philox stream,
// blocks 0 and 1, words in order, computed directly into registers) are
// fetched together after the attraction and the tail update, ahead of the
// sequential repulsions.  powf(d2, b - 1) and powf(d2, b) share one log.
GM_D void sgd_edge(float *emb, int row, int j, int kk, float ep, float &ns, float &nn, int n,
                   uint64_t M, float rounding, float alpha, float fe, float gamma, float a,
                   float b, float nsr_inv, uint64_t seed, unsigned &my_edges, unsigned &my_negs) {
  ++my_edges;
  float *cp = emb + (size_t)j * 2;
  float *op = emb + (size_t)kk * 2;
  const float2 cpv = ld_pos(cp), opv = ld_pos(op);
  float cur0 = cpv.x, cur1 = cpv.y;
  const float ep_neg = __fmul_rn(ep, nsr_inv);
  const int n_neg = sgd_n_neg(fe, nn, ep_neg);
  int rr[kNegAhead];
  float2 qq[kNegAhead];
  if (n_neg > 0) {
    const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
    uint32_t w[8];
    philox_block((uint32_t)row, 0u, kTagNegSample, 0u, k0, k1, w);
    if (n_neg > 4) philox_block((uint32_t)row, 1u, kTagNegSample, 0u, k0, k1, w + 4);
#pragma unroll
    for (int p = 0; p < kNegAhead; ++p) {
      if (p < n_neg) {
        rr[p] = (int)fastmod(w[p], M, (uint32_t)n);
      }
    }
  }
  const float dx = __fsub_rn(cur0, opv.x), dy = __fsub_rn(cur1, opv.y);
  const float d2 = __fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy));
  float attr = 0.0f;
  if (d2 > 0.0f) {
    const float lg = gm_logf(d2);
    const float bm1 = __fsub_rn(b, 1.0f);
    const float p_bm1 = bm1 == 0.0f ? 1.0f : gm_expf(__fmul_rn(bm1, lg));
    const float p_b = b == 0.0f ? 1.0f : gm_expf(__fmul_rn(b, lg));
    attr = __fdiv_rn(__fmul_rn(__fmul_rn(-2.0f, __fmul_rn(a, b)), p_bm1),
                     __fadd_rn(__fmul_rn(a, p_b), 1.0f));
  }
  float g0 = __fmul_rn(fclip(__fmul_rn(attr, dx)), alpha);
  float g1 = __fmul_rn(fclip(__fmul_rn(attr, dy)), alpha);
  cur0 = __fadd_rn(cur0, g0);
  cur1 = __fadd_rn(cur1, g1);
  const float t0 = trunc_grad(rounding, -g0), t1 = trunc_grad(rounding, -g1);
  // both coordinates in one vector reduction (each element added
  // atomically, exactly as two scalar adds; rows are 8-byte aligned)
  atomicAdd(reinterpret_cast<float2 *>(op), make_float2(t0, t1));
  ns = __fadd_rn(ns, ep);
  // the samples' positions are read after the attraction, where the
  // reference reads them: by then the epoch's attraction updates are landing,
  // and the repulsion must see them (read at the start of the edge, they
  // give a measurably different layout); fetched together, one round trip
#pragma unroll
  for (int p = 0; p < kNegAhead; ++p)
    if (p < n_neg) qq[p] = ld_pos(emb + (size_t)rr[p] * 2);
  if (n_neg > 0) {
    const float two_gb = __fmul_rn(__fmul_rn(2.0f, gamma), b);
    const float a4 = __fmul_rn(4.0f, alpha);
    // one negative sample: repulsion from q, head moved in sequence
    auto negative = [&](int r, float q0, float q1) {
      if (r == j) return;
      const float ex = __fsub_rn(cur0, q0), ey = __fsub_rn(cur1, q1);
      const float d2n = __fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey));
      float rep = 0.0f;
      // repulsion: d2n^b by the hardware exp2 / log2 (__powf); these sampled
      // Hogwild updates are compared statistically, and the attraction
      // above keeps the series pow
      if (d2n > 0.0f)
        rep = __fdiv_rn(two_gb, __fmul_rn(__fadd_rn(0.001f, d2n),
                                          __fadd_rn(__fmul_rn(a, __powf(d2n, b)), 1.0f)));
      const float h0 = (rep > 0.0f) ? __fmul_rn(fclip(__fmul_rn(rep, ex)), alpha) : a4;
      const float h1 = (rep > 0.0f) ? __fmul_rn(fclip(__fmul_rn(rep, ey)), alpha) : a4;
      cur0 = __fadd_rn(cur0, h0);
      cur1 = __fadd_rn(cur1, h1);
      g0 = __fadd_rn(g0, h0);
      g1 = __fadd_rn(g1, h1);
    };
#pragma unroll
    for (int p = 0; p < kNegAhead; ++p) {
      if (p < n_neg) negative(rr[p], qq[p].x, qq[p].y);
    }
    if (n_neg > kNegAhead) {
      // draws past kNegAhead: the same stream from block 2 on
      Philox g;
      philox_init(g, seed, (uint32_t)row, kTagNegSample);
      g.block = kNegAhead / 4;
      for (int p = kNegAhead; p < n_neg; ++p) {
        const int r = (int)fastmod(philox_next(g), M, (uint32_t)n);
        const float2 q = ld_pos(emb + (size_t)r * 2);
        negative(r, q.x, q.y);
      }
    }
    nn = __fadd_rn(nn, __fmul_rn((float)n_neg, ep_neg));
    my_negs += (unsigned)n_neg;
  }
  atomicAdd(reinterpret_cast<float2 *>(cp),
            make_float2(trunc_grad(rounding, g0), trunc_grad(rounding, g1)));
}

// Edges [first, nnz) step stride of one epoch, state in global memory.
GM_D void sgd_epoch_edges(float *emb, const int *head, const int *tail, const float *eps,
                          float *next_s, float *next_n, int nnz, int n, uint64_t M,
                          float rounding, float alpha, int epoch, float gamma, float a, float b,
                          float nsr_inv, uint64_t seed, int first, int stride,
                          unsigned &my_edges, unsigned &my_negs) {
  const float fe = (float)epoch;
  for (int row = first; row < nnz; row += stride) {
    float ns = next_s[row];
    if (ns > fe) continue;
    float nn = next_n[row];
    sgd_edge(emb, row, head[row], tail[row], eps[row], ns, nn, n, M, rounding, alpha, fe, gamma, a,
             b, nsr_inv, seed, my_edges, my_negs);
    next_s[row] = ns;
    next_n[row] = nn;
  }
}

GM_D void sgd_stats(unsigned my_edges, unsigned my_negs, unsigned long long *stat) {
  if (!stat) return;
  for (int o = 16; o > 0; o >>= 1) {
    my_edges += __shfl_xor_sync(0xffffffffu, my_edges, o);
    my_negs += __shfl_xor_sync(0xffffffffu, my_negs, o);
  }
  if ((threadIdx.x & 31) == 0 && my_edges) {
    atomicAdd(&stat[7], (unsigned long long)my_edges);
    atomicAdd(&stat[8], (unsigned long long)my_negs);
  }
}

// One SGD epoch per launch.
__global__ void k_sgd_epoch(float *emb, const int *head, const int *tail,
                            const int *iscal, const float *eps, float *next_s,
                            float *next_n, float alpha, int epoch, float gamma, float a,
                            float b, float nsr_inv, uint64_t seed, const float *fscal,
                            unsigned long long *stat) {
  unsigned my_edges = 0, my_negs = 0;
  const int n = iscal[IS_N];
  const uint64_t M = ~0ull / (uint64_t)max(n, 1) + 1ull;
  sgd_epoch_edges(emb, head, tail, eps, next_s, next_n, iscal[IS_NNZ2], n, M,
                  fscal[FS_ROUND], alpha, epoch, gamma, a, b, nsr_inv, seed,
                  blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, my_edges,
                  my_negs);
  sgd_stats(my_edges, my_negs, stat);
}

// Grid-wide barrier of a co-resident (cooperative) grid on a monotonic
// arrival counter: the barrier after epoch e completes when the counter
// reaches (e + 1) * gridDim.x.  The wait is bounded; on timeout it records
// kDevErrSpin and returns false, and every block then leaves its epoch loop.
constexpr unsigned kBarrierSpinLimit = 1u << 24;
GM_D unsigned ld_acquire(const unsigned *p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// Arrival: the CTA's work for this epoch is done (bar.sync), made visible
// (fence) and counted.
GM_D void grid_arrive(unsigned *count) {
  __syncthreads();
  if (threadIdx.x == 0)
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
}
// Wait until every CTA has arrived (count >= target); bounded.
GM_D bool grid_wait(unsigned *count, unsigned target, unsigned *err) {
  __shared__ int s_ok;
  if (threadIdx.x == 0) {
    int ok = 1;
    unsigned it = 0;
    while (ld_acquire(count) < target) {
      if (++it > kBarrierSpinLimit) {
        ok = 0;
        atomicOr(err, kDevErrSpin);
        break;
      }
      __nanosleep(16);
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// All epochs in one cooperative launch, a grid barrier between epochs (the
// reference's kernel boundary): learning rate and seed advance exactly as the
// host loop of the per-epoch form.  A thread's first kRegEdges edges keep
// their indices and sampling clocks in registers for the whole call, the next
// `held` in shared memory, and only the rest
// goes to global memory: with every later edge there, each of a thread's turns
// began with the round trip of its clock.  The order of the turns, which the
// Hogwild updates depend on, is the same.  20,000 rows (480k edges, 7 turns a
// thread), 200 epochs: 5.53 -> 5.2 ms.
constexpr int kRegEdges = 2;
constexpr int kSgdThreads = 512;
constexpr int kSgdTurnBytes = 20 * kSgdThreads;                  // shared memory of one turn
constexpr int kSgdMaxHeld = (227 * 1024 - 64) / kSgdTurnBytes;
// kHeld: the schedule may take more turns than the registers hold.
template <bool kHeld>
__global__ void __launch_bounds__(kSgdThreads)
    k_sgd_persistent(float *emb, const int *head, const int *tail, const int *iscal,
                     const float *eps, float *next_s, float *next_n, float alpha0, int n_epochs,
                     float gamma, float a, float b, float nsr_inv, uint64_t seed,
                     const float *fscal, unsigned *bar, unsigned *err, int held,
                     unsigned long long *stat) {
  extern __shared__ __align__(16) unsigned char sgd_raw[];
  // this thread's five words of turn t: t * 5 * kSgdThreads, a row apart
  float *held_at = reinterpret_cast<float *>(sgd_raw) + threadIdx.x;
  enum { kNs = 0, kNn = kSgdThreads, kEps = 2 * kSgdThreads, kHead = 3 * kSgdThreads, kTail = 4 * kSgdThreads };
  const int nnz = iscal[IS_NNZ2], n = iscal[IS_N];
  const uint64_t M = ~0ull / (uint64_t)max(n, 1) + 1ull;
  const float rounding = fscal[FS_ROUND];
  unsigned my_edges = 0, my_negs = 0;
  // slot i of the grid handles edge i, in the schedule's order (a head's
  // edges in adjacent lanes, as in the reference's one-thread-per-edge
  // epochs).  Warp-sized runs of slots are dealt round-robin over the CTAs
  // (run w to CTA w mod gridDim.x), so the active edges spread over every SM
  // instead of filling the first few; the map from (CTA, thread) to slot is
  // a bijection on [0, gridDim.x * blockDim.x).
  const int first = (((int)threadIdx.x >> 5) * (int)gridDim.x + (int)blockIdx.x) * 32 + ((int)threadIdx.x & 31);
  const int stride = gridDim.x * blockDim.x;
  int rrow[kRegEdges], rj[kRegEdges], rk[kRegEdges];
  float rep[kRegEdges], rns[kRegEdges], rnn[kRegEdges];
#pragma unroll
  for (int t = 0; t < kRegEdges; ++t) {
    const int slot = first + t * stride;
    if (slot < nnz) {
      const int row = slot;
      rrow[t] = row;
      rj[t] = head[row], rk[t] = tail[row], rep[t] = eps[row];
      rns[t] = next_s[row], rnn[t] = next_n[row];
    }
  }
  // turns past the registers, the first `held` of them in shared memory
  int turns = 0;
  for (int row = first + kRegEdges * stride; kHeld && row < nnz; row += stride) {
    if (turns < held) {
      float *w = held_at + turns * 5 * kSgdThreads;
      w[kNs] = next_s[row], w[kNn] = next_n[row], w[kEps] = eps[row];
      w[kHead] = __int_as_float(head[row]), w[kTail] = __int_as_float(tail[row]);
    }
    ++turns;
  }
  float alpha = alpha0;
  for (int ep = 0; ep < n_epochs; ++ep) {
    const float fe = (float)ep;
    const uint64_t sd = seed + (uint64_t)ep;
#pragma unroll
    for (int t = 0; t < kRegEdges; ++t) {
      if (first + t * stride < nnz && rns[t] <= fe)
        sgd_edge(emb, rrow[t], rj[t], rk[t], rep[t], rns[t], rnn[t], n, M, rounding, alpha, fe,
                 gamma, a, b, nsr_inv, sd, my_edges, my_negs);
    }
    for (int t = 0; kHeld && t < turns; ++t) {
      const int row = first + (kRegEdges + t) * stride;
      float *w = held_at + t * 5 * kSgdThreads;
      const bool in = t < held;
      float ns = in ? w[kNs] : next_s[row];
      if (ns > fe) continue;
      float nn = in ? w[kNn] : next_n[row];
      sgd_edge(emb, row, in ? __float_as_int(w[kHead]) : head[row],
               in ? __float_as_int(w[kTail]) : tail[row], in ? w[kEps] : eps[row], ns, nn, n, M, rounding,
               alpha, fe, gamma, a, b, nsr_inv, sd, my_edges, my_negs);
      (in ? w[kNs] : next_s[row]) = ns;
      (in ? w[kNn] : next_n[row]) = nn;
    }
    alpha = __fmul_rn(alpha0, __fsub_rn(1.0f, __fdiv_rn((float)ep, (float)n_epochs)));
    if (ep + 1 < n_epochs) {
      grid_arrive(bar);
      if (!grid_wait(bar, (unsigned)(ep + 1) * gridDim.x, err)) break;
    }
  }
  sgd_stats(my_edges, my_negs, stat);
}

__global__ void k_epoch_init(const float *eps, int nnz, float nsr_inv, float *next_s,
                             float *next_n) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nnz) return;
  next_s[q] = eps[q];
  next_n[q] = __fmul_rn(eps[q], nsr_inv);
}

// x-range of the embedding (first component) for the noise scale.
__global__ void k_xrange_partial(const float *emb, int n, float *part) {
  pdl_enter();
  __shared__ float smin[256], smax[256];
  const int t = threadIdx.x;
  float mn = FLT_MAX, mx = -FLT_MAX;
  for (int i = blockIdx.x * 256 + t; i < n; i += gridDim.x * 256) {
    const float v = emb[(size_t)i * 2];
    mn = fminf(mn, v);
    mx = fmaxf(mx, v);
  }
  smin[t] = mn;
  smax[t] = mx;
  __syncthreads();
  for (int s = 128; s > 0; s >>= 1) {
    if (t < s) {
      smin[t] = fminf(smin[t], smin[t + s]);
      smax[t] = fmaxf(smax[t], smax[t + s]);
    }
    __syncthreads();
  }
  if (t == 0) {
    part[2 * blockIdx.x] = smin[0];
    part[2 * blockIdx.x + 1] = smax[0];
  }
}

// The noise scale from the partial ranges (at most 256, one per thread), then
// two components per batch row.
__global__ void __launch_bounds__(256)
    k_add_noise(float *emb, const int *batch, int nb, const float *part, int nparts,
                float noise_scale, uint64_t seed) {
  pdl_enter();
  __shared__ float s_mn[8], s_mx[8];
  const int t = threadIdx.x, tid = blockIdx.x * blockDim.x + t;
  float mn = FLT_MAX, mx = -FLT_MAX;
  if (t < nparts) {
    mn = part[2 * t];
    mx = part[2 * t + 1];
  }
  float *p = nullptr;
  float z = 0.0f;
  if (tid < nb * 2) {
    p = emb + (size_t)batch[tid >> 1] * 2 + (tid & 1);
    Philox g;
    philox_init(g, seed, (uint32_t)tid, kTagNoise);
    z = gm_normal(g);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if ((t & 31) == 0) {
    s_mn[t >> 5] = mn;
    s_mx[t >> 5] = mx;
  }
  __syncthreads();
  if (!p) return;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    mn = fminf(mn, s_mn[w]);
    mx = fmaxf(mx, s_mx[w]);
  }
  *p = __fadd_rn(*p, __fmul_rn(z, __fmul_rn(noise_scale, __fsub_rn(mx, mn))));
}

// Rows not selected this round move to the membership-weighted mean of their
// neighbours' positions, read from a snapshot (reference :811-894).  Ids
// outside [0, n) are skipped.  A thread per row, kHeurAhead neighbours at a
// time: their ids and distances, then their positions, are on their way
// together (one after another they made the kernel's latency: 13 us for 70,000
// rows at k = 15, this form 9.7 us).
constexpr int kHeurAhead = 8;
__global__ void k_heuristic(const uint32_t *pub_idx, const float *pub_dist, int n, int k,
                            int euclid, const float *sigma, const float *rho,
                            const int *unsel, int nu, const float *snap, float *emb) {
  pdl_enter();
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nu) return;
  const int row = unsel[q];
  const float sg = sigma[row], rh = rho[row];
  float wsum = 0.0f, a0 = 0.0f, a1 = 0.0f;
  // (column 0 is the row itself)
  for (int k0 = 1; k0 < k; k0 += kHeurAhead) {
    int col[kHeurAhead];
    float dist[kHeurAhead];
    float2 pos[kHeurAhead];
#pragma unroll
    for (int i = 0; i < kHeurAhead; ++i) {
      const bool in = k0 + i < k;
      col[i] = in ? (int)eidx(pub_idx, k, row, k0 + i) : row;
      dist[i] = in ? edist(pub_dist, k, row, k0 + i, euclid) : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < kHeurAhead; ++i) {
      if (col[i] == row || !valid_d(dist[i]) || col[i] < 0 || col[i] >= n) col[i] = -1;
      pos[i] = col[i] >= 0 ? *reinterpret_cast<const float2 *>(snap + (size_t)col[i] * 2)
                           : make_float2(0.0f, 0.0f);
    }
#pragma unroll
    for (int i = 0; i < kHeurAhead; ++i) {
      if (col[i] < 0) continue;
      const float w = membership(dist[i], rh, sg);
      wsum = __fadd_rn(wsum, w);
      a0 = __fmaf_rn(w, pos[i].x, a0);
      a1 = __fmaf_rn(w, pos[i].y, a1);
    }
  }
  if (wsum > 0.0f) {
    emb[(size_t)row * 2] = __fdiv_rn(a0, wsum);
    emb[(size_t)row * 2 + 1] = __fdiv_rn(a1, wsum);
  }
}

__global__ void k_mark_rows(const int *rows, int nr, int *flag) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < nr) flag[rows[i]] = 1;
}

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

}  // namespace

void launch_mark_rows(const int *rows, int nr, int *flag, cudaStream_t s) {
  if (nr <= 0) return;
  launch(k_mark_rows, cdiv(nr, 256), 256, 0, s, rows, nr, flag);
  note_launch();
}

void launch_fuzzy_graph(const uint32_t *pub_idx, const float *pub_dist, int n, int k,
                        int euclidean, const int *batch, int nb, double log2_target,
                        EmbedScratch &e, cudaStream_t s) {
  const long total = (long)n * k;
  const int nbl = cdiv(total, 256);
  launch(k_mean_partial, nbl, 256, 0, s, pub_dist, n, k, euclidean, e.partial, e.ipartial, e.deg, e.iscal,
         e.fscal);
  note_launch();
  const float t_hi = (float)log2_target, t_lo = (float)(log2_target - (double)t_hi);
  auto smooth = [&](auto kernel, int lanes) {
    launch(kernel, 1 + cdiv((long)n * lanes, kSmoothThreads), kSmoothThreads, 0, s, pub_dist, n, k,
           euclidean, log2_target, t_hi, isfinite(log2_target) ? t_lo : 0.0f, e.sigma, e.rho, e.partial,
           e.ipartial, nbl, e.fscal, e.iscal + IS_MARKED);
  };
  if (k <= 16) smooth(k_smooth_knn<4>, 4);
  else smooth(k_smooth_knn<8>, 8);
  launch(k_fix_sigma, cdiv(n, 256), 256, 0, s, n, e.fscal, e.sigma, e.iscal + IS_MARKED);
  note_launch(2);
  const int ndir = nb * k;
  if (ndir > 0) {
    launch(k_memb_sym, cdiv(ndir, 256), 256, 0, s, pub_idx, pub_dist, n, k,
           euclidean, e.sigma, e.rho, batch, nb, e.coo_row, e.coo_col, e.coo_val, e.t_row, e.fscal);
    note_launch();
  }
  compact_flags(e.t_row, ndir, -1, e.t_col, e.iscal + IS_EXTRA, e.tmp2, s);
  launch(k_write_extras, cdiv(ndir > 0 ? ndir : 1, 256), 256, 0, s, e.t_col, e.iscal + IS_EXTRA, ndir,
         e.coo_row, e.coo_col, e.coo_val, e.iscal);
  note_launch();
}

void launch_schedule(int n, int nb, int k, float alpha0, int n_epochs, int neg_rate,
                     EmbedScratch &e, cudaStream_t s) {
  if (n <= 0 || n_epochs <= 0 || nb <= 0) {
    cudaMemsetAsync(e.iscal + IS_NNZ2, 0, sizeof(int), s);
    return;
  }
  const int nmax = 2 * nb * k;
  // keep w >= max_w / n_epochs (reference trim_graph, :348-400)
  compact_at_least(e.coo_val, e.fscal + FS_MAXW, n_epochs, e.iscal + IS_NNZ, nmax, e.t_col, e.iscal + IS_NNZ2,
                   e.tmp2, s);
  // t_col holds survivor indices; gather into (t_row, flag_tail, t_val)
  const float nsr_inv = 1.0f / (float)neg_rate;  // inf when 0: no negatives
  launch(k_gather_sched, cdiv(nmax, 256 * kGatherAhead), 256, 0, s, e.t_col, e.iscal, e.coo_row, e.coo_col, e.coo_val,
         e.fscal, n_epochs, nsr_inv, e.t_row, e.flag_tail, e.t_val, e.next_s, e.next_n, e.deg);
  note_launch();
  launch(k_rounding, 1, 1, 0, s, e.iscal, e.fscal, alpha0, n);
  note_launch();
}

void launch_epoch_init(const float *eps, int nnz, int neg_rate, float *next_s,
                       float *next_n, cudaStream_t s) {
  if (nnz <= 0) return;
  k_epoch_init<<<cdiv(nnz, 256), 256, 0, s>>>(eps, nnz, 1.0f / (float)neg_rate, next_s,
                                              next_n);
  note_launch();
}

void launch_sgd(float *emb, const int *head, const int *tail, const float *eps,
                float *next_s, float *next_n, const int *iscal, const float *fscal,
                int grid, float alpha0, float gamma, float a, float b, int n_epochs,
                int neg_rate, uint64_t seed, cudaStream_t s, unsigned long long *stat) {
  if (n_epochs <= 0 || grid <= 0) return;
  const float nsr_inv = 1.0f / (float)neg_rate;
  float alpha = alpha0;
  uint64_t cur_seed = seed;
  for (int ep = 0; ep < n_epochs; ++ep) {
    k_sgd_epoch<<<grid, 256, 0, s>>>(emb, head, tail, iscal, eps, next_s, next_n, alpha, ep,
                                     gamma, a, b, nsr_inv, cur_seed, fscal, stat);
    note_launch();
    // alpha and seed for the next epoch (reference embedding_kernel.cuh:790-792)
    alpha = alpha0 * (1.0f - (float)ep / (float)n_epochs);
    cur_seed += 1;
  }
}

int sgd_persistent_grid(int device) {
  // per device, once (sessions on several host threads may launch at once)
  static std::mutex mu;
  static int grid[64] = {0};
  if (device < 0 || device >= 64) return 0;
  std::lock_guard<std::mutex> g(mu);
  if (!grid[device]) {
    int sms = 0, occ = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_sgd_persistent<false>, kSgdThreads, 0);
    cudaFuncSetAttribute(k_sgd_persistent<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         kSgdMaxHeld * kSgdTurnBytes);
    grid[device] = std::max(1, sms) * std::max(1, std::min(occ, 1));
  }
  return grid[device];
}

cudaError_t launch_sgd_persistent(float *emb, const int *head, const int *tail,
                                  const float *eps, float *next_s, float *next_n,
                                  const int *iscal, const float *fscal, int max_edges, float alpha0,
                                  float gamma, float a, float b, int n_epochs, int neg_rate,
                                  uint64_t seed, unsigned *bar, unsigned *err, int device,
                                  cudaStream_t s, unsigned long long *stat, int max_ctas) {
  if (n_epochs <= 0) return cudaSuccess;
  int grid = sgd_persistent_grid(device);
  if (max_ctas > 0) grid = std::min(grid, max_ctas);
  if (grid <= 0) return cudaErrorInvalidDevice;
  cudaError_t e = cudaMemsetAsync(bar, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return e;
  float nsr_inv = 1.0f / (float)neg_rate;
  const int turns = cdiv(max_edges, (long)grid * kSgdThreads) - kRegEdges;
  int held = std::min(kSgdMaxHeld, std::max(0, turns));
  void *args[] = {&emb, &head, &tail, &iscal, &eps, &next_s, &next_n, &alpha0, &n_epochs,
                  &gamma, &a, &b, &nsr_inv, &seed, &fscal, &bar, &err, &held, &stat};
  e = cudaLaunchCooperativeKernel(turns > 0 ? (const void *)k_sgd_persistent<true>
                                            : (const void *)k_sgd_persistent<false>, dim3(grid), dim3(kSgdThreads),
                                  args, (size_t)held * kSgdTurnBytes, s);
  note_launch();
  return e;
}

void launch_add_noise(float *emb, int n, const int *batch, int nb, float noise_scale,
                      uint64_t seed, EmbedScratch &e, cudaStream_t s) {
  if (nb <= 0 || noise_scale == 0.0f || n <= 0) return;
  const int nparts = min(cdiv(n, 256), 256);
  launch(k_xrange_partial, nparts, 256, 0, s, emb, n, e.partial);
  note_launch();
  launch(k_add_noise, cdiv(nb * 2, 256), 256, 0, s, emb, batch, nb, e.partial, nparts, noise_scale, seed);
  note_launch();
}

void launch_heuristic(const uint32_t *pub_idx, const float *pub_dist, int n, int k,
                      int euclidean, const int *unsel, int nu, float *emb,
                      EmbedScratch &e, cudaStream_t s) {
  if (nu <= 0 || n <= 0 || k <= 0) return;
  cudaMemcpyAsync(e.snap, emb, sizeof(float) * 2 * (size_t)n, cudaMemcpyDeviceToDevice, s);
  launch(k_heuristic, cdiv(nu, 128), 128, 0, s, pub_idx, pub_dist, n, k, euclidean, e.sigma, e.rho, unsel,
         nu, e.snap, emb);
  note_launch();
}

}  // namespace gm
