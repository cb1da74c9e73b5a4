// Insertion phase: NN-Descent insertion of a contiguous batch of new rows.
// Restates the reference's insertion_kernel.cuh (run_insertion, :926-1095)
// with a deterministic reverse step and a canonical FP32 distance.
#include <algorithm>
#include <climits>

#include "gm_common.cuh"
#include "gm_kernels.h"
#include "gm_rowdot.cuh"

namespace gm {

namespace {

// ||x||^2 for each batch row by a sequential fma chain over the features, and
// its square root rounded up (snorms).  Cosine: the row is normalised in place
// afterwards and its norm is 1.0 (reference: preprocess_l2_norms_kernel,
// insertion_kernel.cuh:31-81).  kNormRows rows per CTA, staged in shared memory
// a chunk of up to kNormChunk features at a time (16-byte cp.async by all
// threads: rows are 16-byte aligned, ld a multiple of 4); lanes 0..kNormRows-1
// of warp 0 run the chains, four features a read (the padding is zero, which
// adds nothing).  Bound by the chain, 1.6 us for
// 784 features: 500 rows x 784 took 9.2 us with a read per feature and a row's
// loads waiting for the row's before, 6.2 us so.
constexpr int kNormRows = 4, kNormChunk = 1024;
__global__ void __launch_bounds__(256)
    k_row_norms(float *X, float *norms, float *snorms, int ld, int d, int row0, int nrows,
                int cosine) {
  pdl_enter();
  __shared__ __align__(16) float tile[kNormRows][kNormChunk + 4];
  __shared__ float s_scale[kNormRows];
  const int r0 = blockIdx.x * kNormRows;
  const int rows = min(kNormRows, nrows - r0);
  const int tid = threadIdx.x, lane = tid & 31;
  float acc = 0.0f;
  for (int c0 = 0; c0 < d; c0 += kNormChunk) {
    const int w = min(kNormChunk, d - c0);
    const int w4 = (w + 3) >> 2;  // float4 columns (the row padding is zero)
    for (int c = tid; c < w4; c += blockDim.x)
#pragma unroll
      for (int r = 0; r < kNormRows; ++r)
        if (r < rows) dot_cp16(&tile[r][4 * c], X + (size_t)(row0 + r0 + r) * ld + c0 + 4 * c);
    dot_commit();
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    if (tid < rows) {
#pragma unroll 8
      for (int c = 0; c < w4; ++c) {
        const float4 v = *reinterpret_cast<const float4 *>(&tile[lane][4 * c]);
        acc = __fmaf_rn(v.x, v.x, acc);
        acc = __fmaf_rn(v.y, v.y, acc);
        acc = __fmaf_rn(v.z, v.z, acc);
        acc = __fmaf_rn(v.w, v.w, acc);
      }
    }
    __syncthreads();
  }
  if (tid < rows) {
    const size_t row = (size_t)(row0 + r0 + lane);
    float nv = acc;
    s_scale[lane] = 0.0f;
    if (cosine) {
      s_scale[lane] = __fsqrt_rn(acc);
      nv = 1.0f;
    }
    norms[row] = nv;
    snorms[row] = __fsqrt_ru(nv);
  }
  __syncthreads();
  if (cosine) {
    for (int r = 0; r < rows; ++r) {
      const float nrm = s_scale[r];
      if (!(nrm > 0.0f)) continue;
      float *x = X + (size_t)(row0 + r0 + r) * ld;
      for (int c = tid; c < d; c += blockDim.x) x[c] = __fdiv_rn(x[c], nrm);
    }
  }
}

// Random unique initial neighbours: up to 16 from the recent window
// [window_start, n), the rest from [0, n); distances FLT_MAX
// (reference: initialize_random_neighbors_kernel, insertion_kernel.cuh:170-248).
// A warp per row tests 32 draws of the row's Philox stream at once: a draw is
// taken when it is not the row, not yet listed and the first of its value
// among the 32, in draw order, and the stream stops at the draw that fills the
// phase, so the list is that of one draw at a time.  Bound by latency: one
// thread per row took 32 us for 500 rows on 4 of 152 SMs, this form under 6 us.
constexpr int kInitWarps = 4;
__global__ void __launch_bounds__(kInitWarps * 32)
    k_random_init(Key *g_key, int row0, int nrows, int n, int window_start, uint64_t seed) {
  pdl_enter();
  __shared__ int s_list[kInitWarps][kListW];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rl = blockIdx.x * kInitWarps + warp;
  if (rl >= nrows) return;
  const int gid = row0 + rl;
  int *lst = s_list[warp];
  int f = 0;
  uint32_t t = 0;  // draws consumed
  // takes the lanes' values c where ok, first come first, until `limit` are
  // listed; returns the number of lanes consumed
  auto take = [&](int c, bool ok, int lanes, int limit) {
    for (int q = 0; q < f; ++q) ok &= lst[q] != c;
    const unsigned same = __match_any_sync(0xffffffffu, ok ? c : -1 - lane);
    ok &= (__ffs(same) - 1) == lane;
    const unsigned bal = __ballot_sync(0xffffffffu, ok);
    const int rank = __popc(bal & ((1u << lane) - 1u)), need = limit - f;
    const bool mine = ok && rank < need;
    if (mine) lst[f + rank] = c;
    const unsigned last = __ballot_sync(0xffffffffu, mine && rank == need - 1);
    f += min(need, __popc(bal));
    __syncwarp();
    return last ? __ffs(last) : lanes;
  };
  auto draws = [&](int lo, int size, int limit, uint32_t max_att) {
    uint32_t att = 0;
    while (f < limit && att < max_att) {
      const int lanes = (int)min(32u, max_att - att);
      uint32_t w[4];
      const uint32_t at = t + (uint32_t)lane;
      philox_block((uint32_t)gid, at >> 2, kTagInitNeighbors, 0u, (uint32_t)seed,
                   (uint32_t)(seed >> 32), w);
      const uint32_t m = at & 3u;
      const uint32_t v = m == 0 ? w[0] : m == 1 ? w[1] : m == 2 ? w[2] : w[3];
      const int c = lo + (int)(v % (uint32_t)size);
      const int used = take(c, lane < lanes && c != gid, lanes, limit);
      t += (uint32_t)used;
      att += (uint32_t)used;
    }
  };
  if (n > 1) {
    const int max_fill = min(kListW, n - 1);
    const int wsize = n - window_start;
    const int wquota = min(kListW / 2, max(0, wsize - 1));
    draws(window_start, wsize, wquota, (uint32_t)wquota * 16u);
    // Full-range phase; bounded, then a deterministic sweep as a fallback.
    draws(0, n, max_fill, 1u << 20);
    for (int c0 = 0; f < max_fill && c0 < n; c0 += 32)
      take(c0 + lane, c0 + lane < n && c0 + lane != gid, 32, max_fill);
  }
  g_key[(size_t)gid * kListW + lane] = lane < f ? make_key(FLT_MAX, lst[lane]) : kEmptyKey;
}

// Two-hop candidates, one warp per batch row.  Position p = kk*k + j visits
// slot kk of neighbour j (round robin); a position is kept if its id is in
// range, not self, not a current neighbour and its first occurrence; the
// first 256 kept positions in order are the candidates
// (reference: sample_forward_candidates_kernel, insertion_kernel.cuh:250-321).
// First occurrences come from a shared-memory hash table of the ids (linear
// probing) that keeps each id's smallest position; the row's own neighbours are
// entered at position -1.  Positions are taken kHopBlock slots of every
// neighbour at a time, in order, and the rest is left unread once 256 are
// kept, so the table holds at most k + 256 + kHopBlock k ids, whatever k is.
// Candidates of the previous iteration keep the distance they have (and were
// offered then); only the others are listed in todo, by slot.
// Comparing every position with every earlier one was O(k^4): 36 us for 500
// rows at k = 15 and 606 us for 10,000 at k = 30; this form 10 us and 70 us (142 us
// with every position read).
// exist_only: only candidates below row0 are written (see launch_nnd_insert).
constexpr int kSampWarps = 4;
constexpr int kHopBlock = 8;
GM_HD int hop_slots(int k) {  // hash slots: a power of two, at most two thirds full
  int h = 32;
  while (h < 1024 && h < k * k + k + (k * k + k) / 2) h *= 2;
  return h;
}
static_assert(kListW + kMaxCand + kHopBlock * kListW <= 2 * 1024 / 3, "hash table too full");
static_assert(kSampWarps * (2 * 1024 + kListW + kHopBlock * kListW + kMaxCand / 32) * 4 <= 48 * 1024,
              "shared memory");
// table ids, table positions, neighbours, the block's slots, known candidates
GM_HD size_t hop_ints(int k) {
  return (size_t)2 * hop_slots(k) + kListW + kHopBlock * kListW + kMaxCand / 32;
}
struct HopOut {
  int *cand;        // 256 per row
  int *cnt;         // per row
  float *dist;      // 256 per row: known distances are written
  uint8_t *todo;    // 256 per row: slots without a known distance (null: all)
  int *todo_cnt;    // per row
};
__global__ void __launch_bounds__(kSampWarps * 32)
    k_sample_candidates(const Key *g_key, int row0, int nrows, int n, int k, int slots,
                        int exist_only, HopOut o, int iter, const int *changed) {
  pdl_enter();
  if (changed && *changed == 0) return;
  extern __shared__ __align__(16) int smem_sc[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rl = blockIdx.x * kSampWarps + warp;
  if (rl >= nrows) return;
  int *hid = smem_sc + (size_t)warp * hop_ints(k);
  int *hpos = hid + slots;
  int *nb = hpos + slots;
  int *at = nb + kListW;  // the block's positions -> table slot (-1: none)
  unsigned *known = reinterpret_cast<unsigned *>(at + kHopBlock * kListW);
  const int gid = row0 + rl;
  int *out = o.cand + (size_t)rl * kMaxCand;
  float *dist = o.dist + (size_t)rl * kMaxCand;
  // the previous iteration's candidates
  int pid[kMaxCand / 32];
  float pd[kMaxCand / 32];
  const bool reuse = o.todo && iter > 0;
  if (reuse) {
    const int pc = o.cnt[rl];
#pragma unroll
    for (int c = 0; c < kMaxCand / 32; ++c) {
      const int i = c * 32 + lane;
      pid[c] = i < pc ? out[i] : -1;
      pd[c] = i < pc ? dist[i] : 0.0f;
    }
  }
  const int mine = key_id(g_key[(size_t)gid * kListW + lane]);
  nb[lane] = (lane < k && mine >= 0 && mine < n) ? mine : kIdSentinel;
  if (lane < kMaxCand / 32) known[lane] = 0u;
  for (int i = lane * 4; i < slots; i += 128) {
    *reinterpret_cast<int4 *>(hid + i) = make_int4(-1, -1, -1, -1);
    *reinterpret_cast<int4 *>(hpos + i) = make_int4(INT_MAX, INT_MAX, INT_MAX, INT_MAX);
  }
  __syncwarp();
  const unsigned mask = (unsigned)slots - 1u;
  auto first_slot = [&](int id) { return ((unsigned)id * 2654435761u >> 10) & mask; };
  auto enter = [&](int id, int pos) {
    unsigned h = first_slot(id);
    for (;;) {
      const int old = atomicCAS(&hid[h], -1, id);
      if (old == -1 || old == id) break;
      h = (h + 1u) & mask;
    }
    atomicMin(&hpos[h], pos);
    return (int)h;
  };
  if (nb[lane] != kIdSentinel) enter(nb[lane], -1);
  __syncwarp();
  // lane: slot kb + lane % 8 of neighbours lane / 8, lane / 8 + 4, ...
  constexpr int kSpan = 32 / kHopBlock, kAhead = kListW / kSpan;
  const int sub = lane % kHopBlock;
  int base = 0;
  for (int kb = 0; kb < k && base < kMaxCand; kb += kHopBlock) {
    const int kk = kb + sub;
    int e[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int j = lane / kHopBlock + u * kSpan;
      const int nbr = (j < k && kk < k) ? nb[j] : kIdSentinel;
      e[u] = nbr != kIdSentinel ? key_id(g_key[(size_t)nbr * kListW + kk]) : -1;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int j = lane / kHopBlock + u * kSpan;
      if (j < k && kk < k)
        at[sub * k + j] = ((uint32_t)e[u] < (uint32_t)n && e[u] != gid) ? enter(e[u], kk * k + j) : -1;
    }
    __syncwarp();
    const int p_end = min(kHopBlock, k - kb) * k;
    for (int p0 = 0; p0 < p_end && base < kMaxCand; p0 += 32) {
      const int p = p0 + lane;
      const int sl = p < p_end ? at[p] : -1;
      const int id = sl >= 0 ? hid[sl] : -1;
      const bool keep = sl >= 0 && hpos[sl] == kb * k + p && !(exist_only && id >= row0);
      const unsigned bal = __ballot_sync(0xffffffffu, keep);
      const int idx = base + __popc(bal & ((1u << lane) - 1u));
      if (keep && idx < kMaxCand) {
        out[idx] = id;
        hpos[sl] = -2 - idx;  // below every position: later entries change nothing
      }
      base += __popc(bal);
    }
    __syncwarp();
  }
  const int cnt = min(base, kMaxCand);
  if (lane == 0) o.cnt[rl] = cnt;
  if (!o.todo) return;
  if (reuse) {
#pragma unroll
    for (int c = 0; c < kMaxCand / 32; ++c) {
      if (pid[c] < 0) continue;
      unsigned h = first_slot(pid[c]);
      while (hid[h] != -1 && hid[h] != pid[c]) h = (h + 1u) & mask;
      const int idx = hid[h] == pid[c] ? -2 - hpos[h] : -1;
      if (idx >= 0) {
        dist[idx] = pd[c];
        atomicOr(&known[idx >> 5], 1u << (idx & 31));
      }
    }
    __syncwarp();
  }
  int left = 0;
  for (int c = 0; c * 32 < cnt; ++c) {
    const bool open = c * 32 + lane < cnt && !((known[c] >> lane) & 1u);
    const unsigned bal = __ballot_sync(0xffffffffu, open);
    if (open)
      o.todo[(size_t)rl * kMaxCand + left + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)(c * 32 + lane);
    left += __popc(bal);
  }
  if (lane == 0) o.todo_cnt[rl] = left;
}

// Candidate distances and, for existing candidates (id < row0), the reverse
// offers (reference: compute_candidate_distances_kernel,
// insertion_kernel.cuh:337-405, and :548-640, which scatters up to 32
// arrivals per row; here every one is kept, one of the reference's outcomes).
// A warp takes (row, chunk of 32 candidates) tasks in a grid stride: 32
// canonical chains (gm_rowdot.cuh), then each offer below its target's last
// entry is put on one of the target's chains.  todo (null: every candidate)
// lists the slots to do.
// Bound by L2: a row's candidates are 100-200 feature rows.  An insertion of
// 500 rows x 784 features at k = 15 took 1.35 ms over its ten iterations with
// a CTA per row, two barriers per chunk and every offer merged under its
// target's lock; 0.36 ms with one iteration of this form but the locks (the
// recent window's rows get most of the offers); 0.05 ms with the chains, their merge
// included.
constexpr int kCandWarps = 2;
__global__ void __launch_bounds__(kCandWarps * 32)
    k_candidate_offers(const float *X, const float *norms, int ld, int row0, int first, int nrows, int chunks,
                       const int *cand, const uint8_t *todo, const int *todo_cnt,
                       float *cand_dist, const Key *g_key, OfferChains chains, const int *changed,
                       unsigned long long *stat) {
  pdl_enter();
  if (changed && *changed == 0) return;
  __shared__ __align__(16) RowDotTiles tiles[kCandWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tasks = nrows * chunks;
  for (int task = blockIdx.x * kCandWarps + warp; task < tasks; task += gridDim.x * kCandWarps) {
    const int rl = task / chunks, i = (task - rl * chunks) * 32 + lane;
    const int cnt = todo_cnt[rl];
    if (i - lane >= cnt) continue;
    const int gid = first + rl;
    const size_t e = (size_t)rl * kMaxCand + (i < cnt && todo ? todo[(size_t)rl * kMaxCand + i] : i);
    const int j = i < cnt ? cand[e] : gid;
    if (stat && lane == 0) atomicAdd(&stat[4], (unsigned long long)(min(32, cnt - i) + (i == 0)));
    const float dot = warp_row_dot(X, ld, X + (size_t)gid * ld, j, tiles[warp]);
    const float dv = canon_dist(norms[gid], norms[j], dot);
    if (i < cnt) {
      cand_dist[e] = dv;
      if (j < row0 && dv >= 0.0f && make_key(dv, gid) < g_key[(size_t)j * kListW + kListW - 1])
        chains.next[e] = atomicExch(&chains.heads[(size_t)j * 32 + (gid & 31)], (int)e);
    }
  }
}

// Merges the offers on each existing row's chains into its list, a warp per
// row, a chain per lane, without a lock: no other warp of this launch touches
// the row.  The order of offers does not matter (warp_insert).
constexpr int kOfferWarps = 8;
__global__ void __launch_bounds__(kOfferWarps * 32)
    k_merge_offers(Key *g_key, int row0, int first, OfferChains chains, const float *dist,
                   const int *e_row, int *dirty, int *changed_out, const int *changed) {
  pdl_enter();
  if (changed && *changed == 0) return;
  const int lane = threadIdx.x & 31;
  const int j = blockIdx.x * kOfferWarps + (threadIdx.x >> 5);
  if (j >= row0) return;
  const unsigned full = 0xffffffffu;
  int e = chains.heads[(size_t)j * 32 + lane];
  if (!__any_sync(full, e >= 0)) return;
  chains.heads[(size_t)j * 32 + lane] = -1;
  Key *row = g_key + (size_t)j * kListW;
  Key mine = row[lane];
  bool moved = false;
  while (__any_sync(full, e >= 0)) {
    Key ck = ~(Key)0;
    if (e >= 0) {
      ck = make_key(dist[e], first + (e_row ? e_row[e] : e / kMaxCand));
      e = chains.next[e];
    }
    unsigned todo = __ballot_sync(full, ck < __shfl_sync(full, mine, kListW - 1));
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1u;
      moved |= warp_insert(mine, __shfl_sync(full, ck, src)) < kListW;
    }
  }
  if (!moved) return;
  row[lane] = mine;
  if (lane == 0) {
    dirty[j] = 1;
    if (changed_out) *changed_out = 1;
  }
}

// Forward merge of a batch row's candidates into its own list, a warp per
// row.  The reference sorts all 256 slots with -1 sentinels first and stops
// at the first sentinel (insertion_kernel.cuh:407-534), so the merge only
// takes effect when all 256 slots hold valid candidates; that rule is kept.
// Both of its sequential insertion sorts (the 32 best candidates, skipping
// ties with the tail; then those into the list) run one element at a time,
// each scan from the tail as one ballot: lane q holds entry q, and the place
// is after the last entry the element does not precede.  One thread per row
// took 468 us for 10,000 rows at k = 30, this form 52 us.
constexpr int kFwdWarps = 4;
__global__ void __launch_bounds__(kFwdWarps * 32)
    k_forward_merge(Key *g_key, int row0, int nrows, const int *cand, const int *cand_cnt,
                    const float *cand_dist, int *changed_out, const int *changed) {
  pdl_enter();
  if (changed && *changed == 0) return;
  const int lane = threadIdx.x & 31;
  const int rl = blockIdx.x * kFwdWarps + (threadIdx.x >> 5);
  if (rl >= nrows || cand_cnt[rl] < kMaxCand) return;
  const unsigned full = 0xffffffffu;
  // entry insertion among entries [0, lim), shifting entries [pos, lim) up
  auto place = [&](float &ed, int &ei, float dv, int id, int lim) {
    const bool before = dv < ed || (dv == ed && id < ei);
    const unsigned stay = __ballot_sync(full, !before) & (lim >= 32 ? full : (1u << lim) - 1u);
    const int pos = stay ? 32 - __clz(stay) : 0;
    const float pd = __shfl_up_sync(full, ed, 1);
    const int pi = __shfl_up_sync(full, ei, 1);
    if (lane > pos && lane <= lim) {
      ed = pd;
      ei = pi;
    } else if (lane == pos) {
      ed = dv;
      ei = id;
    }
  };
  float sd = -1.0f;
  int si = -1;
  // the first 32 fill the list, the others pass when below its tail
  for (int c0 = 0; c0 < kMaxCand; c0 += 32) {
    const int id = cand[(size_t)rl * kMaxCand + c0 + lane];
    const float dv = cand_dist[(size_t)rl * kMaxCand + c0 + lane];
    // (a NaN passes and can take the tail's place, and anything passes a NaN
    // there: with one among the 32 each is tested in its turn)
    unsigned todo = c0 ? __ballot_sync(full, !(dv >= __shfl_sync(full, sd, 31))) : full;
    if (__any_sync(full, dv != dv)) todo = full;
    while (todo) {
      const int src = __ffs(todo) - 1;
      todo &= todo - 1u;
      const float v = __shfl_sync(full, dv, src);
      if (c0 && v >= __shfl_sync(full, sd, 31)) continue;
      place(sd, si, v, __shfl_sync(full, id, src), c0 ? kListW - 1 : src);
    }
  }
  Key *gk = g_key + (size_t)(row0 + rl) * kListW;
  const Key old = gk[lane];
  int li = key_id(old);
  float lf = key_dist(old);
  bool updated = false;
  for (int i = 0; i < kListW; ++i) {
    const int id = __shfl_sync(full, si, i);
    const float dv = __shfl_sync(full, sd, i);
    if (__any_sync(full, li == id)) continue;
    const float td = __shfl_sync(full, lf, kListW - 1);
    if (dv > td || dv < 0.0f || (dv == td && id >= __shfl_sync(full, li, kListW - 1))) break;
    place(lf, li, dv, id, kListW - 1);
    updated = true;
  }
  if (updated) {
    gk[lane] = make_key(lf, li);
    if (changed_out && lane == 0) *changed_out = 1;
  }
}

// Copies the first k working entries into the authoritative list (the
// reference's CPU diff, insertion_kernel.cuh:1034-1089) and publishes the row
// with sentinels for invalid or self ids plus the validity flag in column k
// (impl.cuh:103-144, matrix_utils.cuh:128-174).  A warp per row, entry j on
// lane j, in a grid stride (the listed rows are counted on the device): with a
// thread per row every access of a warp was to 32 rows, 82 us for up to 160,000
// rows at k = 30, this form under 15 us.
constexpr int kAdoptWarps = 8;
__global__ void __launch_bounds__(kAdoptWarps * 32)
    k_adopt_publish(const Key *g_key, int *knn_ids, float *knn_dists, uint32_t *pub_idx,
                    float *pub_dist, int k, int row0, int nrows, const int *rows,
                    const int *n_rows_dev, int n) {
  pdl_enter();
  const int lane = threadIdx.x & 31;
  const int total = nrows + (n_rows_dev ? *n_rows_dev : 0);
  for (int i = blockIdx.x * kAdoptWarps + (threadIdx.x >> 5); i < total; i += gridDim.x * kAdoptWarps) {
    const int row = (i < nrows) ? row0 + i : rows[i - nrows];
    const Key key = g_key[(size_t)row * kListW + lane];
    const int e = key_id(key);
    const float dv = key_dist(key);
    const int id = e >= 0 ? e : -e - 1;
    const bool valid = lane < k && id >= 0 && id < n && id != row;
    if (lane < k) {
      knn_ids[(size_t)row * k + lane] = e;
      knn_dists[(size_t)row * k + lane] = dv;
      pub_idx[(size_t)row * (k + 1) + lane] = valid ? (uint32_t)id : kPubIdxSentinel;
      pub_dist[(size_t)row * (k + 1) + lane] = valid ? dv : FLT_MAX;
    }
    const bool any = __any_sync(0xffffffffu, valid);
    if (lane == 0) pub_idx[(size_t)row * (k + 1) + k] = any ? 1u : 0u;
  }
}

// New rows' embedding: N(0,1), then (if a pre-batch neighbour has a finite
// distance) the exp(-(d - d_min))-weighted mean of the pre-batch neighbours
// (reference: insertion_kernel.cuh:790-907).  A warp per row: weights and
// positions of the neighbours on the lanes, the sums in list order by
// shuffles.  One thread per row took 14.5 us for 500 rows at k = 15, on four
// SMs; this form 4 us.
constexpr int kInitEmbWarps = 4;
__global__ void __launch_bounds__(kInitEmbWarps * 32)
    k_embed_init(const Key *g_key, float *emb, int k, int row0, int nrows, int n) {
  pdl_enter();
  const int lane = threadIdx.x & 31;
  const int rl = blockIdx.x * kInitEmbWarps + (threadIdx.x >> 5);
  if (rl >= nrows) return;
  const unsigned full = 0xffffffffu;
  const int row = row0 + rl;
  const Key key = g_key[(size_t)row * kListW + lane];
  const int id = key_id(key);
  const float ds = key_dist(key);
  const bool use = lane < k && id >= 0 && id < n && id < row0;
  float2 p = make_float2(0.0f, 0.0f);
  if (use) p = *reinterpret_cast<const float2 *>(emb + (size_t)id * 2);
  float dmin = use && ds < FLT_MAX ? ds : FLT_MAX;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) dmin = fminf(dmin, __shfl_xor_sync(full, dmin, o));
  Philox g;
  philox_init(g, 42ull, (uint32_t)row, kTagInitEmbedding);
  float e0 = gm_normal(g);
  float e1 = gm_normal(g);
  if (dmin != FLT_MAX) {
    const float w = use ? gm_expf(-__fsub_rn(ds, dmin)) : 0.0f;
    float wsum = 0.0f, a0 = 0.0f, a1 = 0.0f;
    for (unsigned m = __ballot_sync(full, use); m; m &= m - 1u) {
      const int j = __ffs(m) - 1;
      const float wj = __shfl_sync(full, w, j);
      wsum = __fadd_rn(wsum, wj);
      a0 = __fmaf_rn(wj, __shfl_sync(full, p.x, j), a0);
      a1 = __fmaf_rn(wj, __shfl_sync(full, p.y, j), a1);
    }
    if (wsum > 0.0f) {
      e0 = __fdiv_rn(a0, wsum);
      e1 = __fdiv_rn(a1, wsum);
    }
  }
  if (lane == 0) *reinterpret_cast<float2 *>(emb + (size_t)row * 2) = make_float2(e0, e1);
}

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

}  // namespace

void launch_row_norms(const DevState &st, int row0, int nrows, cudaStream_t s) {
  if (nrows <= 0) return;
  launch(k_row_norms, cdiv(nrows, kNormRows), 256, 0, s, st.X, st.norms, st.snorms, st.ld, st.d, row0,
         nrows, st.cosine);
  note_launch();
}

void launch_merge_offers(const DevState &st, int row0, int first, const OfferChains &chains,
                         const float *dist, const int *e_row, int *changed_out, const int *changed,
                         cudaStream_t s) {
  launch(k_merge_offers, cdiv(row0, kOfferWarps), kOfferWarps * 32, 0, s, st.g_key, row0, first, chains,
         dist, e_row, st.dirty, changed_out, changed);
  note_launch();
}

void launch_nnd_insert(const DevState &st, const UpdScratch &u, int row0, int nrows, int n, int window_start,
                       uint64_t seed, const CandScratch &c, int *changed, int sms,
                       const std::function<void(bool)> &timed, cudaStream_t s) {
  if (nrows <= 0) return;
  launch(k_random_init, cdiv(nrows, kInitWarps), kInitWarps * 32, 0, s, st.g_key, row0, nrows, n,
         window_start, seed);
  note_launch();
  const int k = st.k, P = k * k;
  // Below 256 positions (k <= 15) the forward merge, which wants 256
  // candidates, never runs, so the batch rows' lists stay as drawn and only
  // the offers to existing rows (ids below row0) can have an effect.  Those
  // all come in the first iteration: an offer inserts a batch row's id, which
  // moves the list's other entries back or not at all, so a row's two-hop ids
  // below row0 in a later iteration are among those of the first, and an
  // offer made before is listed, or was rejected by entries that only get
  // smaller.  One iteration then gives the state after kInsertIters, and its
  // candidates need not hold batch rows.  (Sampling, distances and offers of
  // 500 rows x 784 at k = 15: 1.70 ms an insertion with ten iterations, 0.37 ms
  // with the one, 0.07 ms with the sampling and the offers as they are now.)
  const bool merges = P >= kMaxCand;
  const int iters = merges ? kInsertIters : (row0 > 0 ? 1 : 0);
  const int slots = hop_slots(k);
  const size_t smem = (size_t)kSampWarps * hop_ints(k) * sizeof(int);
  const int chunks = cdiv(std::min(P, kMaxCand), 32);
  // the chains' heads lie over one of the update's sample lists (n_cap x 32,
  // not in use during an insertion)
  const OfferChains chains{u.fwd_new, c.next};
  if (row0 > 0) cudaMemsetAsync(chains.heads, 0xff, (size_t)row0 * 32 * sizeof(int), s);
  if (merges) cudaMemsetAsync(changed, 0, kInsertIters * sizeof(int), s);
  for (int it = 0; it < iters; ++it) {
    // an iteration that follows one without any change repeats it: its
    // launches return at once
    const int *go = it > 0 ? changed + it - 1 : nullptr;
    int *mark = merges ? changed + it : nullptr;
    launch(k_sample_candidates, cdiv(nrows, kSampWarps), kSampWarps * 32, smem, s, st.g_key, row0, nrows, n,
           k, slots, merges ? 0 : 1, HopOut{c.cand, c.cnt, c.dist, merges ? c.todo : nullptr, c.todo_cnt},
           it, go);
    note_launch();
    for (int r = 0; r < nrows; r += kOfferRows) {
      const int m = std::min(kOfferRows, nrows - r);
      const size_t at = (size_t)r * kMaxCand;
      const int grid = (int)std::min<long>(cdiv((long)m * chunks, kCandWarps), 24L * std::max(sms, 1));
      timed(true);
      launch(k_candidate_offers, grid, kCandWarps * 32, 0, s, st.X, st.norms, st.ld, row0, row0 + r, m,
             chunks, c.cand + at, merges ? c.todo + at : nullptr, (merges ? c.todo_cnt : c.cnt) + r,
             c.dist + at, st.g_key, chains, go, st.stat);
      note_launch();
      timed(false);
      if (row0 > 0) launch_merge_offers(st, row0, row0 + r, chains, c.dist + at, nullptr, mark, go, s);
    }
    if (merges) {
      launch(k_forward_merge, cdiv(nrows, kFwdWarps), kFwdWarps * 32, 0, s, st.g_key, row0, nrows, c.cand,
             c.cnt, c.dist, mark, go);
      note_launch();
    }
  }
}

void launch_adopt_and_publish(const DevState &st, int row0, int nrows,
                              const int *rows, const int *n_rows_dev, int n_rows_max,
                              int n, cudaStream_t s) {
  const int total = nrows + n_rows_max;
  if (total <= 0) return;
  launch(k_adopt_publish, std::min(cdiv(total, kAdoptWarps), 2048), kAdoptWarps * 32, 0, s, st.g_key,
         st.knn_ids, st.knn_dists, st.pub_idx, st.pub_dist, st.k, row0, nrows, rows, n_rows_dev, n);
  note_launch();
}

void launch_embed_init(const DevState &st, int row0, int nrows, int n,
                       cudaStream_t s) {
  if (nrows <= 0) return;
  launch(k_embed_init, cdiv(nrows, kInitEmbWarps), kInitEmbWarps * 32, 0, s, st.g_key, st.emb, st.k, row0,
         nrows, n);
  note_launch();
}

}  // namespace gm
