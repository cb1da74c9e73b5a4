// Update phase: one NN-Descent local-join round over a batch of rows.
// Restates the reference's UpdateAlgo (update_kernel.cuh:689-1054) with the
// sampling, reverse lists, merge and publish all on the device.
#include <algorithm>
#include <climits>
#include <mutex>

#include "gm_common.cuh"
#include "gm_kernels.h"
#include "gm_rowdot.cuh"

namespace gm {

namespace {

// Per-row Bloom filter: 4 sets of 512 bits, 4 hashes (reference
// buffers.cuh:35-137).  Row r owns words [r*64, r*64+64).
GM_D uint32_t bloom_h0(uint32_t v) {
  v *= 1103515245u;
  v += 12345u;
  v ^= v << 13;
  v ^= v >> 17;
  v ^= v << 5;
  return v;
}
GM_D uint32_t bloom_h1(uint32_t v) {
  v *= 1664525u;
  v += 1013904223u;
  v ^= v << 13;
  v ^= v >> 17;
  v ^= v << 5;
  return v;
}
// The four bits of a key: set key % 4, bits (h0 + i h1) % 512 of it.
GM_D int bloom_bit(uint32_t key, int i) {
  return (int)((key % 4u) * 512u + (bloom_h0(key) + (uint32_t)i * bloom_h1(key)) % 512u);
}

// Zeroes the per-row state of an update round and its counters.
__global__ void k_update_reset(int n, int4 *sizes, int *dirty, int *cnt_new, int *cnt_old,
                               int *counters, int n_counters) {
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_counters) counters[i] = 0;
  if (i >= n) return;
  sizes[i] = make_int4(0, 0, 0, 0);
  dirty[i] = 0;
  cnt_new[i] = 0;
  cnt_old[i] = 0;
}

// New/old samples of each batch row from its authoritative k-list: new
// entries (up to 32) are sampled, marked old and recorded in the Bloom
// filter; old entries the filter has not seen are sampled (up to 32)
// (reference: UpdateAlgo::sample_graph, update_kernel.cuh:750-807).
// A warp per row, entry j on lane j.  In list order an old entry sees the bits
// that the new entries before it have set: each new entry's bits are handed
// round and the lanes behind it note the ones they ask for.  The position of
// each sample among its target's sources (pos_*, any order) is taken here, so
// that the reverse lists need no second count.  One thread per row took 26 us
// for 2,000 rows at k = 15, this form 5 us.
constexpr int kSgWarps = 8;
__global__ void __launch_bounds__(kSgWarps * 32)
    k_sample_graph(int *knn_ids, uint32_t *bloom, const int *batch, int nb, int n, int k,
                   int *fwd_new, int *fwd_old, int *pos_new, int *pos_old, int *cnt_new,
                   int *cnt_old, int4 *sizes) {
  pdl_enter();
  __shared__ uint32_t s_bits[kSgWarps][64];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * kSgWarps + warp;
  if (i >= nb) return;
  const unsigned full = 0xffffffffu, lt = (1u << lane) - 1u;
  const int row = batch[i];
  int *list = knn_ids + (size_t)row * k;
  uint32_t *bits = bloom + (size_t)row * 64;
  uint32_t *sb = s_bits[warp];
  const int e = lane < k ? list[lane] : kIdSentinel;
  sb[lane] = bits[lane];
  sb[lane + 32] = bits[lane + 32];
  __syncwarp();
  const int id = e >= 0 ? e : -e - 1;
  const bool valid = lane < k && (uint32_t)id < (uint32_t)n;
  const bool isnew = valid && e >= 0;
  int b[4];
  unsigned seen = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    b[q] = bloom_bit((uint32_t)id, q);
    if (valid && ((sb[b[q] >> 5] >> (b[q] & 31)) & 1u)) seen |= 1u << q;
  }
  __syncwarp();
  const unsigned news = __ballot_sync(full, isnew);
  for (unsigned m = news; m; m &= m - 1u) {
    const int src = __ffs(m) - 1;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int x = __shfl_sync(full, b[p], src);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (src < lane && b[q] == x) seen |= 1u << q;
    }
  }
  const bool isold = valid && e < 0 && seen != 15u;
  const unsigned olds = __ballot_sync(full, isold);
  const size_t at = (size_t)row * kSamples;
  if (isnew) {
    list[lane] = -id - 1;
    const int s = __popc(news & lt);
    fwd_new[at + s] = id;
    pos_new[at + s] = atomicAdd(&cnt_new[id], 1);
#pragma unroll
    for (int q = 0; q < 4; ++q) atomicOr(&sb[b[q] >> 5], 1u << (b[q] & 31));
  }
  if (isold) {
    const int s = __popc(olds & lt);
    fwd_old[at + s] = id;
    pos_old[at + s] = atomicAdd(&cnt_old[id], 1);
  }
  __syncwarp();
  if (news) {
    bits[lane] = sb[lane];
    bits[lane + 32] = sb[lane + 32];
  }
  if (lane == 0) sizes[row] = make_int4(__popc(news), 0, __popc(olds), 0);
}

// A segment of the source array for every target's new, then old sources
// (segments in any order; both together hold at most one entry per list slot
// of the batch, so n_cap x 32 entries are enough).
__global__ void k_rev_segments(int n, const int *cnt_new, const int *cnt_old, int *off_new,
                               int *off_old, int *total) {
  pdl_enter();
  const int j = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
  const int a = j < n ? cnt_new[j] : 0, c = j < n ? cnt_old[j] : 0;
  int v = a + c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  int base = 0;
  if (lane == 31 && v) base = atomicAdd(total, v);
  base = __shfl_sync(0xffffffffu, base, 31) + v - a - c;
  if (j < n) {
    off_new[j] = base;
    off_old[j] = base + a;
  }
}

__global__ void k_rev_place(const int *batch, int nb, const int *fwd_new, const int *fwd_old,
                            const int *pos_new, const int *pos_old, const int4 *sizes,
                            const int *off_new, const int *off_old, int *src) {
  pdl_enter();
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= nb * kSamples) return;
  const int row = batch[tid / kSamples], s = tid % kSamples;
  const size_t at = (size_t)row * kSamples + s;
  const int4 sz = sizes[row];
  if (s < sz.x) src[off_new[fwd_new[at]] + pos_new[at]] = row;
  if (s < sz.z) src[off_old[fwd_old[at]] + pos_old[at]] = row;
}

// Join lists of every row with new samples or sources: N = forward-new, then
// reverse-new not in forward-new; O = forward-old, then reverse-old not in
// forward-old.  A reverse list is its target's 32 smallest source ids in
// ascending order.  (The reference keeps the first 32 atomic arrivals,
// add_rev_edges_kernel, update_kernel.cuh:122-146; ascending ids are one of
// its outcomes and make the round deterministic.)  A warp per row; the kept
// reverse samples replace the positions in rev_*, sizes becomes (forward new,
// kept reverse new, forward old, kept reverse old), and rows with a pair to
// form are appended to the small (at most 32 members) or the large node list
// and get a place in the pool for their block (any order; its words in
// off_new / off_old, low and high half).
constexpr int kListWarps = 8;
// Words of a node's block: per member its chain entry (next, node) and id,
// then the N x (N ++ O) tile; a whole number of chain entries.
GM_D int join_block_words(int nN, int nC) { return (nC * (nN + 3) + 1) & ~1; }
GM_D int warp_smallest(const int *src, int c) {
  // lane l: the l-th smallest of c distinct ids (INT_MAX past the end)
  const int lane = threadIdx.x & 31;
  const unsigned full = 0xffffffffu;
  int mine = INT_MAX;
  for (int c0 = 0; c0 < c; c0 += 32) {
    const int v = c0 + lane < c ? src[c0 + lane] : INT_MAX;
    unsigned todo = __ballot_sync(full, v < __shfl_sync(full, mine, 31));
    while (todo) {
      const int x = __shfl_sync(full, v, __ffs(todo) - 1);
      todo &= todo - 1u;
      const unsigned after = __ballot_sync(full, x < mine);
      if (!after) continue;
      const int pos = __ffs(after) - 1;
      const int prev = __shfl_up_sync(full, mine, 1);
      if (lane > pos) mine = prev;
      else if (lane == pos) mine = x;
    }
  }
  return mine;
}
__global__ void __launch_bounds__(kListWarps * 32)
    k_join_lists(int n, const int *fwd_new, const int *fwd_old, int *rev_new, int *rev_old,
                 const int *cnt_new, const int *cnt_old, int *off_new, int *off_old,
                 const int *src, int4 *sizes, int *small_nodes, int *large_nodes, int *counts,
                 unsigned long long *pool_words) {
  pdl_enter();
  __shared__ int s_cls[kListWarps], s_words[kListWarps];
  __shared__ int s_base[2];
  __shared__ unsigned long long s_pool;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = blockIdx.x * kListWarps + warp;
  const unsigned full = 0xffffffffu;
  int cls = 0, words = 0;
  if (j < n) {
    const int4 sz = sizes[j];
    const int cn = cnt_new[j];
    if (sz.x + cn > 0) {
      const int co = cnt_old[j];
      const size_t at = (size_t)j * kSamples;
      auto side = [&](const int *fwd, int *rev, int nf, int c, int off) {
        const int f = lane < nf ? fwd[at + lane] : -1;
        const int r = warp_smallest(src + off, c);
        bool keep = lane < c && r != INT_MAX;
        for (int q = 0; q < nf; ++q) keep &= __shfl_sync(full, f, q) != r;
        const unsigned bal = __ballot_sync(full, keep);
        if (keep) rev[at + __popc(bal & ((1u << lane) - 1u))] = r;
        return __popc(bal);
      };
      const int rn = side(fwd_new, rev_new, sz.x, cn, off_new[j]);
      const int ro = side(fwd_old, rev_old, sz.z, co, off_old[j]);
      if (lane == 0) sizes[j] = make_int4(sz.x, rn, sz.z, ro);
      const int m = sz.x + rn + sz.z + ro;
      cls = m < 2 ? 0 : m <= 32 ? 1 : 2;
      words = cls ? join_block_words(sz.x + rn, m) : 0;
    }
  }
  if (lane == 0) {
    s_cls[warp] = cls;
    s_words[warp] = words;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    int c = 0;
    for (int w = 0; w < kListWarps; ++w) c += s_cls[w] == (int)threadIdx.x + 1;
    s_base[threadIdx.x] = c ? atomicAdd(&counts[threadIdx.x], c) : 0;
  } else if (threadIdx.x == 2) {
    int c = 0;
    for (int w = 0; w < kListWarps; ++w) c += s_words[w];
    s_pool = c ? atomicAdd(pool_words, (unsigned long long)c) : 0ull;
  }
  __syncthreads();
  if (lane == 0 && cls) {
    int at = s_base[cls - 1];
    unsigned long long pos = s_pool;
    for (int w = 0; w < warp; ++w) {
      at += s_cls[w] == cls;
      pos += (unsigned long long)s_words[w];
    }
    (cls == 1 ? small_nodes : large_nodes)[at] = j;
    off_new[j] = (int)(uint32_t)pos;
    off_old[j] = (int)(pos >> 32);
  }
}

// Local join of a node's lists N and O, in two kernels (reference:
// local_join_kernel, update_kernel.cuh:377-687).
//
// k_join_tiles forms the distances of N x (N ++ O), FP32, a sequential fma
// chain per pair, and stores the tile in the node's block of the pool.  W
// warps work on a node: the CTA's four on a large one, a single warp on a small
// one (at most 32 members), the four warps of a CTA on different nodes.  The
// members' rows come 32 features at a time by 16-byte cp.async into a ring of
// kJoinRing slots (36 words a row: conflict-free 16-byte reads), each row once;
// member row r of N is on warp r % W, member column c on lane c % 32, so a
// thread's products take its own columns and broadcast rows, and its sums stay
// in registers until the tile goes over the ring.  A member whose list some
// offer can change then goes on one of its row's 32 chains (heads[row * 32 +
// node % 32]); a node without one leaves its block unwritten.
//
// k_join_merge, a warp per row, walks the row's chains, 32 memberships at a
// time, and offers it the other side of each tile: as a member of N all other
// members, as a member of O the members of N.
//
// A round whose blocks do not fit the pool takes several passes, each over the
// nodes whose block starts in its part of the (virtual) pool.
//
// Bound by latency (rows from L2, then list and tile reads), so what counts is
// the number of nodes in flight: 16 an SM here, three with a CTA of eight warps
// per node.  Merging every (node, member) under the member's lock instead, as
// the kernel before did, cost most of its time (about 2.5 us a merge, in turn
// for a row in many nodes: 250 of 272 us at 600 rows).  45 rounds of 2,000 rows
// over 20k x 784 (k = 15): 28.4 ms with a CTA per node, 12.0 with a warp per
// small node and locks, 9.5 now; 10 rounds of 10,000 rows over 100k x 128
// (k = 30): 12.8, 6.1, 5.6 ms.
constexpr int kJoinWarps = 4;
constexpr int kJoinRing = 3;
constexpr int kJoinLd = 36;
constexpr int kJoinCols = 2 * kJoinMax;  // members of a large node

struct JoinArgs {
  const int *fwd_new, *fwd_old, *rev_new, *rev_old;
  const int4 *sizes;
  const int *pos_lo, *pos_hi;   // a node's block: its first word, low and high half
  int *pool;                    // this pass's part, from word pass * part_words on
  unsigned long long part_words;
  int pass;
  int *heads;                   // n_cap x 32 chain heads (-1: none)
  const Key *g_key;
  const float *X, *norms;
  int ld;
  unsigned long long *stat;
};
// The node's first word in this pass's pool; false if it belongs to another.
GM_D bool join_block(const JoinArgs &g, int u, int &at) {
  const unsigned long long pos = ((unsigned long long)(uint32_t)g.pos_hi[u] << 32) | (uint32_t)g.pos_lo[u];
  const unsigned long long from = (unsigned long long)g.pass * g.part_words;
  at = (int)(pos - from);
  return pos >= from && pos - from < g.part_words;
}

template <int W>
GM_D void join_sync() {
  if (W == 1) __syncwarp();
  else __syncthreads();
}

// Products of one feature chunk: the thread's CG column groups against its
// warp's rows, four features at a time.
template <int W, int CG, int R, int C>
GM_D void join_products(const float *slot, int nq, int nr, int w, int lane, float (&acc)[R][C]) {
  for (int f = 0; f < nq; ++f) {
    float4 b[CG];
#pragma unroll
    for (int g = 0; g < CG; ++g)
      b[g] = *reinterpret_cast<const float4 *>(slot + (g * 32 + lane) * kJoinLd + 4 * f);
#pragma unroll
    for (int r0 = 0; r0 < R; r0 += 4) {
      if (r0 >= nr) break;
#pragma unroll
      for (int r = r0; r < r0 + 4; ++r) {
        const float4 a = *reinterpret_cast<const float4 *>(slot + (r * W + w) * kJoinLd + 4 * f);
#pragma unroll
        for (int g = 0; g < CG; ++g) {
          acc[r][g] = __fmaf_rn(a.x, b[g].x, acc[r][g]);
          acc[r][g] = __fmaf_rn(a.y, b[g].y, acc[r][g]);
          acc[r][g] = __fmaf_rn(a.z, b[g].z, acc[r][g]);
          acc[r][g] = __fmaf_rn(a.w, b[g].w, acc[r][g]);
        }
      }
    }
  }
}

template <int W>
GM_D void join_node(int u, const JoinArgs &g, float *ring, int *cid, float *nrm) {
  constexpr int kRows = 32 * W;             // ring rows
  constexpr int kGroups = W == 1 ? 1 : kJoinCols / 32;
  constexpr int kMine = W == 1 ? 32 : kJoinMax / W;  // rows of N per warp
  constexpr int kLdD = kRows + 1;
  int block;
  if (!join_block(g, u, block)) return;
  const int lane = threadIdx.x & 31, w = W == 1 ? 0 : (int)(threadIdx.x >> 5);
  const int t = W == 1 ? lane : (int)threadIdx.x;
  const int4 sz = g.sizes[u];
  const int nN = sz.x + sz.y, nC = nN + sz.z + sz.w;
  const size_t at = (size_t)u * kSamples;
  if (t < kSamples) {
    if (lane < sz.x) cid[lane] = g.fwd_new[at + lane];
    if (lane < sz.y) cid[sz.x + lane] = g.rev_new[at + lane];
    if (lane < sz.z) cid[nN + lane] = g.fwd_old[at + lane];
    if (lane < sz.w) cid[nN + sz.z + lane] = g.rev_old[at + lane];
  }
  join_sync<W>();
  for (int c = t; c < nC; c += 32 * W) nrm[c] = g.norms[cid[c]];

  const int q = t & 7, r0 = t >> 3;
  const float *src[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = r0 + 4 * W * i;
    src[i] = g.X + (size_t)(r < nC ? cid[r] : 0) * g.ld + 4 * q;
  }
  const int nch = (g.ld + 31) / 32;
  auto issue = [&](int c) {
    if (c * 32 + 4 * q < g.ld) {
      float *slot = ring + (size_t)(c % kJoinRing) * kRows * kJoinLd + 4 * q;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = r0 + 4 * W * i;
        if (r < nC) dot_cp16(slot + r * kJoinLd, src[i] + c * 32);
      }
    }
    dot_commit();
  };
  float acc[kMine][kGroups];
#pragma unroll
  for (int r = 0; r < kMine; ++r)
#pragma unroll
    for (int c = 0; c < kGroups; ++c) acc[r][c] = 0.0f;
  const int nr = (nN - w + W - 1) / W;  // rows of this warp
  for (int c = 0; c < kJoinRing - 1; ++c) issue(c);
  for (int c = 0; c < nch; ++c) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kJoinRing - 2) : "memory");
    join_sync<W>();  // chunk c has landed, and every thread is done with chunk c - 1
    issue(c + kJoinRing - 1);
    const float *slot = ring + (size_t)(c % kJoinRing) * kRows * kJoinLd;
    const int nq = min(32, g.ld - c * 32) >> 2;
    if (W == 1 || nC <= 32) join_products<W, 1>(slot, nq, nr, w, lane, acc);
    else if (nC <= 64) join_products<W, (W == 1 ? 1 : 2)>(slot, nq, nr, w, lane, acc);
    else if (nC <= 96) join_products<W, (W == 1 ? 1 : 3)>(slot, nq, nr, w, lane, acc);
    else join_products<W, kGroups>(slot, nq, nr, w, lane, acc);
  }
  join_sync<W>();  // every product is done before the tile overwrites the ring
  float *D = ring;
#pragma unroll
  for (int r = 0; r < kMine; ++r)
#pragma unroll
    for (int c = 0; c < kGroups; ++c) {
      const int row = r * W + w, col = c * 32 + lane;
      if (row < nN && col < nC) D[row * kLdD + col] = canon_dist(nrm[row], nrm[col], acc[r][c]);
    }
  join_sync<W>();

  // members that an offer acts on (below the last entry of the member's list
  // and not listed already), one member per warp at a time, the next one's
  // list on its way
  const unsigned full = 0xffffffffu;
  int2 *ent = reinterpret_cast<int2 *>(g.pool + block);
  bool any = false;
  Key next = w < nC ? g.g_key[(size_t)cid[w] * kListW + lane] : 0;
  for (int tt = w; tt < nC; tt += W) {
    const Key list = next;
    if (tt + W < nC) next = g.g_key[(size_t)cid[tt + W] * kListW + lane];
    const int idt = cid[tt];
    const bool in_n = tt < nN;
    const int ncand = in_n ? nC : nN;
    const Key worst = __shfl_sync(full, list, kListW - 1);
    bool act = false;
    for (int c0 = 0; c0 < ncand && !act; c0 += 32) {
      const int c = c0 + lane;
      Key ck = ~(Key)0;
      if (c < ncand && c != tt && cid[c] != idt)
        ck = make_key(in_n ? D[tt * kLdD + c] : D[c * kLdD + tt], cid[c]);
      unsigned todo = __ballot_sync(full, ck < worst);
      while (todo && !act) {
        const Key x = __shfl_sync(full, ck, __ffs(todo) - 1);
        todo &= todo - 1u;
        act = !__any_sync(full, list == x);
      }
    }
    if (act && lane == 0)
      ent[tt] = make_int2(atomicExch(&g.heads[(size_t)idt * 32 + (u & 31)], block / 2 + tt), u);
    any |= act;
  }
  if (W == 1 ? any : __syncthreads_or(any)) {
    int *ids = g.pool + block + 2 * nC;
    float *out = reinterpret_cast<float *>(ids + nC);
    for (int c = t; c < nC; c += 32 * W) ids[c] = cid[c];
    for (int r = w; r < nN; r += W)
      for (int c = lane; c < nC; c += 32) out[r * nC + c] = D[r * kLdD + c];
  }
  if (g.stat && t == 0) {
    atomicAdd(&g.stat[0], 1ull);
    atomicAdd(&g.stat[1], (unsigned long long)nC);
    atomicAdd(&g.stat[2], (unsigned long long)nN * (unsigned long long)nC);
  }
}

// Persistent CTAs take the large nodes together, then their warps the small
// ones, by tickets (counts[0] / counts[1] small / large nodes, counts[2] /
// counts[3] their tickets).
struct JoinSmem {
  float ring[kJoinRing * kJoinCols * kJoinLd];
  int cid[kJoinCols];
  float nrm[kJoinCols];
  int ticket;
};
static_assert(kJoinRing * kJoinCols * kJoinLd >= kJoinMax * (kJoinCols + 1) && kJoinRing * 32 * kJoinLd >= 32 * 33,
              "a node's tile does not fit its ring");
__global__ void __launch_bounds__(kJoinWarps * 32, 4)
    k_join_tiles(const int *small_nodes, const int *large_nodes, int *counts, JoinArgs g) {
  pdl_enter();
  extern __shared__ __align__(16) unsigned char join_raw[];
  JoinSmem &S = *reinterpret_cast<JoinSmem *>(join_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n_small = counts[0], n_large = counts[1];
  for (;;) {
    __syncthreads();  // the previous node's shared data is no longer read
    if (threadIdx.x == 0) S.ticket = n_large ? atomicAdd(&counts[3], 1) : 0;
    __syncthreads();
    if (S.ticket >= n_large) break;
    join_node<kJoinWarps>(large_nodes[S.ticket], g, S.ring, S.cid, S.nrm);
  }
  int next = 0;
  if (lane == 0 && n_small) next = atomicAdd(&counts[2], 1);
  for (;;) {
    const int i = __shfl_sync(0xffffffffu, next, 0);
    if (i >= n_small) break;
    if (lane == 0) next = atomicAdd(&counts[2], 1);
    __syncwarp();
    join_node<1>(small_nodes[i], g, S.ring + (size_t)warp * kJoinRing * 32 * kJoinLd, S.cid + warp * 32,
                 S.nrm + warp * 32);
    __syncwarp();
  }
}

constexpr int kJmWarps = 8;
__global__ void __launch_bounds__(kJmWarps * 32)
    k_join_merge(int n, JoinArgs g, Key *g_key, int *dirty, int k) {
  pdl_enter();
  const int lane = threadIdx.x & 31;
  const int t = blockIdx.x * kJmWarps + (threadIdx.x >> 5);
  if (t >= n) return;
  const unsigned full = 0xffffffffu;
  int e = g.heads[(size_t)t * 32 + lane];
  if (!__any_sync(full, e >= 0)) return;
  g.heads[(size_t)t * 32 + lane] = -1;
  Key *row = g_key + (size_t)t * kListW;
  Key mine = row[lane];
  int minpos = kListW;
  const int2 *entries = reinterpret_cast<const int2 *>(g.pool);
  for (unsigned live; (live = __ballot_sync(full, e >= 0)) != 0u;) {
    // lane: its membership's ids, tile, member number and list sizes
    int ids = 0, c = 0, nN = 0, nC = 0;
    if (e >= 0) {
      const int2 ent = entries[e];
      int block;
      join_block(g, ent.y, block);
      const int4 sz = g.sizes[ent.y];
      nN = sz.x + sz.y;
      nC = nN + sz.z + sz.w;
      c = e - block / 2;
      ids = block + 2 * nC;
      e = ent.x;
    }
    // candidate c0 + lane of membership m (all ones: none)
    auto key_of = [&](int m, int c0) {
      const int mi = __shfl_sync(full, ids, m), mc = __shfl_sync(full, c, m);
      const int mN = __shfl_sync(full, nN, m), mC = __shfl_sync(full, nC, m);
      const bool in_n = mc < mN;
      const int i = c0 + lane;
      if (i >= (in_n ? mC : mN) || i == mc) return ~(Key)0;
      const int id = g.pool[mi + i];
      const float d = __int_as_float(g.pool[mi + mC + (in_n ? mc * mC + i : i * mC + mc)]);
      return id == t ? ~(Key)0 : make_key(d, id);
    };
    Key ahead = key_of(__ffs(live) - 1, 0);
    while (live) {
      const int m = __ffs(live) - 1;
      live &= live - 1u;
      const int mc = __shfl_sync(full, c, m), mN = __shfl_sync(full, nN, m);
      const int ncand = mc < mN ? __shfl_sync(full, nC, m) : mN;
      Key ck = ahead;
      if (live) ahead = key_of(__ffs(live) - 1, 0);
      for (int c0 = 0;;) {
        unsigned todo = __ballot_sync(full, ck < __shfl_sync(full, mine, kListW - 1));
        while (todo) {
          const int s = __ffs(todo) - 1;
          todo &= todo - 1u;
          minpos = min(minpos, warp_insert(mine, __shfl_sync(full, ck, s)));
        }
        c0 += 32;
        if (c0 >= ncand) break;
        ck = key_of(m, c0);
      }
    }
  }
  if (minpos == kListW) return;
  row[lane] = mine;
  if (lane == 0) {
    dirty[t] = max(dirty[t], minpos < k ? 2 : 1);
    if (g.stat) atomicAdd(&g.stat[3], 1ull);
  }
}

// update_graph + sort_lists + publish (reference: update_kernel.cuh:810-878,
// 986-1050) for every row, as the reference does: a row whose working list
// did not change this round can still gain an entry, when an id that was a
// placeholder in its k-list (and so skipped as a duplicate) has since been
// pushed out of the k-list.
// A warp per row, entry j of both lists on lane j.  Most rows change nothing:
// every working entry that could enter is listed already, and none does.
// Otherwise the working entries are taken in order, as insert_to_ordered_list
// does (update_kernel.cuh:87-120).  One thread per row took 206 us for 100,000
// rows at k = 30, this form 56 us.
constexpr int kMpWarps = 8;
__global__ void __launch_bounds__(kMpWarps * 32)
    k_merge_publish(const Key *g_key, int *knn_ids, float *knn_dists, const int *dirty,
                    uint32_t *pub_idx, float *pub_dist, int k, int n, int *edge_counter,
                    int *report_flag) {
  pdl_enter();
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * kMpWarps + (threadIdx.x >> 5);
  if (row >= n) return;
  const unsigned full = 0xffffffffu, ks = k >= 32 ? full : (1u << k) - 1u;
  int *kl = knn_ids + (size_t)row * k;
  float *kd = knn_dists + (size_t)row * k;
  int le = lane < k ? kl[lane] : 0;
  float lv = lane < k ? kd[lane] : 0.0f;
  const Key key = g_key[(size_t)row * kListW + lane];
  const float nd = key_dist(key);
  const int nid = key_id(key);
  auto listed_id = [](int e) { return e >= 0 ? e : -e - 1; };
  const float tail0 = __shfl_sync(full, lv, k - 1);
  // entries up to the first empty or placeholder one
  const unsigned end = __ballot_sync(full, nd == FLT_MAX);
  const bool cand = (end ? lane < __ffs(end) - 1 : true) && nid >= 0 && nid < n && nid != row &&
                    !(nd > tail0);
  bool dup = false;
  for (int q = 0; q < k; ++q) dup |= __shfl_sync(full, listed_id(le), q) == nid;
  int h = 0, edges = 0;
  unsigned todo = __ballot_sync(full, cand);
  if (!__any_sync(full, cand && !dup)) todo = 0;
  while (todo) {
    const int j = __ffs(todo) - 1;
    todo &= todo - 1u;
    const float d = __shfl_sync(full, nd, j);
    const int id = __shfl_sync(full, nid, j);
    if (d > __shfl_sync(full, lv, k - 1)) continue;
    if (__ballot_sync(full, listed_id(le) == id) & ks) continue;
    const unsigned above = __ballot_sync(full, lv > d) & ks;
    if (!above) continue;
    const int idx = __ffs(above) - 1;
    const int pe = __shfl_up_sync(full, le, 1);
    const float pv = __shfl_up_sync(full, lv, 1);
    if (lane > idx) {
      le = pe;
      lv = pv;
    } else if (lane == idx) {
      le = id;
      lv = d;
    }
    h = 2;
    ++edges;
  }
  h = max(h, dirty[row]);
  int report = 0;
  if (h >= 1) {
    // sort_lists: ascending (dist, id_with_flag)
    if (__any_sync(full, lane < k && lv != lv)) {
      // (a NaN has no rank: the insertion sort itself, an entry at a time; an
      // entry goes behind the last one before it that is not above it)
      for (int a = 1; a < k; ++a) {
        const int e = __shfl_sync(full, le, a);
        const float v = __shfl_sync(full, lv, a);
        const bool above = lv > v || (lv == v && le > e);
        const unsigned stay = __ballot_sync(full, !above) & ((1u << a) - 1u);
        const int pos = stay ? 32 - __clz(stay) : 0;
        const int pe = __shfl_up_sync(full, le, 1);
        const float pv = __shfl_up_sync(full, lv, 1);
        if (lane > pos && lane <= a) {
          le = pe;
          lv = pv;
        } else if (lane == pos) {
          le = e;
          lv = v;
        }
      }
    } else {
      int rank = 0;
      for (int q = 0; q < k; ++q) {
        const float v = __shfl_sync(full, lv, q);
        const int e = __shfl_sync(full, le, q);
        rank += v < lv || (v == lv && (e < le || (e == le && q < lane)));
      }
      int from = 0;
      for (int q = 0; q < k; ++q)
        if (__shfl_sync(full, rank, q) == lane) from = q;
      le = __shfl_sync(full, le, from);
      lv = __shfl_sync(full, lv, from);
    }
    if (lane < k) {
      kl[lane] = le;
      kd[lane] = lv;
    }
    if (h == 2) {
      const int id = listed_id(le);
      const bool valid = lane < k && id >= 0 && id < n && id != row;
      if (lane < k) {
        pub_idx[(size_t)row * (k + 1) + lane] = valid ? (uint32_t)id : kPubIdxSentinel;
        pub_dist[(size_t)row * (k + 1) + lane] = valid ? lv : FLT_MAX;
      }
      if (__any_sync(full, valid)) {
        if (lane == 0) pub_idx[(size_t)row * (k + 1) + k] = 1u;
        report = 1;
      }
    }
  }
  if (lane == 0) {
    report_flag[row] = report;
    if (edges) atomicAdd(edge_counter, edges);
  }
}

inline int cdiv(long a, long b) { return (int)((a + b - 1) / b); }

}  // namespace

void launch_join_nodes(const DevState &st, const UpdScratch &u, const int *batch, int nb, int n,
                       int *small_nodes, int *large_nodes, int *counters, cudaStream_t s) {
  if (nb <= 0 || n <= 0) return;
  // new sources are counted in u.cnt, old ones in u.fill; the positions of the
  // samples wait in the batch rows' reverse lists until k_join_lists writes them
  int *off_new = u.off, *off_old = u.hflag;
  launch(k_update_reset, cdiv(std::max(n, kUpdCounters), 256), 256, 0, s, n, u.sizes, st.dirty, u.cnt,
         u.fill, counters, kUpdCounters);
  launch(k_sample_graph, cdiv(nb, kSgWarps), kSgWarps * 32, 0, s, st.knn_ids, st.bloom, batch, nb, n, st.k,
         u.fwd_new, u.fwd_old, u.rev_new, u.rev_old, u.cnt, u.fill, u.sizes);
  launch(k_rev_segments, cdiv(n, 256), 256, 0, s, n, u.cnt, u.fill, off_new, off_old,
         counters + kUpdSources);
  launch(k_rev_place, cdiv((long)nb * kSamples, 256), 256, 0, s, batch, nb, u.fwd_new, u.fwd_old, u.rev_new,
         u.rev_old, u.sizes, off_new, off_old, u.csr);
  launch(k_join_lists, cdiv(n, kListWarps), kListWarps * 32, 0, s, n, u.fwd_new, u.fwd_old, u.rev_new,
         u.rev_old, u.cnt, u.fill, off_new, off_old, u.csr, u.sizes, small_nodes, large_nodes,
         counters + kUpdNodes, (unsigned long long *)(counters + kUpdPool));
  note_launch(5);
}

size_t join_pool_words(int nb, int k) {
  // a node's members are its forward samples and its sources, at most nb k of
  // each over all nodes, and its block takes nN + 3 <= k + 32 + 3 words for
  // each, rounded up to a whole entry
  return 2 * (size_t)nb * (size_t)k * (size_t)(k + kSamples + 4);
}

void launch_local_join(const DevState &st, const UpdScratch &u, const int *small_nodes,
                       const int *large_nodes, int *counters, int *pool, size_t part_words, int pass,
                       int n, cudaStream_t s) {
  if (n <= 0) return;
  const size_t smem = sizeof(JoinSmem);
  // per device, once (sessions on several host threads may launch at once)
  static std::mutex mu;
  static int ctas[32] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  int grid_ctas = 0;
  if (dev < 32) {
    std::lock_guard<std::mutex> g(mu);
    if (!ctas[dev]) {
      cudaFuncSetAttribute(k_join_tiles, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      int sms = 0, per_sm = 0;
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_join_tiles, kJoinWarps * 32, smem);
      ctas[dev] = std::max(1, sms * std::max(per_sm, 1));
    }
    grid_ctas = ctas[dev];
  }
  const int grid = std::min(n, grid_ctas > 0 ? grid_ctas : 1024);
  // the sources' array is free once the join lists stand: chain heads
  const JoinArgs g{u.fwd_new, u.fwd_old, u.rev_new, u.rev_old, u.sizes, u.off, u.hflag, pool,
                   (unsigned long long)part_words, pass, u.csr, st.g_key, st.X, st.norms, st.ld,
                   st.stat};
  if (pass == 0) cudaMemsetAsync(u.csr, 0xff, (size_t)n * 32 * sizeof(int), s);
  else cudaMemsetAsync(counters + kUpdNodes + 2, 0, 2 * sizeof(int), s);  // the tickets
  launch(k_join_tiles, grid, kJoinWarps * 32, smem, s, small_nodes, large_nodes, counters + kUpdNodes, g);
  launch(k_join_merge, cdiv(n, kJmWarps), kJmWarps * 32, 0, s, n, g, st.g_key, st.dirty, st.k);
  note_launch(2);
}

void launch_merge_publish(const DevState &st, int n, int *edge_counter, int *report_flag, cudaStream_t s) {
  if (n <= 0) return;
  launch(k_merge_publish, cdiv(n, kMpWarps), kMpWarps * 32, 0, s, st.g_key, st.knn_ids, st.knn_dists,
         st.dirty, st.pub_idx, st.pub_dist, st.k, n, edge_counter, report_flag);
  note_launch();
}

}  // namespace gm
