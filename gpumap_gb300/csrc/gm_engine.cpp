// Session engine: host-side policy of the progressive cycle, all numeric
// state on the device.  The queue, cursor, seed and completion rules restate
// the reference's GPUMAP::Impl (impl.cuh:29-533); the O(n) host copies and
// host merges of the reference are replaced by device kernels, so per-cycle
// host work and PCIe/C2C traffic scale with the batch, not with n.
#include "gm_engine.h"

#include "gm_common.cuh"
#include "gm_pool.h"

#include <algorithm>
#include <cfloat>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <unordered_set>

#include <unistd.h>

namespace gm {

namespace {

using Clock = std::chrono::high_resolution_clock;

void ck(cudaError_t e, const char *what) {
  if (e == cudaSuccess) return;
  cudaGetLastError();
  if (e == cudaErrorMemoryAllocation)
    throw Error(GM_ERR_OOM, std::string(what) + ": " + cudaGetErrorString(e));
  throw Error(GM_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

size_t round_up(size_t v, size_t m) { return (v + m - 1) / m * m; }

// Takes a half-made set of buffers back when one of them cannot be had.
template <typename F>
struct Undo {
  F f;
  bool done = false;
  ~Undo() {
    if (!done) f();
  }
};
template <typename F>
Undo(F) -> Undo<F>;

// From 256 two-hop positions on, insertion iterates and keeps distances.
bool reuses_dists(int k) { return k * k >= kMaxCand; }
// Insertion scratch for r batch rows (CandScratch).
size_t cand_bytes(size_t r, int k) {
  return r * ((size_t)kMaxCand * (sizeof(int) + sizeof(float)) + sizeof(int)) +
         (reuses_dists(k) ? r * (kMaxCand + sizeof(int)) : 0) +
         std::min<size_t>(r, kOfferRows) * kMaxCand * sizeof(int);
}

}  // namespace

template <typename... A>
void Session::log(const char *fmt, A... a) const {
  if (p_.verbose) {
    std::fprintf(stderr, fmt, a...);
    std::fflush(stderr);
  }
}

Session::Session(const gm_params &p) : p_(p) {
  if (p.n_components != 2)
    throw Error(GM_ERR_INVALID, "n_components must be 2");
  if (p.n_neighbors < 1 || p.n_neighbors > (uint64_t)kListW)
    throw Error(GM_ERR_INVALID, "n_neighbors must be in [1, 32]");
  if (p.n_features < 1) throw Error(GM_ERR_INVALID, "n_features must be >= 1");
  if (p.metric != GM_METRIC_EUCLIDEAN && p.metric != GM_METRIC_COSINE)
    throw Error(GM_ERR_INVALID, "unknown metric");
  if (p.precision != 0 && p.precision != 1)
    throw Error(GM_ERR_INVALID, "precision must be 0 (FP32 NN-Descent) or 1 (exact, BF16 tensor cores)");
  if (p.overlap != 0 && p.overlap != 1) throw Error(GM_ERR_INVALID, "overlap must be 0 or 1");
  if (p.n_instances > (uint64_t)(1u << 30))
    throw Error(GM_ERR_INVALID, "n_instances exceeds 2^30");
  if (p.n_features > (uint64_t)(1u << 24)) throw Error(GM_ERR_INVALID, "n_features too large");

  if (p.device >= 0) ck(cudaSetDevice(p.device), "cudaSetDevice");
  ck(cudaGetDevice(&device_), "cudaGetDevice");
  ck(cudaFree(nullptr), "CUDA context");
  try {
    build();
  } catch (...) {
    release_all();
    device_bound(device_, fixed_bytes_);
    throw;
  }
}

// Streams, buffers and their first contents.
void Session::build() {
  const gm_params &p = p_;
  ck(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "cudaStreamCreate");
  ck(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, device_), "attr");
  int host_tables = 0;
  ck(cudaDeviceGetAttribute(&host_tables, cudaDevAttrPageableMemoryAccessUsesHostPageTables, device_),
     "attr");
  // (not in overlap mode: beside the SGD the reads take 154 us for 500 rows x
  // 784 instead of 18, and the staging copy is hidden behind it: 163.7 ms for a
  // 70k x 784 build against 159.7 staged)
  reads_host_ = host_tables != 0 && !p.overlap;
  if (p.overlap) {
    // the embedding stream gets the higher priority: its cooperative SGD
    // launch is placed as soon as SMs free up
    int lo = 0, hi = 0;
    ck(cudaDeviceGetStreamPriorityRange(&lo, &hi), "stream priorities");
    ck(cudaStreamCreateWithPriority(&estream_, cudaStreamNonBlocking, hi), "cudaStreamCreate");
    ck(cudaStreamCreateWithPriority(&estream_alt_, cudaStreamNonBlocking, hi), "cudaStreamCreate");
    for (cudaEvent_t *e : {&ev_pub_, &ev_emb_, &ev_snap_, &ev_init_, &ev_hpin_, &ev_hpin_alt_})
      ck(cudaEventCreateWithFlags(e, cudaEventDisableTiming), "cudaEventCreate");
  }

  const size_t N = p.n_instances, d = p.n_features, k = p.n_neighbors;
  st_.n_cap = (int)N;
  st_.d = (int)d;
  st_.ld = (int)round_up(d, 4);
  st_.k = (int)k;
  st_.cosine = p.metric == GM_METRIC_COSINE;
  const size_t Nm = std::max<size_t>(N, 1);

  auto dalloc = [&](size_t bytes) -> void * {
    void *ptr = nullptr;
    ck(device_alloc(&ptr, std::max<size_t>(bytes, 16), device_, stream_), "cudaMalloc");
    allocs_.push_back(ptr);
    fixed_bytes_ += std::max<size_t>(bytes, 16);
    return ptr;
  };
  st_.X = (float *)dalloc(Nm * st_.ld * sizeof(float));
  st_.norms = (float *)dalloc(Nm * sizeof(float));
  st_.snorms = (float *)dalloc(Nm * sizeof(float));
  st_.g_key = (unsigned long long *)dalloc(Nm * kListW * sizeof(unsigned long long));
  st_.dirty = (int *)dalloc(Nm * sizeof(int));
  st_.knn_ids = (int *)dalloc(Nm * k * sizeof(int));
  st_.knn_dists = (float *)dalloc(Nm * k * sizeof(float));
  st_.pub_idx = (uint32_t *)dalloc(Nm * (k + 1) * sizeof(uint32_t));
  st_.pub_dist = (float *)dalloc(Nm * (k + 1) * sizeof(float));
  st_.emb = (float *)dalloc(Nm * 2 * sizeof(float));
  st_.bloom = (uint32_t *)dalloc(Nm * 64 * sizeof(uint32_t));
  d_stat_ = (unsigned long long *)dalloc(16 * sizeof(unsigned long long));
  st_.stat = d_stat_;

  us_.fwd_new = (int *)dalloc(Nm * kSamples * sizeof(int));
  us_.fwd_old = (int *)dalloc(Nm * kSamples * sizeof(int));
  us_.rev_new = (int *)dalloc(Nm * kSamples * sizeof(int));
  us_.rev_old = (int *)dalloc(Nm * kSamples * sizeof(int));
  us_.sizes = (int4 *)dalloc(Nm * sizeof(int4));
  us_.cnt = (int *)dalloc(Nm * sizeof(int));
  us_.off = (int *)dalloc((Nm + 1) * sizeof(int));
  us_.fill = (int *)dalloc(Nm * sizeof(int));
  us_.csr = (int *)dalloc(Nm * kSamples * sizeof(int));
  us_.hflag = (int *)dalloc(Nm * sizeof(int));

  d_rows_ = (int *)dalloc(Nm * sizeof(int));
  d_rows2_ = (int *)dalloc(Nm * sizeof(int));
  d_batch_ = (int *)dalloc(Nm * sizeof(int));
  d_cnt_ = (int *)dalloc(kCounters * sizeof(int));
  st_.err = (unsigned *)(d_cnt_ + kErrAt);
  d_tmp_ = (int *)dalloc(compact_tmp_ints((int)Nm) * sizeof(int) + 64);

  // the embedding phase has its own batch, scan scratch, counters and
  // pinned staging, so that it can run beside the other phases (two sets
  // in overlap mode, one per side)
  auto alloc_side = [&](EmbedScratch &e, int *&cnt) {
    e.flag = (int *)dalloc(Nm * sizeof(int));
    e.unsel = (int *)dalloc(Nm * sizeof(int));
    e.sigma = (float *)dalloc(Nm * sizeof(float));
    e.rho = (float *)dalloc(Nm * sizeof(float));
    e.deg = (int *)dalloc(Nm * sizeof(int));
    e.snap = (float *)dalloc(Nm * 2 * sizeof(float));
    e.fscal = (float *)dalloc(16 * sizeof(float));
    e.iscal = (int *)dalloc(16 * sizeof(int));
    e.cap_partial = (Nm * k + 255) / 256 + 512;
    e.partial = (float *)dalloc(e.cap_partial * 2 * sizeof(float));
    e.ipartial = (int *)dalloc(e.cap_partial * sizeof(int));
    e.batch = (int *)dalloc(Nm * sizeof(int));
    e.tmp = (int *)dalloc(compact_tmp_ints((int)Nm) * sizeof(int) + 64);
    if (p.overlap) {
      e.pub_idx_snap = (uint32_t *)dalloc(Nm * (k + 1) * sizeof(uint32_t));
      e.pub_dist_snap = (float *)dalloc(Nm * (k + 1) * sizeof(float));
    }
    cnt = (int *)dalloc(16 * sizeof(int));
  };
  alloc_side(es_, es_cnt_);
  if (p.overlap) alloc_side(es_alt_, es_cnt_alt_);

  pin_bytes_ = (Nm + kCounters) * sizeof(uint32_t);
  ck(host_alloc((void **)&h_pin_, pin_bytes_), "cudaMallocHost");
  ck(host_alloc((void **)&h_emb_pin_, pin_bytes_), "cudaMallocHost");
  if (p.overlap) ck(host_alloc((void **)&h_emb_pin_alt_, pin_bytes_), "cudaMallocHost");
  if (p.precision == 1) {
    // split-BF16 shadow rows (hi | lo, 2 x dh bf16 each) plus a block of
    // candidate / pair scratch for the worst case (every column a
    // candidate of every block row): 28 bytes per (block row, row).  The
    // block takes up to 1,024 rows (fewer, longer launches) within an
    // eighth of the device's memory and at most 32 GB, and at least 128
    dh_ = exact_dh((int)d);
    xh_ = dalloc(Nm * (size_t)dh_ * 4);
    size_t free_b = 0, total_b = 0;
    ck(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo");
    const size_t budget = std::min<size_t>(total_b / 8, (size_t)32 << 30);
    ex_block_ = (int)std::max<size_t>(128, std::min<size_t>(1024, budget / (Nm * 28)));
    ex_block_ = ex_block_ / 128 * 128;
    // the approximate tile itself is only stored on request (tests), in
    // a buffer allocated then
    ex_cand_ = (int *)dalloc((size_t)ex_block_ * Nm * sizeof(int));
    xs_.cand = ex_cand_;
    xs_.cand_d = (float *)dalloc((size_t)ex_block_ * Nm * sizeof(float));
    xs_.row_cnt = (int *)dalloc((size_t)ex_block_ * sizeof(int));
    xs_.pool_cap = (long)ex_block_ * (long)Nm;
    xs_.pool_j = (int *)dalloc((size_t)xs_.pool_cap * sizeof(int));
    xs_.pool_m = (int *)dalloc((size_t)xs_.pool_cap * sizeof(int));
    xs_.pool_d = (float *)dalloc((size_t)xs_.pool_cap * sizeof(float));
    xs_.pair_j = (int *)dalloc((size_t)xs_.pool_cap * sizeof(int));
    xs_.pair_m = (int *)dalloc((size_t)xs_.pool_cap * sizeof(int));
    xs_.row_t = (float *)dalloc((size_t)ex_block_ * sizeof(float));
    xs_.seed = (float *)dalloc((size_t)ex_block_ * sizeof(float));
    // pre-candidate segments: one per (block row, CTA of a row tile), for
    // every grid width a block can take (at most one CTA per column tile),
    // and room for every column up to kExactRoomTiles column tiles (one more,
    // as CTAs with two tiles each may make one up)
    const int tiles = (int)((Nm + 255) / 256);
    const int room = (std::min(tiles, kExactRoomTiles) + 1) * 256;
    xs_.pre_gx = std::min(std::max(sms_, 1), tiles);
    xs_.pre_cap = std::max(kPreCap, (room + xs_.pre_gx - 1) / xs_.pre_gx);
    xs_.pre = (unsigned long long *)dalloc((size_t)ex_block_ * xs_.pre_gx * xs_.pre_cap *
                                           sizeof(unsigned long long));
    xs_.pre_ub = (float *)dalloc((size_t)ex_block_ * xs_.pre_gx * xs_.pre_cap * sizeof(float));
    // (no block of fewer tiles samples more of them than 32)
    xs_.mins_ld = std::max(exact_seed_tiles((int)((Nm + 255) / 256)), 32) * 8;
    xs_.mins = (float *)dalloc((size_t)ex_block_ * xs_.mins_ld * sizeof(float));
    xs_.pre_cnt = (int *)dalloc((size_t)ex_block_ * xs_.pre_gx * sizeof(int));
    xs_.pre_over = (int *)dalloc(sizeof(int));
    xs_.heaps = (float *)dalloc((size_t)ex_block_ * std::max(sms_, 1) * 32 * sizeof(float));
    xs_.pcnt = (int *)dalloc((size_t)ex_block_ * sizeof(int));
    xs_.poff = (int *)dalloc(((size_t)ex_block_ + 1) * sizeof(int));
    xs_.pfill = (int *)dalloc((size_t)ex_block_ * sizeof(int));
    xs_.ptask = (int *)dalloc(((size_t)ex_block_ + 1) * sizeof(int));
    xs_.heads = us_.fwd_new;  // not in use during an insertion
    xs_.counter = (int *)dalloc(16 * sizeof(int));
  }

  // Initial contents: zero features (padding must stay zero), empty lists,
  // "no neighbour" published rows, zero embedding.
  cudaStream_t s = stream_;
  ck(cudaMemsetAsync(st_.X, 0, Nm * st_.ld * sizeof(float), s), "memset");
  ck(cudaMemsetAsync(st_.norms, 0, Nm * sizeof(float), s), "memset");
  ck(cudaMemsetAsync(st_.snorms, 0, Nm * sizeof(float), s), "memset");
  fill_u64(st_.g_key, kEmptyKey, Nm * kListW, s);
  ck(cudaMemsetAsync(st_.dirty, 0, Nm * sizeof(int), s), "memset");
  fill_u32(st_.knn_ids, (uint32_t)kIdSentinel, Nm * k, s);
  fill_u32(st_.knn_dists, kFltMaxBits, Nm * k, s);
  fill_u32(st_.pub_idx, kPubIdxSentinel, Nm * (k + 1), s);
  fill_u32(st_.pub_dist, kFltMaxBits, Nm * (k + 1), s);
  ck(cudaMemsetAsync(st_.emb, 0, Nm * 2 * sizeof(float), s), "memset");
  ck(cudaMemsetAsync(st_.bloom, 0, Nm * 64 * sizeof(uint32_t), s), "memset");
  ck(cudaMemsetAsync(d_cnt_, 0, kCounters * sizeof(int), s), "memset");
  ck(cudaMemsetAsync(d_stat_, 0, 16 * sizeof(unsigned long long), s), "memset");
  ck(cudaMemsetAsync(us_.sizes, 0, Nm * sizeof(int4), s), "memset");
  for (EmbedScratch *e : {&es_, &es_alt_}) {
    if (!e->sigma) continue;
    ck(cudaMemsetAsync(e->sigma, 0, Nm * sizeof(float), s), "memset");
    ck(cudaMemsetAsync(e->rho, 0, Nm * sizeof(float), s), "memset");
    ck(cudaMemsetAsync(e->iscal, 0, 16 * sizeof(int), s), "memset");
    ck(cudaMemsetAsync(e->fscal, 0, 16 * sizeof(float), s), "memset");
  }
  if (xh_) ck(cudaMemsetAsync(xh_, 0, Nm * (size_t)dh_ * 4, s), "memset");
  ck(cudaGetLastError(), "init fill");
  ck(cudaStreamSynchronize(s), "init sync");
  if (xh_) {
    if (!make_row_maps(xh_, (int)Nm, dh_, &maps_))
      throw Error(GM_ERR_CUDA, "cuTensorMapEncodeTiled unavailable or failed");
  }
  upd_q_.reset(N);
  ensure_embed(es_, 1);
  if (p.overlap) ensure_embed(es_alt_, 1);
}

// The fixed buffers, after every stream has been waited for.
void Session::release_memory() {
  if (stream_) cudaStreamSynchronize(stream_);
  for (void *q : allocs_) device_free(q, stream_);
  allocs_.clear();
  // (the pool can give a block back only after its free has been waited for)
  if (stream_) cudaStreamSynchronize(stream_);
  for (uint32_t **h : {&h_pin_, &h_emb_pin_, &h_emb_pin_alt_}) {
    host_free(*h, pin_bytes_);
    *h = nullptr;
  }
}

void Session::release_streams() {
  for (cudaEvent_t *e : {&ev_pub_, &ev_emb_, &ev_snap_, &ev_init_, &ev_hpin_, &ev_hpin_alt_}) {
    if (*e) cudaEventDestroy(*e);
    *e = nullptr;
  }
  for (cudaStream_t *q : {&estream_, &estream_alt_, &stream_}) {
    if (*q) cudaStreamDestroy(*q);
    *q = nullptr;
  }
}

// Waits for both embedding sides.
void Session::sync_embed_streams() {
  for (cudaStream_t q : {estream_, estream_alt_})
    if (q) ck(cudaStreamSynchronize(q), "cudaStreamSynchronize");
}

void Session::free_embed(EmbedScratch &e) {
  auto drop = [&](auto *&...p) { ((device_free(p, stream_), p = nullptr), ...); };
  drop(e.coo_row, e.coo_col, e.coo_val, e.t_row, e.t_col, e.flag_tail, e.t_val, e.next_s, e.next_n, e.tmp2);
  e.cap_coo = 0;
}

// Everything the session holds, however far it was built; its work has been
// waited for.
void Session::release_all() {
  if (cstream_) cudaStreamSynchronize(cstream_);
  for (cudaStream_t q : {estream_, estream_alt_})
    if (q) cudaStreamSynchronize(q);
  free_cand();
  device_free(join_pool_, stream_);
  join_pool_ = nullptr;
  free_embed(es_);
  free_embed(es_alt_);
  release_memory();
  for (auto &slot : ring_) {
    if (slot.done) cudaEventDestroy(slot.done);
    host_free(slot.buf, slot.cap);
  }
  if (cstream_) cudaStreamDestroy(cstream_);
  release_streams();
}

Session::~Session() {
  // everything on the device: a consumer's stream may still be reading a view,
  // and the pool hands the memory on (cudaFree would have waited as well)
  int current = 0;
  cudaGetDevice(&current);
  if (current != device_) cudaSetDevice(device_);
  cudaDeviceSynchronize();
  if (current != device_) cudaSetDevice(current);
  const size_t held = device_bytes();
  for (auto &e : ev_pool_) cudaEventDestroy(e);
  for (auto &pr : ev_pending_) {
    cudaEventDestroy(pr.a);
    cudaEventDestroy(pr.b);
  }
  release_all();
  device_closed(device_, held);
}

void Session::sync() { ck(cudaStreamSynchronize(stream_), "cudaStreamSynchronize"); }

// The consumer stream waits (on the device) for the work queued so far on
// the main and the embedding streams; the main stream already waits for
// every row transfer.
void Session::order_after(cudaStream_t consumer) const {
  for (cudaStream_t producer : {stream_, estream_, estream_alt_}) {
    if (!producer) continue;
    cudaEvent_t ev = nullptr;
    ck(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "cudaEventCreate");
    const cudaError_t e1 = cudaEventRecord(ev, producer);
    const cudaError_t e2 = e1 == cudaSuccess ? cudaStreamWaitEvent(consumer, ev, 0) : e1;
    cudaEventDestroy(ev);  // the wait keeps the recorded work
    ck(e2, "stream wait");
  }
}

// Waits for every phase in flight, the overlapped embedding included, and
// reports a device error bit raised meanwhile.
void Session::drain() {
  sync();
  sync_embed_streams();
  emb_pending_ = snap_pending_ = init_wait_ = false;
  check_device_error("embedding");
}

void Session::raise_device_error(unsigned bits) {
  ck(cudaMemcpyAsync(st_.err, &bits, sizeof(bits), cudaMemcpyHostToDevice, stream_), "error bits");
  sync();
}

void Session::check_launch_error(const char *phase) {
  // a launch the runtime refused (resources, configuration) is reported
  // once, by the next query of the last error
  const cudaError_t le = cudaGetLastError();
  if (le != cudaSuccess) ck(le, (std::string(phase) + " launch").c_str());
}

void Session::check_device_error(const char *phase) {
  check_launch_error(phase);
  ck(cudaMemcpyAsync(h_pin_ + kErrAt, st_.err, sizeof(unsigned), cudaMemcpyDeviceToHost, stream_), "err");
  sync();
  report_device_error(phase, h_pin_[kErrAt]);
}

void Session::report_device_error(const char *phase, unsigned e) {
  if (e == 0u) return;
  cudaMemsetAsync(st_.err, 0, sizeof(unsigned), stream_);
  throw Error(GM_ERR_DEVICE, std::string(phase) + ": a bounded device wait ran out (bits " +
                                 std::to_string(e) + ")");
}

// Ends a phase that compacted a row list into d_rows_ (count in d_cnt_[0], at
// most `bound` rows): its counters, error word and first rows come in one wait
// (three waits, for the count, the rows and the error word, were 30 us a
// phase).  Counters are then at h_pin_, the rows after them; returns their
// number.  Error bits are kept for end_phase, so that the caller's queues are
// brought up to date first.
size_t Session::finish_phase(const char *phase, size_t bound) {
  check_launch_error(phase);
  const size_t ahead = std::min(bound, kRowsAhead);
  uint32_t *rows = h_pin_ + kCounters;
  ck(cudaMemcpyAsync(h_pin_, d_cnt_, kCounters * sizeof(int), cudaMemcpyDeviceToHost, stream_), "counts");
  if (ahead)
    ck(cudaMemcpyAsync(rows, d_rows_, ahead * sizeof(int), cudaMemcpyDeviceToHost, stream_), "rows");
  sync();
  err_bits_ |= h_pin_[kErrAt];
  err_read_ = true;
  const size_t n = h_pin_[0];
  if (n > ahead) {
    ck(cudaMemcpyAsync(rows + ahead, d_rows_ + ahead, (n - ahead) * sizeof(int), cudaMemcpyDeviceToHost,
                       stream_), "rows");
    sync();
  }
  return n;
}

// After a phase: reports the error bits it read.  A phase that had nothing to do
// read none; then, in overlap mode, the word is read here, because the embedding
// still in flight at the last report may have set it since.
void Session::end_phase(const char *phase) {
  const bool read = err_read_;
  const unsigned bits = err_bits_;
  err_read_ = false;
  err_bits_ = 0;
  if (read) report_device_error(phase, bits);
  else if (p_.overlap) check_device_error(phase);
  else check_launch_error(phase);
}

void Session::free_cand() {
  for (void *q : {(void *)cs_.cand, (void *)cs_.cnt, (void *)cs_.dist, (void *)cs_.todo,
                  (void *)cs_.todo_cnt, (void *)cs_.next})
    device_free(q, stream_);
  cs_ = CandScratch{};
  cand_rows_ = 0;
}

void Session::ensure_cand(size_t rows) {
  if (rows <= cand_rows_) return;
  sync();
  free_cand();
  const size_t r = std::max<size_t>(rows, 1024), slots = r * kMaxCand;
  Undo whole{[&] { free_cand(); }};
  auto get = [&](auto *&p, size_t n) {
    ck(device_alloc((void **)&p, n * sizeof(*p), device_, stream_), "cudaMalloc cand");
  };
  get(cs_.cand, slots);
  get(cs_.cnt, r);
  get(cs_.dist, slots);
  if (reuses_dists(st_.k)) {
    get(cs_.todo, slots);
    get(cs_.todo_cnt, r);
  }
  get(cs_.next, std::min<size_t>(r, kOfferRows) * kMaxCand);
  whole.done = true;
  cand_rows_ = r;
}

// The join pool: words for every block of a round, up to kJoinPartWords.  Where
// the device has no room for them a smaller pool does, with more passes: the
// round's batch has left the queue, and the update needed no memory of its own
// before it had a pool.
void Session::ensure_join(size_t words) {
  size_t w = join_part(words);
  if (w <= join_words_) return;
  sync();
  device_free(join_pool_, stream_);
  join_pool_ = nullptr;
  join_words_ = 0;
  for (;; w = (w / 2 + 1) & ~(size_t)1) {
    const cudaError_t e = device_alloc((void **)&join_pool_, (w + kJoinSlackWords) * sizeof(int), device_, stream_);
    if (e == cudaSuccess) break;
    if (e != cudaErrorMemoryAllocation || w <= kJoinLeastWords) ck(e, "cudaMalloc join");
  }
  join_words_ = w;
}

void Session::set_join_part(size_t words) {
  drain();
  device_free(join_pool_, stream_);
  join_pool_ = nullptr;
  join_words_ = 0;
  join_part_max_ = std::max<size_t>(2, std::min(words, kJoinPartWords) & ~(size_t)1);
}

void Session::set_pre_cap(int cap) {
  drain();
  xs_.pre_cap = std::max(0, std::min(cap, kPreCap));
  xs_.pre_fixed = true;
}

void Session::set_keep_tile(bool on) {
  if (on && p_.precision == 1 && !ex_D_) {
    drain();
    const size_t bytes = (size_t)ex_block_ * std::max<size_t>(p_.n_instances, 1) * sizeof(float);
    void *ptr = nullptr;
    ck(device_alloc(&ptr, bytes, device_, stream_), "cudaMalloc tile");
    allocs_.push_back(ptr);
    fixed_bytes_ += bytes;
    ex_D_ = (float *)ptr;
    xs_.D = ex_D_;
  }
  keep_tile_ = on;
}

size_t Session::device_bytes() const {
  size_t b = fixed_bytes_;
  b += cand_bytes(cand_rows_, st_.k);
  b += join_bytes();
  for (const EmbedScratch *e : {&es_, &es_alt_})
    if (e->cap_coo) b += e->cap_coo * 9 * 4 + (compact_tmp_ints((int)e->cap_coo) + 64) * sizeof(int);
  return b;
}

size_t Session::growth_bytes(uint32_t n_ins, uint32_t n_upd, uint32_t n_emb) const {
  size_t g = 0;
  if (n_upd > 0 && !upd_done_) {
    const size_t rows = std::min<size_t>(n_upd, n_inserted_ + n_ins);
    const size_t w = join_part(join_pool_words((int)rows, st_.k));
    // (the pool it has goes first)
    if (w > join_words_) g += (w + kJoinSlackWords) * sizeof(int) - join_bytes();
  }
  if (p_.precision == 0 && n_ins > cand_rows_) {
    const size_t r = std::max<size_t>(n_ins, 1024);
    g += cand_bytes(r, st_.k);
  }
  // an embedding batch takes the queued new rows plus the cursor's rows
  const size_t nb = std::max<size_t>(n_emb, n_inserted_ + n_ins - emb_new_head_);
  const size_t c = std::max<size_t>(2 * std::max<size_t>(nb, 1) * (size_t)st_.k, 4096);
  // (in overlap mode the next phase runs on the other side)
  const EmbedScratch &next = p_.overlap ? es_alt_ : es_;
  if (n_emb > 0 && c > next.cap_coo) g += c * 9 * 4 + (compact_tmp_ints((int)c) + 64) * sizeof(int);
  return g;
}

void Session::ensure_embed(EmbedScratch &e, size_t nb) {
  const size_t need = 2 * std::max<size_t>(nb, 1) * (size_t)st_.k;
  if (need <= e.cap_coo) return;
  sync();
  sync_embed_streams();
  free_embed(e);
  const size_t c = std::max(need, (size_t)4096);
  Undo whole{[&] { free_embed(e); }};
  auto get = [&](auto *&p, size_t n) {
    ck(device_alloc((void **)&p, n * sizeof(*p), device_, stream_), "cudaMalloc coo");
  };
  get(e.coo_row, c);
  get(e.coo_col, c);
  get(e.coo_val, c);
  get(e.t_row, c);
  get(e.t_col, c);
  get(e.flag_tail, c);
  get(e.t_val, c);
  get(e.next_s, c);
  get(e.next_n, c);
  get(e.tmp2, compact_tmp_ints((int)c) + 64);
  sync();  // (the embedding may run on another stream)
  whole.done = true;
  e.cap_coo = c;
}

// ---------------------------------------------------------------------------
// statistics: CUDA events around the launches of interest
// ---------------------------------------------------------------------------
void Session::timed_begin(int slot, cudaStream_t s) {
  if (!stats_on_) return;
  if (!s) s = stream_;
  cudaEvent_t a, b;
  if (ev_pool_.size() >= 2) {
    a = ev_pool_.back();
    ev_pool_.pop_back();
    b = ev_pool_.back();
    ev_pool_.pop_back();
  } else {
    cudaEventCreate(&a);
    cudaEventCreate(&b);
  }
  cudaEventRecord(a, s);
  ev_pending_.push_back({a, b, slot});
}

void Session::timed_end(int slot, cudaStream_t s) {
  if (!stats_on_ || ev_pending_.empty()) return;
  (void)slot;
  cudaEventRecord(ev_pending_.back().b, s ? s : stream_);
}

// Accumulates the event pairs in order; without `block`, stops at the first
// pair still in flight (an overlapped embedding) and keeps the rest.
void Session::collect_timings(bool block) {
  if (ev_pending_.empty()) return;
  size_t done = 0;
  for (auto &pr : ev_pending_) {
    if (!block && cudaEventQuery(pr.b) != cudaSuccess) {
      cudaGetLastError();
      break;
    }
    ++done;
    float ms = 0.0f;
    if (cudaEventSynchronize(pr.b) == cudaSuccess && cudaEventElapsedTime(&ms, pr.a, pr.b) == cudaSuccess) {
      if (pr.slot == 0) {
        stats_.join_ms += ms;
        stats_.join_launches += 1;
      } else if (pr.slot == 1) {
        stats_.cand_ms += ms;
        stats_.cand_launches += 1;
      } else if (pr.slot == 2) {
        stats_.sgd_ms += ms;
        stats_.sgd_launches += 1;
      } else if (pr.slot == 3) {
        stats_.exact_ms += ms;
        stats_.exact_launches += 1;
      } else if (pr.slot == 4) {
        stats_.screen_ms += ms;
      }
    }
    ev_pool_.push_back(pr.a);
    ev_pool_.push_back(pr.b);
  }
  ev_pending_.erase(ev_pending_.begin(), ev_pending_.begin() + (long)done);
}

void Session::reset_stats() {
  sync();
  collect_timings();
  stats_ = gm_stats{};
  cudaMemsetAsync(d_stat_, 0, 16 * sizeof(unsigned long long), stream_);
  launch_counter_reset();
  sync();
}

void Session::get_stats(gm_stats *out) {
  sync();
  sync_embed_streams();
  collect_timings(true);
  unsigned long long h[16];
  ck(cudaMemcpy(h, d_stat_, sizeof(h), cudaMemcpyDeviceToHost), "stats");
  stats_.join_nodes = h[0];
  stats_.join_rows = h[1];
  stats_.join_pairs = h[2];
  stats_.join_merges = h[3];
  stats_.cand_rows = h[4];
  stats_.exact_pairs = h[5];
  stats_.exact_rescored = h[6];
  stats_.sgd_edges = h[7];
  stats_.sgd_negatives = h[8];
  stats_.exact_overflow_blocks = h[9];
  stats_.kernel_launches = launch_counter();
  *out = stats_;
}

// The kernel loads whole floats, so rows at an address that is not a multiple
// of four go through the staging copy, for which alignment does not matter (a
// misaligned load would end the context).
Ingest ingest_route(const void *rows, bool page_locked, bool reads_host) {
  if (page_locked) return Ingest::kCopy;
  const bool aligned = (reinterpret_cast<uintptr_t>(rows) & (alignof(float) - 1)) == 0;
  return reads_host && aligned ? Ingest::kInPlace : Ingest::kStaged;
}

// ---------------------------------------------------------------------------
// append (reference impl.cuh:77-101)
// ---------------------------------------------------------------------------
// Appends rows at [n_inserted, +n_rows) of X (row stride ld; reference
// append_host, matrix_utils.cuh:50-63, a cudaMemcpy2DAsync into stride d+1).
// Host rows are copied on a stream of their own, so that the next chunk's
// transfer runs beside work still going (an overlapped embedding); the main
// stream waits for it on the device.  Rows in page-locked memory are copied
// from where they are.  Pageable rows are read in place by a kernel where the
// GPU shares the CPU's page tables (launch_copy_rows) and the rows are aligned
// to floats; else they go through two pinned staging slots (waiting only for the slot's previous
// transfer).  Where the caller's buffer is read, the call returns after the
// copy, so that the buffer can be reused.
void Session::append(const float *rows, size_t n_rows, size_t n_cols, bool on_device) {
  if (closed_) throw Error(GM_ERR_CLOSED, "session is closed");
  if (n_rows == 0) return;
  if (n_cols != p_.n_features)
    throw Error(GM_ERR_RUNTIME, "n_features mismatch with numpy array second dimension.");
  if (rows == nullptr) throw Error(GM_ERR_RUNTIME, "null input rows");
  if (n_inserted_ + n_rows > p_.n_instances)
    throw Error(GM_ERR_CAPACITY, "Exceeding maximum number of rows in storage");
  float *dst = st_.X + n_inserted_ * (size_t)st_.ld;
  const size_t pitch = (size_t)st_.ld * sizeof(float), width = n_cols * sizeof(float);
  if (on_device) {
    ck(cudaMemcpy2DAsync(dst, pitch, rows, width, width, n_rows, cudaMemcpyDeviceToDevice, stream_),
       "append copy");
  } else {
    if (!cstream_) {
      ck(cudaStreamCreateWithFlags(&cstream_, cudaStreamNonBlocking), "cudaStreamCreate");
      for (auto &slot : ring_) ck(cudaEventCreateWithFlags(&slot.done, cudaEventDisableTiming), "cudaEventCreate");
    }
    cudaPointerAttributes attr{};
    const bool pinned = cudaPointerGetAttributes(&attr, rows) == cudaSuccess &&
                        (attr.type == cudaMemoryTypeHost || attr.type == cudaMemoryTypeManaged);
    cudaGetLastError();
    RingSlot &slot = ring_[ring_next_];
    ring_next_ = (ring_next_ + 1) % kRingSlots;
    const float *src = rows;
    const Ingest route = ingest_route(rows, pinned, reads_host_);
    if (route == Ingest::kStaged) {
      const size_t bytes = n_rows * width;
      ck(cudaEventSynchronize(slot.done), "ingest slot");  // its previous transfer
      if (slot.cap < bytes) {
        host_free(slot.buf, slot.cap);
        slot.buf = nullptr;
        slot.cap = 0;
        ck(host_alloc(&slot.buf, std::max<size_t>(bytes, (size_t)8 << 20)), "cudaMallocHost ingest");
        slot.cap = std::max<size_t>(bytes, (size_t)8 << 20);
      }
      std::memcpy(slot.buf, rows, bytes);
      src = (const float *)slot.buf;
    }
    if (route == Ingest::kInPlace) {
      // one read per page on the CPU: a page whose entry the kernel has
      // withdrawn for a moment (NUMA balancing does, also of a VM on its host) costs the
      // GPU a fault of 0.7 ms, the CPU one of a microsecond
      static const size_t page = (size_t)std::max<long>(sysconf(_SC_PAGESIZE), 4096);
      const volatile char *b = (const volatile char *)rows;
      for (size_t at = 0; at < n_rows * width; at += page) (void)b[at];
      (void)b[n_rows * width - 1];
      launch_copy_rows(src, dst, n_rows, st_.d, st_.ld, sms_, cstream_);
      ck(cudaGetLastError(), "append copy");
    } else {
      ck(cudaMemcpy2DAsync(dst, pitch, src, width, width, n_rows, cudaMemcpyHostToDevice, cstream_),
         "append copy");
    }
    ck(cudaEventRecord(slot.done, cstream_), "ingest event");
    ck(cudaStreamWaitEvent(stream_, slot.done, 0), "ingest wait");
    if (route != Ingest::kStaged) {
      // the caller's buffer is in use until the transfer ends: block here
      // rather than let the caller overwrite it (the slot event covers it)
      ck(cudaEventSynchronize(slot.done), "append copy");
    }
  }
  n_inserted_ += n_rows;
}

// ---------------------------------------------------------------------------
// run (reference impl.cuh:146-218)
// ---------------------------------------------------------------------------
gm_result Session::run(uint32_t n_ins, uint32_t n_upd, uint32_t n_emb) {
  if (closed_) throw Error(GM_ERR_CLOSED, "session is closed");
  gm_result r{};
  log("[GPUMAP] run() start: insert=%u update=%u embed=%u inserted=%zu\n", n_ins, n_upd, n_emb,
      n_inserted_);
  // overlap mode: with no update in between, the new rows' embedding moves to
  // the start of this run's embedding phase (it must follow the phase in
  // flight, which the insertion itself need not wait for)
  defer_init_ = p_.overlap && n_upd == 0 && n_emb != 0 && !emb_done_;
  if (!ins_done_) {
    const auto t0 = Clock::now();
    r.n_insertion_ops = insert(n_ins);
    end_phase("insertion");
    const auto t1 = Clock::now();
    r.insertion_time = std::chrono::duration<float>(t1 - t0).count();
    ins_done_ = (ins_head_ == n_inserted_) && n_inserted_ == p_.n_instances;
    log("[GPUMAP] insert done: actual=%u time=%.3fs\n", r.n_insertion_ops, r.insertion_time);
  }
  if (n_upd != 0 && !upd_done_) {
    size_t changed = 0;
    const auto t0 = Clock::now();
    r.n_update_ops = update(n_upd, changed);
    end_phase("update");
    const auto t1 = Clock::now();
    r.n_update_changed_edges = changed;
    r.update_time = std::chrono::duration<float>(t1 - t0).count();
    log("[GPUMAP] update done: actual=%u changed_edges=%zu time=%.3fs\n", r.n_update_ops,
        changed, r.update_time);
  }
  r.embedding_pending_edges = n_inserted_;
  if (n_emb != 0 && n_inserted_ != 0 && !emb_done_) {
    const auto t0 = Clock::now();
    r.n_embedding_ops = embed(n_emb);
    if (!p_.overlap) {
      check_device_error("embedding");
    } else {
      check_launch_error("embedding");
    }
    const auto t1 = Clock::now();
    r.embedding_time = std::chrono::duration<float>(t1 - t0).count();
    log("[GPUMAP] embed done: actual=%u time=%.3fs\n", r.n_embedding_ops, r.embedding_time);
  }
  flush_init();
  defer_init_ = false;
  collect_timings(!p_.overlap);
  stats_.phase_s[0] += r.insertion_time;
  stats_.phase_s[1] += r.update_time;
  stats_.phase_s[2] += r.embedding_time;
  r.n_inserted_instances = n_inserted_;
  r.insertion_queue_size = n_inserted_ - ins_head_;
  r.update_queue_size = upd_q_.size();
  r.embedding_queue_size = r.embedding_pending_edges;
  r.insertion_completed = ins_done_;
  r.update_completed = upd_done_;
  r.embedding_completed = emb_done_;
  return r;
}

// ---------------------------------------------------------------------------
// insertion (reference impl.cuh:220-253, insertion_kernel.cuh:926-1095)
// ---------------------------------------------------------------------------
uint32_t Session::insert(uint32_t n_ops) {
  const size_t qsize = n_inserted_ - ins_head_;
  if (qsize == 0 || n_ops == 0) return 0;
  const size_t B = std::min<size_t>(n_ops, qsize);
  const int row0 = (int)ins_head_;
  ins_head_ += B;
  batch_hist_.push_back((uint32_t)row0);
  if ((int)batch_hist_.size() > kWindowBatches) batch_hist_.pop_front();
  const int window_start = (int)batch_hist_.front();
  const int seed_i = (int)(n_ops * 9973u + (uint32_t)n_inserted_ * 7919u);
  const uint64_t seed = (uint64_t)(int64_t)seed_i;
  const int n = (int)n_inserted_;
  const int nb = (int)B;
  cudaStream_t s = stream_;

  if (!bloom_clean_) {
    ck(cudaMemsetAsync(st_.bloom, 0, (size_t)st_.n_cap * 64 * sizeof(uint32_t), s), "bloom");
    bloom_clean_ = true;
  }
  ck(cudaMemsetAsync(st_.dirty, 0, (size_t)n * sizeof(int), s), "dirty");
  launch_row_norms(st_, row0, nb, s);
  // the previous insertion's rows get their embedding at the start of the
  // embedding phase that followed it, from their working lists: no list
  // changes before that has run
  auto wait_init = [&] {
    if (init_wait_) ck(cudaStreamWaitEvent(s, ev_init_, 0), "wait row embedding");
    init_wait_ = false;
  };
  if (p_.precision == 1) {
    // exact lists: every batch row against every inserted row on the tensor
    // cores, re-scored in FP32 where the split-BF16 bound cannot decide
    launch_to_bf16(st_, xh_, dh_, row0, nb, s);
    // columns: the rows inserted so far (rows appended but still queued have
    // no norms or shadow rows yet)
    const int ncol = row0 + nb;
    ck(cudaMemsetAsync(xs_.heads, 0xff, (size_t)row0 * 32 * sizeof(int), s), "heads");
    for (int b0 = 0; b0 < nb; b0 += ex_block_) {
      const int rows = std::min(ex_block_, nb - b0);
      timed_begin(3);
      launch_exact_dist(st_, maps_, dh_, row0, b0, rows, ncol, xs_, (long)ncol, keep_tile_, sms_, s);
      timed_end(3);
      wait_init();
      timed_begin(4);
      launch_exact_screen(st_, row0, b0, rows, ncol, xs_, (long)ncol, sms_, s);
      timed_end(4);
      // algorithmic work: three BF16 products per padded feature (hi.hi,
      // hi.lo, lo.hi) for every pair, once (the seed pass, and pass 2 after
      // an overflow, are overhead on the same pairs)
      const uint64_t flops = 6ull * (uint64_t)rows * (uint64_t)ncol * (uint64_t)dh_;
      stats_.exact_flops += (double)(stats_on_ ? flops : 0);
    }
  } else {
    ensure_cand(B);
    wait_init();
    launch_nnd_insert(st_, us_, row0, nb, n, window_start, seed, cs_, d_cnt_ + kFlagsAt, sms_,
                      [this](bool begin) { begin ? timed_begin(1) : timed_end(1); }, s);
  }
  // existing rows whose list changed, ascending
  compact_flags(st_.dirty, row0, -1, d_rows_, d_cnt_, d_tmp_, s);
  // the embedding phase in flight reads the published table until its
  // snapshot (overlap mode) and the embedding until it ends
  if (snap_pending_) ck(cudaStreamWaitEvent(s, ev_snap_, 0), "wait snapshot");
  else if (emb_pending_) ck(cudaStreamWaitEvent(s, ev_emb_, 0), "wait embedding");
  launch_adopt_and_publish(st_, row0, nb, d_rows_, d_cnt_, row0, n, s);
  if (defer_init_) {
    // the new rows' embedding waits for the phase in flight; it runs at the
    // start of this run's embedding phase
    init_pending_ = nb > 0;
    init_row0_ = (int)row0;
    init_nb_ = nb;
    init_n_ = (int)n;
  } else {
    if (emb_pending_) ck(cudaStreamWaitEvent(s, ev_emb_, 0), "wait embedding");
    launch_embed_init(st_, row0, nb, n, s);
  }
  const size_t nd = finish_phase("insertion", (size_t)row0);
  if (!defer_init_) emb_pending_ = snap_pending_ = false;  // the stream waited for it above
  // affected = batch rows then changed existing rows (insertion_kernel.cuh:1039-1089)
  for (int i = 0; i < nb; ++i) upd_q_.push((uint32_t)(row0 + i));
  for (size_t i = 0; i < nd; ++i) upd_q_.push(h_pin_[kCounters + i]);
  return (uint32_t)B;
}

// ---------------------------------------------------------------------------
// update (reference impl.cuh:255-333)
// ---------------------------------------------------------------------------
uint32_t Session::update(uint32_t n_ops, size_t &changed) {
  changed = 0;
  const size_t n = n_inserted_;
  if (n_ops == 0 || upd_done_ || n == 0) return 0;
  // the update republishes rows the embedding in flight reads (until its
  // snapshot in overlap mode) and changes working lists
  if (snap_pending_) ck(cudaStreamWaitEvent(stream_, ev_snap_, 0), "wait snapshot");
  else if (emb_pending_) ck(cudaStreamWaitEvent(stream_, ev_emb_, 0), "wait embedding");
  if (init_wait_) ck(cudaStreamWaitEvent(stream_, ev_init_, 0), "wait row embedding");
  init_wait_ = false;
  const size_t threshold = (size_t)(0.0001f * (float)n);
  uint32_t left = n_ops;
  while (left > 0) {
    std::vector<uint32_t> batch;
    if ((size_t)left >= n) {
      upd_q_.pop_n(upd_q_.size());
      batch.resize(n);
      std::iota(batch.begin(), batch.end(), 0u);
    } else if ((size_t)left >= upd_q_.size()) {
      batch = upd_q_.pop_n(upd_q_.size());
      std::vector<char> seen(n, 0);
      for (uint32_t v : batch) seen[v] = 1;
      std::uniform_int_distribution<uint32_t> dist(0, (uint32_t)(n - 1));
      uint32_t start = dist(rng_);
      while (batch.size() < (size_t)left) {
        const uint32_t c = (start++) % (uint32_t)n;
        if (!seen[c]) {
          seen[c] = 1;
          batch.push_back(c);
        }
      }
    } else {
      batch = upd_q_.pop_n(left);
    }
    if (batch.empty()) break;
    const size_t raw = batch.size();
    std::vector<uint32_t> affected;
    changed += update_round(batch, affected);
    left -= (uint32_t)raw;
    for (uint32_t v : affected) upd_q_.push(v);
    if (upd_q_.size() < threshold) {
      upd_done_ = (n == p_.n_instances);
      break;
    }
  }
  return n_ops - left;
}

// One UpdateAlgo::run (update_kernel.cuh:913-1054) on a batch.
size_t Session::update_round(std::vector<uint32_t> &batch, std::vector<uint32_t> &affected) {
  std::sort(batch.begin(), batch.end());
  batch.erase(std::unique(batch.begin(), batch.end()), batch.end());
  const int nb = (int)batch.size();
  const int n = (int)n_inserted_;
  cudaStream_t s = stream_;
  std::memcpy(h_pin_, batch.data(), (size_t)nb * sizeof(uint32_t));
  ck(cudaMemcpyAsync(d_batch_, h_pin_, (size_t)nb * sizeof(int), cudaMemcpyHostToDevice, s),
     "batch");
  int *counters = d_cnt_ + 2;  // after the report count (8-byte aligned)
  const size_t bound = join_pool_words(nb, st_.k);
  ensure_join(bound);
  bloom_clean_ = false;
  launch_join_nodes(st_, us_, d_batch_, nb, n, d_rows_, d_rows2_, counters, s);
  timed_begin(0);
  launch_local_join(st_, us_, d_rows_, d_rows2_, counters, join_pool_, join_words_, 0, n, s);
  if (bound > join_words_) {
    // the pool may not hold every block: as many passes as their words take
    ck(cudaMemcpyAsync(h_pin_, counters + kUpdPool, sizeof(uint64_t), cudaMemcpyDeviceToHost, s), "words");
    sync();
    uint64_t words = 0;
    std::memcpy(&words, h_pin_, sizeof(words));
    for (int pass = 1; (uint64_t)pass * join_words_ < words; ++pass)
      launch_local_join(st_, us_, d_rows_, d_rows2_, counters, join_pool_, join_words_, pass, n, s);
  }
  timed_end(0);
  launch_merge_publish(st_, n, counters + kUpdEdges, us_.hflag, s);
  compact_flags(us_.hflag, n, -1, d_rows_, d_cnt_, d_tmp_, s);
  const size_t na = finish_phase("update", (size_t)n);
  const int edges = (int)h_pin_[2 + kUpdEdges];
  affected.assign(h_pin_ + kCounters, h_pin_ + kCounters + na);
  return (size_t)edges;
}

// ---------------------------------------------------------------------------
// embedding (reference impl.cuh:335-500)
// ---------------------------------------------------------------------------
uint32_t Session::embed(uint32_t n_ops) {
  const size_t n = n_inserted_;
  if (n_ops == 0 || n == 0) return 0;
  const size_t total_n = p_.n_instances;
  std::vector<uint32_t> batch;
  if ((size_t)n_ops >= n) {
    emb_new_head_ = n_inserted_;
    batch.resize(n);
    std::iota(batch.begin(), batch.end(), 0u);
    emb_cursor_ = n - 1;
    if (emb_cursor_ == total_n - 1 && upd_done_) ++sweeps_;
  } else {
    for (size_t v = emb_new_head_; v < n_inserted_; ++v) batch.push_back((uint32_t)v);
    emb_new_head_ = n_inserted_;
    size_t left = batch.size() >= (size_t)n_ops ? 0 : (size_t)n_ops - batch.size();
    if (left > 0) {
      std::vector<char> seen(n, 0);
      for (uint32_t v : batch) seen[v] = 1;
      size_t cursor = (emb_cursor_ == SIZE_MAX) ? 0 : (emb_cursor_ + 1) % n;
      for (size_t checked = 0; left > 0 && checked < n; ++checked) {
        if (!seen[cursor]) {
          seen[cursor] = 1;
          batch.push_back((uint32_t)cursor);
          emb_cursor_ = cursor;
          if (emb_cursor_ == total_n - 1 && upd_done_) ++sweeps_;
          --left;
        }
        cursor = (cursor + 1) % n;
      }
    }
  }
  log("[GPUMAP] embed batch_size=%zu cursor=%zu\n", batch.size(), emb_cursor_);
  const int nb = (int)batch.size();
  const int ni = (int)n;
  const int k = st_.k;
  cudaStream_t s = stream_;
  if (p_.overlap) {
    // this phase takes the other side (stream, scratch, staging); it reads
    // the table the insertion just published
    std::swap(estream_, estream_alt_);
    std::swap(es_, es_alt_);
    std::swap(es_cnt_, es_cnt_alt_);
    std::swap(h_emb_pin_, h_emb_pin_alt_);
    std::swap(ev_hpin_, ev_hpin_alt_);
    ck(cudaEventRecord(ev_pub_, stream_), "record publish");
    ck(cudaStreamWaitEvent(estream_, ev_pub_, 0), "wait publish");
    s = estream_;
    // the side's staging was last read by the upload two phases ago
    ck(cudaEventSynchronize(ev_hpin_), "staging");
  }
  ensure_embed(es_, (size_t)nb);
  std::memcpy(h_emb_pin_, batch.data(), (size_t)nb * sizeof(uint32_t));
  ck(cudaMemcpyAsync(es_.batch, h_emb_pin_, (size_t)nb * sizeof(int), cudaMemcpyHostToDevice, s),
     "batch");
  if (p_.overlap) ck(cudaEventRecord(ev_hpin_, s), "record staging");
  const int euclid = p_.metric == GM_METRIC_EUCLIDEAN;
  const double target = std::log2((double)(k - 1));
  launch_fuzzy_graph(st_.pub_idx, st_.pub_dist, ni, k, euclid, es_.batch, nb, target, es_, s);
  if (sweeps_ > 2) emb_done_ = upd_done_;
  const uint64_t noise_seed = 42ull ^ (uint64_t)sweeps_;
  const int nu = ni - nb;
  const uint32_t *heur_idx = st_.pub_idx;
  const float *heur_dist = st_.pub_dist;
  // the rows the reposition step moves (those not in the batch) depend only
  // on the batch: queued before the phase waits for the previous one (after
  // the schedule, whose compaction shares the flag scratch)
  auto select_unsel = [&] {
    if (nu <= 0) return;
    ck(cudaMemsetAsync(es_.flag, 0, (size_t)ni * sizeof(int), s), "flags");
    launch_mark_rows(es_.batch, nb, es_.flag, s);
    compact_flags(es_.flag, ni, 0, es_.unsel, es_cnt_, es_.tmp, s);
  };
  if (!p_.overlap) {
    launch_add_noise(st_.emb, ni, es_.batch, nb, 0.001f, noise_seed, es_, s);
    launch_schedule(ni, nb, k, p_.alpha, (int)p_.max_epoch, (int)p_.negative_sample_rate, es_, s);
    select_unsel();
  } else {
    // the fuzzy set and schedule read only the published table: they run
    // beside the previous phase's SGD.  The reposition step reads the table
    // as it is now (a snapshot: the next insertion may publish before it
    // runs).  Noise, the new rows' embedding and the SGD read the embedding
    // and wait for the previous phase.
    launch_schedule(ni, nb, k, p_.alpha, (int)p_.max_epoch, (int)p_.negative_sample_rate, es_, s);
    select_unsel();
    if (nu > 0) {
      const size_t w = (size_t)ni * (size_t)(k + 1);
      ck(cudaMemcpyAsync(es_.pub_idx_snap, st_.pub_idx, w * sizeof(uint32_t), cudaMemcpyDeviceToDevice,
                         s), "snapshot");
      ck(cudaMemcpyAsync(es_.pub_dist_snap, st_.pub_dist, w * sizeof(float), cudaMemcpyDeviceToDevice,
                         s), "snapshot");
      heur_idx = es_.pub_idx_snap;
      heur_dist = es_.pub_dist_snap;
    }
    ck(cudaEventRecord(ev_snap_, s), "record snapshot");
    snap_pending_ = true;
    if (emb_pending_) ck(cudaStreamWaitEvent(s, ev_emb_, 0), "wait embedding");
    const bool init = init_pending_;
    if (init) launch_embed_init(st_, init_row0_, init_nb_, init_n_, s);
    launch_add_noise(st_.emb, ni, es_.batch, nb, 0.001f, noise_seed, es_, s);
    if (init) {
      // recorded last before the SGD: what waits for it (the next insertion's
      // screen) fills every SM, and a cooperative launch that comes after it
      // waits for half of them to drain (35 us a cycle when recorded before
      // the noise)
      ck(cudaEventRecord(ev_init_, s), "record row embedding");
      init_pending_ = false;
      init_wait_ = true;
    }
  }
  timed_begin(2, s);
  run_sgd((int)std::min<size_t>(2 * (size_t)nb * (size_t)k, INT32_MAX), s);
  timed_end(2, s);
  if (nu > 0) launch_heuristic(heur_idx, heur_dist, ni, k, euclid, es_.unsel, nu, st_.emb, es_, s);
  if (p_.overlap) {
    ck(cudaEventRecord(ev_emb_, s), "record embedding");
    emb_pending_ = true;
  }
  return (uint32_t)nb;
}

// A deferred embedding of new rows whose phase did not run: on the main
// stream, after the phase in flight.
void Session::flush_init() {
  if (!init_pending_) return;
  if (emb_pending_) ck(cudaStreamWaitEvent(stream_, ev_emb_, 0), "wait embedding");
  launch_embed_init(st_, init_row0_, init_nb_, init_n_, stream_);
  init_pending_ = false;
}

// The max_epoch SGD epochs of one embedding call: one cooperative launch
// with a grid barrier between epochs (sizes are read from device scalars).
void Session::run_sgd(int max_edges, cudaStream_t s) {
  if (p_.max_epoch == 0) return;
  // overlapped: half the SMs, the other half stays free for the next cycle's
  // distance work (the per-epoch time does not depend on it)
  const int max_ctas = p_.overlap ? std::max(1, sms_ / 2) : 0;
  ck(launch_sgd_persistent(st_.emb, es_.t_row, es_.flag_tail, es_.t_val, es_.next_s, es_.next_n,
                     es_.iscal, es_.fscal, max_edges, p_.alpha, 1.0f, p_.a, p_.b, (int)p_.max_epoch,
                     (int)p_.negative_sample_rate, 42ull, (unsigned *)(es_.iscal + kIscalBarrier),
                     st_.err, device_, s, st_.stat, max_ctas),
     "SGD launch");
}

void Session::close() {
  if (closed_) return;
  cudaStreamSynchronize(stream_);
  for (cudaStream_t q : {estream_, estream_alt_})
    if (q) cudaStreamSynchronize(q);
  emb_pending_ = snap_pending_ = init_wait_ = false;
  closed_ = true;
}

void Session::debug_scalars(int64_t *out, int cnt) const {
  int iscal[16] = {0};
  unsigned err = 0;
  cudaStreamSynchronize(stream_);
  for (cudaStream_t q : {estream_, estream_alt_})
    if (q) cudaStreamSynchronize(q);
  cudaMemcpy(iscal, es_.iscal, sizeof(iscal), cudaMemcpyDeviceToHost);
  cudaMemcpy(&err, st_.err, sizeof(err), cudaMemcpyDeviceToHost);
  unsigned long long wide = 0;
  cudaMemcpy(&wide, d_stat_ + 10, sizeof(wide), cudaMemcpyDeviceToHost);
  int64_t v[12] = {(int64_t)n_inserted_,
                   (int64_t)ins_head_,
                   (int64_t)emb_new_head_,
                   emb_cursor_ == SIZE_MAX ? -1 : (int64_t)emb_cursor_,
                   (int64_t)sweeps_,
                   iscal[0],
                   iscal[1],
                   iscal[2],
                   iscal[3],
                   (int64_t)upd_q_.size(),
                   (int64_t)err,
                   (int64_t)wide};
  for (int i = 0; i < cnt && i < 12; ++i) out[i] = v[i];
}

}  // namespace gm
