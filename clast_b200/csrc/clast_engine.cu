// clast_engine.cu -- host orchestration of the device path and the C ABI
// declared in include/clast_gpu.h.
//
// One context owns one CUDA stream and a scratch pool.  An index keeps its
// target window resident in HBM (bases with joints, padded with 'N', plus the
// hash table, the filter and the resolved entries).  A search runs the whole hit
// pipeline of CDeviceHitList (CDeviceHitList.cu:228-423) for a batch of query
// windows against a group of target windows with two host synchronisations (hit
// total, result total).
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <climits>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/clast_gpu.h"
#include "clast_device.cuh"
#include "clast_kernels.cuh"
#include "clast_workspace.h"
#include "clast_engine.h"

using namespace clast;

namespace clast {
thread_local cudaStream_t g_alloc_stream = nullptr;
}  // namespace clast





namespace {

template <class T>
T read_scalar(const T* dev, cudaStream_t st) {
  T v;
  CLAST_CK(cudaMemcpyAsync(&v, dev, sizeof(T), cudaMemcpyDeviceToHost, st));
  CLAST_CK(cudaStreamSynchronize(st));
  return v;
}

}  // namespace


namespace {

// CDeviceHashTable::CDeviceHashTable (CDeviceHashTable.cu:143-174) for the
// window whose padded bases are already in ix->bases.
// *failed (zeroed by the caller, read once all windows are queued) counts
// table records that fell outside the table.
void build_index_device(Workspace& ws, cudaStream_t st, const clast_params* p, clast_index* ix,
                        unsigned long long* failed) {
  const int l = p->lmer;
  const int64_t n = ix->n;
  const char* bases = ix->bases.p + kPad;
  uint64_t* packed = ws.get<uint64_t>("ix_packed", (size_t)(n / 32 + 4));
  uint64_t* nmask = ws.get<uint64_t>("ix_nmask", (size_t)(n / 64 + 4));
  pack_bases(bases, n, packed, nmask, st);
  const int64_t ns = n / p->stride;  // CDeviceHashTable.cu:34
  // samples sorted by code (equal keys adjacent, in window-position order):
  // one word code << pbits | position when both fit in 64 bits, else
  // (code, position) pairs
  int pbits = 1;
  while ((1ll << pbits) < ns) ++pbits;
  if (2 * l + 1 + pbits > 64) pbits = 0;
  uint64_t* items = ws.get<uint64_t>("ix_items", ns);
  uint64_t* items2 = ws.get<uint64_t>("ix_items2", ns);
  int32_t* pos = pbits ? nullptr : ws.get<int32_t>("ix_pos", ns);
  int32_t* pos2 = pbits ? nullptr : ws.get<int32_t>("ix_pos2", ns);
  sample_keys(packed, nmask, ns, p->stride, l, pbits, items, pos, st);
  const int in_alt = radix_sort_u64(ws, items, pos, items2, pos2, ns, pbits, pbits + 2 * l + 1, st);
  // From here on every array is sized for the ns samples (an upper bound of
  // the valid ones and of the kept ones), with no host synchronisation.
  // Hash table: buckets of two records, one bucket per sample, so at most half
  // of the records are used (84 % of the keys then sit in their home bucket),
  // plus a tail for the probe run past the last bucket
  const int64_t nb = std::max<int64_t>(1, ns);
  if (nb >= (int64_t)UINT32_MAX) throw std::invalid_argument("window has too many sampled l-mers");
  ix->nbuckets = (uint32_t)nb;
  ix->entries.alloc(ns);
  ix->kept.alloc(1);
  ix->n_records = 2 * nb + (1 << 16);
  ix->table.alloc((size_t)ix->n_records);
  if (!ix->filter_mem) {
    clast_index* one[1] = {ix};
    alloc_filters(one, 1, filter_shift(ns), st);
  }
  CLAST_CK(cudaMemsetAsync(ix->kept.p, 0, sizeof(int64_t), st));
  const size_t words = (size_t)index_state_words(ns, ix->n_records, p->cut_repeat);
  unsigned long long* state = ws.get<unsigned long long>("ix_state", words);
  CLAST_CK(cudaMemsetAsync(state, 0, words * sizeof(unsigned long long), st));
  index_place(in_alt ? items2 : items, in_alt ? pos2 : pos, ns, pbits, p->stride, l, p->cut_repeat, ix->gateway.p,
              ix->lengths.p, ix->nseqs, ix->nbuckets, ix->entries.p, ix->table.p, ix->n_records, ix->filter,
              ix->fshift, ix->fstride, state, reinterpret_cast<unsigned long long*>(ix->kept.p), failed, st);
  ix->n_keys = ns;
}

// Index of a window whose padded base array is already on the device (its
// filter memory set already, or none).
clast_index* make_index_resident(Workspace& ws, cudaStream_t st, const clast_params* p, DevArray<char>&& padded,
                                 int64_t n_bases, DevArray<int32_t>&& gateway, DevArray<int32_t>&& lengths,
                                 int32_t n_seqs, int32_t t_begin, unsigned long long* failed,
                                 std::unique_ptr<clast_index> ix = std::unique_ptr<clast_index>(new clast_index())) {
  ix->l = p->lmer;
  ix->stride = p->stride;
  ix->cut = p->cut_repeat;
  ix->t_begin = t_begin;
  ix->n = n_bases;
  ix->nseqs = n_seqs;
  ix->bases = std::move(padded);
  ix->gateway = std::move(gateway);
  ix->lengths = std::move(lengths);
  build_index_device(ws, st, p, ix.get(), failed);
  return ix.release();
}

// Index of a window given as host arrays (the reference's seam).
clast_index* make_index(clast_ctx* c, const clast_params* p, const char* bases, int64_t n_bases,
                        const int32_t* gateway, const int32_t* lengths, int32_t n_seqs, int32_t t_begin) {
  DevArray<char> padded;
  DevArray<int32_t> gw, ln;
  gw.alloc(n_seqs);
  ln.alloc(n_seqs);
  padded.alloc((size_t)n_bases + 2 * kPad);
  CLAST_CK(cudaEventRecord(c->ev0, c->st));
  CLAST_CK(cudaMemsetAsync(padded.p, 'N', (size_t)n_bases + 2 * kPad, c->st));
  if (n_bases > 0) CLAST_CK(cudaMemcpyAsync(padded.p + kPad, bases, (size_t)n_bases, cudaMemcpyHostToDevice, c->st));
  if (n_seqs > 0) {
    CLAST_CK(cudaMemcpyAsync(gw.p, gateway, n_seqs * sizeof(int32_t), cudaMemcpyHostToDevice, c->st));
    CLAST_CK(cudaMemcpyAsync(ln.p, lengths, n_seqs * sizeof(int32_t), cudaMemcpyHostToDevice, c->st));
  }
  CLAST_CK(cudaEventRecord(c->ev1, c->st));
  const int64_t k0 = g_kernel_launches;
  unsigned long long* failed = reinterpret_cast<unsigned long long*>(c->ws.get<int64_t>("ix_failed", 1));
  CLAST_CK(cudaMemsetAsync(failed, 0, sizeof(unsigned long long), c->st));
  std::unique_ptr<clast_index> ix(make_index_resident(c->ws, c->st, p, std::move(padded), n_bases, std::move(gw),
                                                      std::move(ln),
                                                      n_seqs, t_begin, failed));
  CLAST_CK(cudaEventRecord(c->ev2, c->st));
  CLAST_CK(cudaEventSynchronize(c->ev2));
  if (read_scalar(reinterpret_cast<int64_t*>(failed), c->st) != 0) throw std::runtime_error("index table overflow");
  float up = 0, bd = 0;
  CLAST_CK(cudaEventElapsedTime(&up, c->ev0, c->ev1));
  CLAST_CK(cudaEventElapsedTime(&bd, c->ev1, c->ev2));
  c->stats.index_upload_ms += up;
  c->stats.index_ms += bd;
  c->stats.index_launches += g_kernel_launches - k0;
  return ix.release();
}

// Device-resident query strands of one batch, packed once for every index: one
// allocation with the padded bases, the 2-bit words and the strand tables.
struct QueryRef;

struct QueryBatch {
  DevArray<char> mem;
  char* bases = nullptr;  // padded
  int64_t n = 0;
  int64_t* start = nullptr;
  int32_t* len = nullptr;
  uint64_t *packed = nullptr, *nmask = nullptr;
  int32_t nstrands = 0;
  char* meta = nullptr;             // the caller's tables, directly behind len
  const int32_t* wstart = nullptr;  // strand index where each window starts, plus the end
  int32_t nwin = 0;
  int32_t min_len = 0, max_len = 0;  // strand lengths (the DP orders hits by rows when they differ)
  static size_t al(size_t b) { return (b + 255) & ~size_t(255); }
  void alloc(int64_t n_bases, int64_t strands, size_t meta_bytes) {
    n = n_bases;
    nstrands = (int32_t)strands;
    const size_t sz[5] = {al((size_t)n + 2 * kPad), al((size_t)(n / 32 + 4) * 8), al((size_t)(n / 64 + 4) * 8),
                          al((size_t)strands * 8), al((size_t)strands * 4)};
    mem.alloc(sz[0] + sz[1] + sz[2] + sz[3] + sz[4] + meta_bytes);
    char* at = mem.p;
    bases = at;
    packed = reinterpret_cast<uint64_t*>(at += sz[0]);
    nmask = reinterpret_cast<uint64_t*>(at += sz[1]);
    start = reinterpret_cast<int64_t*>(at += sz[2]);
    len = reinterpret_cast<int32_t*>(at += sz[3]);
    meta = at + sz[4];
  }
  QueryView view() const {
    QueryView q;
    q.bases = bases + kPad;
    q.n = n;
    q.packed = packed;
    q.nmask = nmask;
    q.start = start;
    q.len = len;
    q.nstrands = nstrands;
    return q;
  }
  void pack(cudaStream_t st) { pack_bases(bases + kPad, n, packed, nmask, st); }
  QueryRef ref() const;
};

// A query batch as the seeding and search stages read it, without ownership
// (a QueryBatch, or clast_search_noalloc's buffers in its fixed scratch).
struct QueryRef {
  QueryView q;
  int64_t n = 0;                     // bases of the strands
  const int32_t* wstart = nullptr;   // strand where each query window starts, plus the end
  int32_t nwin = 0;
  int32_t min_len = 0, max_len = 0;  // strand lengths (the DP orders hits by rows when they differ)
  const int32_t* lens = nullptr;     // the same on the host once the stream has run so far, when given
};

QueryRef QueryBatch::ref() const {
  QueryRef r;
  r.q = view();
  r.n = n;
  r.wstart = wstart;
  r.nwin = nwin;
  r.min_len = min_len;
  r.max_len = max_len;
  return r;
}

// Where search_group puts a group's final hits: take(F, foff, nr) returns the
// arrays for its F hits (and may keep the nr + 1 per-read offsets), or throws
// when they do not fit.
struct HitSink {
  virtual ~HitSink() = default;
  virtual OutView take(int64_t F, const int64_t* foff, int64_t nr, cudaStream_t st) = 0;
};

// A group of target windows searched together, and the limits of its seed
// partitions.
struct Group {
  int nw = 0;
  bool reads = false;             // the strands are reads and their reverse complements, pair by pair
  const clast_index* ix[kMaxSeedWins] = {};
  int32_t load[kMaxSeedWins] = {};
  int64_t part_cap = 0;           // seeds per partition to begin with
  int64_t part_fit = INT64_MAX;   // most the scratch holds (arena mode)
};

// Waits for streams when the scope that holds it is left by an exception: what
// it holds may still be read or written by work queued there.
struct UnwindSync {
  std::vector<cudaStream_t> streams;
  int pending = std::uncaught_exceptions();
  UnwindSync(std::initializer_list<cudaStream_t> s) : streams(s) {}
  ~UnwindSync() {
    if (std::uncaught_exceptions() == pending) return;
    for (cudaStream_t s : streams) cudaStreamSynchronize(s);
    (void)cudaGetLastError();
  }
};

// A group's hits do not fit the 32-bit words of the DP's order.
struct TooManyHits : std::invalid_argument {
  using std::invalid_argument::invalid_argument;
};

// Host copy of the group's counters: waits for the stream.
const GroupCtl& read_ctl(clast_ctx* c, const GroupCtl* dev, cudaStream_t st) {
  CLAST_CK(cudaMemcpyAsync(c->ctl, dev, sizeof(GroupCtl), cudaMemcpyDeviceToHost, st));
  CLAST_CK(cudaStreamSynchronize(st));
  return *c->ctl;
}

// CDeviceHitList for every query window of `qb` against every window of the
// group: seeds, seed filters, DP, result order.  The host waits twice, for the
// hit count and for the result count; every stage runs once for all windows of
// the group, so a small batch pays for some fifteen launches instead of
// twenty-odd per window.  A group whose seed partitions overflowed is seeded
// again with partitions sized from the exact counts.  Returns the results.
int64_t search_group(clast_ctx* c, Workspace& ws, const clast_params* p, const QueryRef& qb, Group& g, HitSink& sink) {
  cudaStream_t st = c->st;
  const QueryView q = qb.q;
  const int nw = g.nw;
  const int64_t nv = (int64_t)q.nstrands * nw, nr = q.nstrands / 2;
  StageTimer& tm = c->timer;
  const size_t mark = ws.arena_used;  // arena mode: everything below is this group's
  // counters and scan states, zeroed together
  const int64_t st1 = scan_state_words(nv), st2 = scan_state_words(nr);
  const size_t ctl_bytes = (sizeof(GroupCtl) + 255) & ~size_t(255);
  const size_t zero_bytes = ctl_bytes + (size_t)(st1 + st2) * sizeof(unsigned long long);
  GroupCtl* ctl = nullptr;
  unsigned long long *state1 = nullptr, *state2 = nullptr;
  int64_t *off = nullptr, *hoff = nullptr;
  int32_t *cnt = nullptr, *nvalid = nullptr, *hcnt = nullptr;
  uint64_t* skey = nullptr;
  uint32_t* sq = nullptr;
  FirstSeeds first{};
  int64_t H = 0;
  for (int attempt = 0;; ++attempt) {
    off = ws.get<int64_t>("s_off", nv);
    cnt = ws.get<int32_t>("s_cnt", nv);
    nvalid = ws.get<int32_t>("s_nvalid", nv);
    skey = ws.get<uint64_t>("s_key", (size_t)g.part_cap * kSeedParts * nw);
    sq = ws.get<uint32_t>("s_q", (size_t)g.part_cap * kSeedParts * nw);
    char* zero = ws.get<char>("s_ctl", zero_bytes);
    ctl = reinterpret_cast<GroupCtl*>(zero);
    state1 = reinterpret_cast<unsigned long long*>(zero + ctl_bytes);
    state2 = state1 + st1;
    hcnt = ws.get<int32_t>("s_hcnt", nv);
    hoff = ws.get<int64_t>("s_hoff", nv + 1);
    uint32_t* lists = ws.get<uint32_t>("s_lists", 3 * nv);
    uint64_t* first_key = nullptr;
    uint32_t* first_q = nullptr;
    CLAST_CK(cudaMemsetAsync(zero, 0, zero_bytes, st));
    tm.begin(st);
    if (!g.reads) {  // any strands, one window
      seed_fused(q, g.ix[0]->view(), g.ix[0]->tview(), p->gap, p->local, ctl->cursor, ctl->kmers[0], off, cnt, nvalid,
                 skey, sq, g.part_cap, st);
    } else {
      first_key = ws.get<uint64_t>("s_first", nv);
      first_q = ws.get<uint32_t>("s_firstq", nv);
      SeedWins W{};
      for (int w = 0; w < nw; ++w) {
        W.w[w] = SeedWin{g.ix[w]->view(), g.ix[w]->tview(), ctl->kmers[w], ctl->seeds[w], 0};
        W.w[w].paired = w % 2 == 1 && g.ix[w]->filter_mem == g.ix[w - 1]->filter_mem &&
                        g.ix[w]->filter == g.ix[w - 1]->filter + 1;
      }
      W.cursor = ctl->cursor;
      W.off = off;
      W.cnt = cnt;
      W.nvalid = nvalid;
      W.hcnt = hcnt;
      W.first_key = first_key;
      W.first_q = first_q;
      W.lists = lists;
      W.n_listed = ctl->n_seeds;
      W.long_reads = ws.get<uint32_t>("s_long", nr);
      W.n_long = ctl->n_stored;
      W.words = 1;
      for (int w = 0; w < nw; ++w)
        if (g.ix[w]->nseqs >= (1 << 20)) W.words = 0;
      W.skey = skey;
      W.sq = sq;
      W.part_cap = g.part_cap;
      seed_reads(q, W, nw, p->width, p->gap, p->local, qb.lens ? INT_MAX : qb.max_len, st);
    }
    first = FirstSeeds{first_key, first_q, nvalid, cnt};
    tm.end(StageTimer::SEED, st);
    // sortSeeds, deletingIsolateSeeds, deleteDuplicateSeeds
    tm.begin(st);
    seed_filter(skey, sq, off, cnt, nvalid, first_q, qb.wstart, qb.nwin, nw, p->width, p->gap, nv, lists, hcnt,
                g.part_cap * nw, ctl, st);
    tm.end(StageTimer::SORT, st, 4);
    scan_i32_to(hcnt, nv, hoff, state1, &ctl->hits, st);
    const GroupCtl& h = read_ctl(c, ctl, st);
    tm.flush();
    int64_t most = 0, kmers = 0, S = 0, stored = 0;
    for (int i = 0; i < kSeedParts; ++i) {
      most = std::max<int64_t>(most, (int64_t)h.cursor[i]);
      stored += (int64_t)h.cursor[i];
      for (int w = 0; w < nw; ++w) {
        kmers += (int64_t)h.kmers[w][i];
        S += (int64_t)h.seeds[w][i];
      }
    }
    if (!g.reads) S = stored;
    if (most <= g.part_cap * nw) {
      c->stats.query_kmers += kmers;
      c->stats.seeds += S;
      c->seed_hint = std::max<int64_t>(c->seed_hint, (stored + stored / 4) / nw);
      H = h.hits;
      break;
    }
    if (attempt > 0) throw std::runtime_error("seed partitions overflowed twice");
    if (most > g.part_fit)  // the partitions this window needs do not fit the scratch
      throw std::invalid_argument("query window needs seed partitions of " + std::to_string(most) +
                                  " seeds; clast_search_noalloc's scratch holds " + std::to_string(g.part_fit) +
                                  " (use clast_search)");
    if (ws.arena) ws.arena_rewind(mark);
    g.part_cap = (most + nw - 1) / nw;  // strands past a full partition wrote nothing: run again
    // a little more the next time (the workspace takes a quarter more anyway):
    // few reads with many seeds each fill some partitions far above the mean
    c->part_hint = std::max(c->part_hint, g.part_cap + g.part_cap / 8);
  }
  if (H >= ((int64_t)1 << 32)) throw TooManyHits("more than 2^32 hits in one window");
  c->stats.hits += H;
  if (H == 0) return 0;
  uint64_t* hk = ws.get<uint64_t>("h_key", H);
  int32_t* hq = ws.get<int32_t>("h_q", H);
  uint32_t* hs = ws.get<uint32_t>("h_s", H);
  gather_hits(skey, sq, off, hcnt, hoff, nv, nw, hk, hq, hs, q.len, p->lmer, 2 * p->gap + 1, first, ctl, st);
  // alignmentHits + calculateEvalue + deleteHits_lowEValue / _tooShort
  DpOut o;
  o.t_idx = ws.get<int32_t>("d_tidx", H);
  o.q_idx = ws.get<int32_t>("d_qidx", H);
  o.t_len = ws.get<int32_t>("d_tlen", H);
  o.q_len = ws.get<int32_t>("d_qlen", H);
  o.match = ws.get<int32_t>("d_match", H);
  o.score = ws.get<int32_t>("d_score", H);
  o.evalue = ws.get<double>("d_e", H);
  o.keep = ws.get<uint8_t>("d_keep", H);
  DpParams dp{p->lmer, p->stride, p->gap, p->local, p->cutoff, p->total_db, p->K, p->lambda};
  // Reads of different lengths: the DP takes the hits longest first, so that a
  // warp's hits have about the same number of rows (the reference sorts them
  // by rows before aligning too, CDeviceHitList_alignmentHits.cu:10-58), by an
  // exact sort of the row counts.  (Length buckets in one counting pass take
  // 0.10 against 0.15 ms for 130,000 hits, but their DP 3.68 against 3.66 ms,
  // and 17.3 against 17.0 ms on 200,000 reads of 50 bp - 10 kbp; a persistent
  // grid taking hits from a queue is slower than the plain one, 17.7 and 4.2 ms.)
  // The longest hits of the order may run one per warp (banded_dp decides
  // from the length buckets, or for equal lengths from the row count).
  const int min_len = qb.lens ? qb.lens[0] : qb.min_len, max_len = qb.lens ? qb.lens[1] : qb.max_len;
  const bool uneven = max_len != min_len && H > 1;
  const int warp_mode = dp_warp_mode_from_env(c->dp_warp);
  const bool long_hits = uneven && max_len - p->lmer >= kDpMaxThreadRows;
  c->stats.dp_order_kind = uneven ? 1 : 0;
  c->stats.dp_queue_chunk = 0;
  DpBuckets buckets;
  const uint64_t* order = nullptr;
  if (uneven) {
    tm.begin(st);
    const int rows_max = std::max(1, max_len - p->lmer + 1);
    int bits = 1;
    while ((1ll << bits) <= rows_max) ++bits;
    uint64_t* ok = ws.get<uint64_t>("h_order", H);
    uint64_t* ok2 = ws.get<uint64_t>("h_order2", H);
    dp_order_keys(hs, nw, q.len, H, p->lmer, rows_max, ok, st);
    order = radix_sort_u64(ws, ok, nullptr, ok2, nullptr, H, 32, 32 + bits, st) ? ok2 : ok;
    if (warp_mode == kDpWarpAuto || long_hits) buckets = dp_bucket_count(ws, hs, nw, q.len, H, p->lmer, st);
    tm.end(StageTimer::DPORDER, st);
  }
  tm.begin(st);
  DpLaunch dl;
  dl.warp = warp_mode;
  dl.long_hits = long_hits;
  dl.buckets = buckets;
  dl.warp_n = &ctl->dp_warp;
  dl.aux = c->st_dp;
  dl.ev_fork = c->ev_dp_fork;
  dl.ev_join = c->ev_dp_join;
  dl.bad = &ctl->bad;
  if (!uneven) dl.uniform_rows = std::max(0, max_len - p->lmer);
  TargetView tv[kMaxSeedWins];
  for (int w = 0; w < nw; ++w) tv[w] = g.ix[w]->tview();
  const long long warp_fixed = banded_dp(tv, nw, q, hk, hq, hs, order, H, dp, o, st, dl);
  tm.end(StageTimer::DP, st);
  // resultSorting + deleteHits_duplicateResult, per read
  tm.begin(st);
  uint64_t* g1 = ws.get<uint64_t>("f_g1", H);
  uint64_t* g2 = ws.get<uint64_t>("f_g2", H);
  int32_t* fsel = ws.get<int32_t>("f_sel", H);
  int32_t* fcnt = ws.get<int32_t>("f_cnt", nr);
  uint32_t* flist = ws.get<uint32_t>("f_list", nr);
  final_order(hk, hq, hs, o, hoff, nr, nw, g1, g2, flist, fcnt, fsel, ctl, st);
  int64_t* foff = ws.get<int64_t>("f_off", nr + 1);
  scan_i32_to(fcnt, nr, foff, state2, &ctl->results, st);
  tm.end(StageTimer::FINAL, st, 3);
  const GroupCtl& h = read_ctl(c, ctl, st);
  tm.flush();
  const int64_t F = h.results;
  c->stats.results += F;
  c->stats.dp_cells += (int64_t)h.cells;
  c->stats.dp_warp_hits += warp_fixed >= 0 ? warp_fixed : h.dp_warp;
  if (h.bad) throw std::runtime_error("internal: a hit named a target sequence or strand outside the window");
  if (F == 0) return 0;
  OutView out = sink.take(F, foff, nr, st);
  for (int w = 0; w < nw; ++w) {
    out.t_first[w] = g.ix[w]->t_begin;
    out.load[w] = g.load[w];
  }
  final_write(hk, hs, o, hoff, nr, nw, fcnt, fsel, foff, out, st);
  return F;
}

// Tables on their way up: in the context's pinned staging buffer, or, larger than
// that may be, in pageable memory (a copy from there returns once it has been read).
struct HostTables {
  clast_ctx* c;
  std::vector<char> own;
  char* p;
  HostTables(clast_ctx* ctx, size_t bytes) : c(ctx), own(bytes <= kStageMax ? 0 : bytes) {
    p = own.empty() ? c->stage(bytes) : own.data();
  }
  void upload(void* dev, size_t bytes, cudaStream_t st) {
    CLAST_CK(cudaMemcpyAsync(dev, p, bytes, cudaMemcpyHostToDevice, st));
    if (own.empty()) c->staged(st);
  }
};

// Seeds per partition that a group begins with.
int64_t first_part_cap(const clast_ctx* c, int64_t n_bases) {
  return std::max<int64_t>(c->seed_hint, n_bases / 16 + (1 << 20)) / kSeedParts + 1;
}

// One search's results in device memory of their own, with the per-read
// offsets kept when the results are to be merged.
struct SlabSink : HitSink {
  ResultSlab slab;
  int32_t n_loads;
  bool keep_offsets;
  const int64_t* foff = nullptr;  // the group's per-read offsets (scratch), until the next group
  DevArray<int64_t> offsets;
  SlabSink(int32_t loads, bool keep) : n_loads(loads), keep_offsets(keep) {}
  OutView take(int64_t F, const int64_t* f, int64_t nr, cudaStream_t st) override {
    slab.alloc(F, n_loads);
    foff = f;
    if (keep_offsets) {
      offsets.alloc(nr + 1);
      CLAST_CK(cudaMemcpyAsync(offsets.p, f, (nr + 1) * sizeof(int64_t), cudaMemcpyDeviceToDevice, st));
    }
    return slab.view();
  }
};

}  // namespace

// ----------------------------------------------------------------------------
// targets / map: whole job with resident indexes
// ----------------------------------------------------------------------------

namespace clast {

int filter_shift(int64_t ns) {
  int fbits = 27;
  if (const char* e = std::getenv("CLAST_FILTER_BITS")) fbits = std::max(16, std::min(32, std::atoi(e)));
  int bits = 12;
  while (bits < fbits && (1ll << bits) < ns * 24) ++bits;
  return 64 - (bits - 5);
}

void alloc_filters(clast_index* const* ix, int n, int fshift, cudaStream_t st) {
  auto mem = std::make_shared<DevArray<uint32_t>>();
  const size_t words = (size_t)n << (64 - fshift);
  mem->alloc(words);
  CLAST_CK(cudaMemsetAsync(mem->p, 0, words * sizeof(uint32_t), st));
  for (int k = 0; k < n; ++k) {
    ix[k]->filter_mem = mem;
    ix[k]->filter = mem->p + k;
    ix[k]->fstride = n;
    ix[k]->fshift = fshift;
  }
}

// Waits for the index builds of clast_targets_create (once), records their
// time in the context's stats and reports a table overflow.
void settle_targets(clast_ctx* ctx, const clast_targets* T) {
  if (T->settled) return;
  CLAST_CK(cudaEventSynchronize(T->ev_done));
  T->settled = true;
  float up = 0, bd = 0;
  CLAST_CK(cudaEventElapsedTime(&up, T->ev_start, T->ev_up));
  CLAST_CK(cudaEventElapsedTime(&bd, T->ev_up, T->ev_done));
  ctx->stats.index_upload_ms = up;
  ctx->stats.index_ms = bd;
  ctx->stats.index_launches = T->launches;
  if (read_scalar(reinterpret_cast<const int64_t*>(T->failed.p), ctx->st) != 0)
    throw std::runtime_error("index table overflow");
  ctx->stats.index_bases = ctx->stats.index_keys = 0;
  for (const auto& w : T->wins) {
    ctx->stats.index_bases += w.ix->n;
    if (w.ix->kept.p) ctx->stats.index_keys += read_scalar(w.ix->kept.p, ctx->st);
  }
}

}  // namespace clast

namespace {


// One read window list per query load (moveQueryWindow, CHostSchedular.cu:12-23):
// the window [qb, qe) grows while gateway(2*qe+2) - gateway(2*qb) < q_vram,
// where every read adds two strands of len + l - 1 bases.  With the prefix
// sums cum(j), which the read offsets give, qe = clamp(first j with cum(j) >=
// cum(qb) + q_vram, minus one, to [qb + 1, n]).
void query_windows(const int64_t* offsets, int64_t r0, int64_t r1, int l, int32_t q_vram,
                   std::vector<int64_t>& win_first_read) {
  const int64_t n = r1 - r0;
  auto cum = [&](int64_t j) { return 2 * ((offsets[r0 + j] - offsets[r0]) + j * (l - 1)); };
  for (int64_t qb = 0; qb < n;) {
    const int64_t lim = cum(qb) + (int64_t)q_vram;
    int64_t lo = qb, hi = n + 1;  // first j in [qb, n] with cum(j) >= lim, n + 1 when there is none
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (mid <= n && cum(mid) < lim) lo = mid + 1;
      else hi = mid;
    }
    const int64_t qe = std::max(qb + 1, std::min(n, lo - 1));
    win_first_read.push_back(r0 + qb);
    qb = qe;
  }
}

}  // namespace

extern "C" {

int clast_ctx_create(int device, clast_ctx** out) {
  if (!out) return CLAST_ERR_ARG;
  *out = nullptr;
  std::unique_ptr<clast_ctx> c(new (std::nothrow) clast_ctx());
  if (!c) return CLAST_ERR_NOMEM;
  c->device = device;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    (void)cudaGetLastError();
    return CLAST_ERR_CUDA;
  }
  if (device < 0 || device >= ndev) return CLAST_ERR_ARG;
  if (cudaSetDevice(device) != cudaSuccess) return CLAST_ERR_CUDA;
  if (cudaStreamCreateWithFlags(&c->st, cudaStreamNonBlocking) != cudaSuccess) return CLAST_ERR_CUDA;
  if (cudaStreamCreateWithFlags(&c->st_copy, cudaStreamNonBlocking) != cudaSuccess) return CLAST_ERR_CUDA;
  if (cudaStreamCreateWithFlags(&c->st_dp, cudaStreamNonBlocking) != cudaSuccess) return CLAST_ERR_CUDA;
  if (cudaEventCreateWithFlags(&c->ev_stage, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&c->ev_dp_fork, cudaEventDisableTiming) != cudaSuccess ||
      cudaEventCreateWithFlags(&c->ev_dp_join, cudaEventDisableTiming) != cudaSuccess)
    return CLAST_ERR_CUDA;
  for (int b = 0; b < kBuildStreams; ++b)
    if (cudaStreamCreateWithFlags(&c->st_build[b], cudaStreamNonBlocking) != cudaSuccess) return CLAST_ERR_CUDA;
  // here and not with the first search, which may be one that must not allocate
  if (cudaMallocHost(reinterpret_cast<void**>(&c->ctl), sizeof(GroupCtl) + 2 * sizeof(int32_t)) != cudaSuccess) {
    (void)cudaGetLastError();
    c->ctl = nullptr;
    return CLAST_ERR_NOMEM;
  }
  c->lens = reinterpret_cast<int32_t*>(c->ctl + 1);
  {  // keep freed pool memory for reuse by later calls of this process
    cudaMemPool_t pool;
    if (cudaDeviceGetDefaultMemPool(&pool, device) == cudaSuccess) {
      uint64_t keep = UINT64_MAX;
      cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    (void)cudaGetLastError();
  }
  if (cudaEventCreate(&c->ev0) != cudaSuccess || cudaEventCreate(&c->ev1) != cudaSuccess ||
      cudaEventCreate(&c->ev2) != cudaSuccess || cudaEventCreate(&c->ev3) != cudaSuccess)
    return CLAST_ERR_CUDA;
  *out = c.release();
  return CLAST_OK;
}

void clast_ctx_destroy(clast_ctx* ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  for (auto& a : ctx->arenas) a->dev.slab.mem.release();  // device copies of results, freed on the stream before it goes
  if (ctx->st) cudaStreamSynchronize(ctx->st);
  for (int b = 0; b < kBuildStreams; ++b)
    if (ctx->st_build[b]) cudaStreamSynchronize(ctx->st_build[b]);
  ctx->ws.release_all();
  for (auto& w : ctx->ws_build) w.release_all();
  for (auto& a : ctx->arenas)
    if (a->p) cudaFreeHost(a->p);
  for (auto& a : ctx->tsv_arenas)
    if (a->p) cudaFreeHost(a->p);
  if (ctx->st_copy) cudaStreamSynchronize(ctx->st_copy);
  if (ctx->staging) cudaFreeHost(ctx->staging);
  if (ctx->ctl) cudaFreeHost(ctx->ctl);
  if (ctx->ev_stage) cudaEventDestroy(ctx->ev_stage);
  if (ctx->ev0) cudaEventDestroy(ctx->ev0);
  if (ctx->ev1) cudaEventDestroy(ctx->ev1);
  if (ctx->ev2) cudaEventDestroy(ctx->ev2);
  if (ctx->ev3) cudaEventDestroy(ctx->ev3);
  if (ctx->ev_dp_fork) cudaEventDestroy(ctx->ev_dp_fork);
  if (ctx->ev_dp_join) cudaEventDestroy(ctx->ev_dp_join);
  if (ctx->st_dp) {
    cudaStreamSynchronize(ctx->st_dp);
    cudaStreamDestroy(ctx->st_dp);
  }
  if (ctx->st_copy) {
    cudaStreamSynchronize(ctx->st_copy);
    cudaStreamDestroy(ctx->st_copy);
  }
  for (int b = 0; b < kBuildStreams; ++b)
    if (ctx->st_build[b]) cudaStreamDestroy(ctx->st_build[b]);
  if (ctx->st) cudaStreamDestroy(ctx->st);
  delete ctx;
}

const char* clast_last_error(const clast_ctx* ctx) { return ctx ? ctx->err.c_str() : "null context"; }

int clast_index_build(clast_ctx* ctx, const clast_params* p, const char* bases, int64_t n_bases,
                      const int32_t* gateway, const int32_t* lengths, int32_t n_seqs, int32_t t_begin,
                      clast_index** out) {
  if (!ctx || !out) return CLAST_ERR_ARG;
  *out = nullptr;
  return guarded(ctx, [&]() -> int {
    check_params(p);
    if (n_bases < 0 || n_seqs < 0 || (n_bases > 0 && !bases) || (n_seqs > 0 && (!gateway || !lengths)))
      throw std::invalid_argument("bad window arrays");
    if (n_bases >= INT32_MAX) throw std::invalid_argument("window larger than 2^31 bases");
    CLAST_CK(cudaSetDevice(ctx->device));
    g_alloc_stream = ctx->st;
    g_kernel_launches = 0;
    ctx->stats.index_ms = ctx->stats.index_upload_ms = 0;
    ctx->stats.index_launches = 0;
    *out = make_index(ctx, p, bases, n_bases, gateway, lengths, n_seqs, t_begin);
    return CLAST_OK;
  });
}

void clast_index_free(clast_index* ix) { delete ix; }

int clast_search(clast_ctx* ctx, const clast_index* ix, const clast_params* p, const char* q_bases,
                 int64_t n_qbases, const int32_t* q_gateway, const int32_t* q_lengths, int32_t n_qseqs,
                 int32_t q_begin, clast_hits* out) {
  if (!ctx || !out) return CLAST_ERR_ARG;
  std::memset(out, 0, sizeof(*out));
  return guarded(ctx, [&]() -> int {
    check_params(p);
    if (!ix) throw std::invalid_argument("index is null");
    if (p->lmer != ix->l || p->stride != ix->stride || p->cut_repeat != ix->cut)
      throw std::invalid_argument("params differ from the ones the index was built with");
    if (n_qseqs < 0 || (n_qseqs & 1) || (q_begin & 1))
      throw std::invalid_argument("query windows hold whole reads: n_qseqs and q_begin must be even");
    if (n_qbases < 0 || (n_qbases > 0 && !q_bases) || (n_qseqs > 0 && (!q_gateway || !q_lengths)))
      throw std::invalid_argument("bad query arrays");
    CLAST_CK(cudaSetDevice(ctx->device));
    g_alloc_stream = ctx->st;
    g_kernel_launches = 0;
    cudaStream_t st = ctx->st;
    int32_t min_len = n_qseqs ? INT32_MAX : 0, max_len = 0;
    // strand starts and lengths and the one query window, staged behind each other as on the device
    const size_t len_at = QueryBatch::al((size_t)n_qseqs * sizeof(int64_t));
    const size_t win_at = len_at + QueryBatch::al((size_t)n_qseqs * sizeof(int32_t));
    const size_t table_bytes = win_at + 2 * sizeof(int32_t);
    HostTables tables(ctx, table_bytes);
    char* host_tables = tables.p;
    int64_t* start = reinterpret_cast<int64_t*>(host_tables);
    for (int32_t i = 0; i < n_qseqs; ++i) {
      start[i] = q_gateway[i];
      if (q_gateway[i] < 0 || q_lengths[i] < 0 || (int64_t)q_gateway[i] + q_lengths[i] > n_qbases)
        throw std::invalid_argument("query sequence outside the base array");
      min_len = std::min(min_len, q_lengths[i]);
      max_len = std::max(max_len, q_lengths[i]);
    }
    if (n_qseqs) std::memcpy(host_tables + len_at, q_lengths, n_qseqs * sizeof(int32_t));
    const int32_t ws2[2] = {0, n_qseqs};
    std::memcpy(host_tables + win_at, ws2, sizeof(ws2));
    QueryBatch qb;
    qb.alloc(n_qbases, n_qseqs, sizeof(ws2));
    qb.min_len = min_len;
    qb.max_len = max_len;
    qb.nwin = 1;
    qb.wstart = reinterpret_cast<const int32_t*>(qb.meta);
    tables.upload(qb.start, table_bytes, st);
    CLAST_CK(cudaMemsetAsync(qb.bases, 'N', kPad, st));
    CLAST_CK(cudaMemsetAsync(qb.bases + kPad + n_qbases, 'N', kPad, st));
    if (n_qbases > 0)
      CLAST_CK(cudaMemcpyAsync(qb.bases + kPad, q_bases, (size_t)n_qbases, cudaMemcpyHostToDevice, st));
    qb.pack(st);
    struct SearchSink : HitSink {
      ResultSlab slab;
      int32_t q_first;
      explicit SearchSink(int32_t q) : q_first(q) {}
      OutView take(int64_t F, const int64_t*, int64_t, cudaStream_t) override {
        slab.alloc(F, 0);
        OutView v = slab.view();
        v.q_id = v.read;
        v.q_first = q_first;
        return v;
      }
    } sink(q_begin);
    int64_t F = 0;
    if (n_qseqs > 0 && ix->n_keys != 0) {
      Group g;
      g.nw = 1;
      g.ix[0] = ix;
      g.part_cap = std::max(first_part_cap(ctx, n_qbases), ctx->part_hint);
      F = search_group(ctx, ctx->ws, p, qb.ref(), g, sink);
    }
    out->n = F;
    // small results: one download into the pinned staging buffer
    const ResultSlab& h = sink.slab;  // q_id in the place of read
    const char* host = nullptr;
    if (F && h.bytes <= kStageMax) {
      char* to = ctx->stage(h.bytes);
      CLAST_CK(cudaMemcpyAsync(to, h.mem.p, h.bytes, cudaMemcpyDeviceToHost, st));
      CLAST_CK(cudaStreamSynchronize(st));
      host = to;
    }
    auto copy = [&](auto*& dst, const auto* dev) {
      dst = static_cast<std::remove_reference_t<decltype(dst)>>(std::malloc((F ? F : 1) * sizeof(*dst)));
      if (!dst) throw std::bad_alloc();
      if (host) std::memcpy(dst, host + (reinterpret_cast<const char*>(dev) - h.mem.p), F * sizeof(*dst));
      else if (F) CLAST_CK(cudaMemcpyAsync(dst, dev, F * sizeof(*dst), cudaMemcpyDeviceToHost, st));
    };
    copy(out->t_id, h.f[3]); copy(out->t_idx, h.f[4]); copy(out->q_id, h.f[0]); copy(out->q_idx, h.f[5]);
    copy(out->t_len, h.f[6]); copy(out->q_len, h.f[7]); copy(out->match, h.f[8]); copy(out->score, h.f[9]);
    copy(out->evalue, h.evalue);
    CLAST_CK(cudaStreamSynchronize(st));
    ctx->last_launches = g_kernel_launches;
    return CLAST_OK;
  });
}

void clast_hits_free(clast_hits* h) {
  if (!h) return;
  std::free(h->t_id); std::free(h->t_idx); std::free(h->q_id); std::free(h->q_idx);
  std::free(h->t_len); std::free(h->q_len); std::free(h->match); std::free(h->score);
  std::free(h->evalue);
  std::memset(h, 0, sizeof(*h));
}

int clast_targets_create(clast_ctx* ctx, const clast_params* p, int32_t t_vram, const clast_seqs* targets,
                         int32_t n_loads, const int64_t* load_sizes, clast_targets** out) {
  if (!ctx || !out) return CLAST_ERR_ARG;
  *out = nullptr;
  return guarded(ctx, [&]() -> int {
    check_params(p);
    if (!targets || n_loads < 0 || (n_loads > 0 && !load_sizes)) throw std::invalid_argument("bad targets");
    int64_t total = 0;
    for (int32_t k = 0; k < n_loads; ++k) total += load_sizes[k];
    if (total != targets->n_seqs) throw std::invalid_argument("load sizes do not add up to n_seqs");
    CLAST_CK(cudaSetDevice(ctx->device));
    g_alloc_stream = ctx->st;
    g_kernel_launches = 0;
    ctx->stats.index_ms = ctx->stats.index_upload_ms = 0;
    ctx->stats.index_launches = 0;
    const double w0 = wall_ms();
    const int l = p->lmer;
    std::unique_ptr<clast_targets> T(new clast_targets());
    T->ctx = ctx;
    T->n_loads = n_loads;
    for (int32_t k = 0; k < n_loads; ++k) T->load_first.push_back(T->load_first.back() + load_sizes[k]);
    cudaStream_t st = ctx->st;
    T->ev_start = ctx->timer.take();
    T->ev_up = ctx->timer.take();
    T->ev_done = ctx->timer.take();
    T->failed.alloc(1);
    // the raw target set on the device, uploaded once unless already resident
    const int64_t nt = targets->n_seqs;
    const int64_t tbytes = nt ? targets->offsets[nt] - targets->offsets[0] : 0;
    // host-resident bases go up on the copy stream window by window, so that a
    // window's index build starts as soon as its bytes have arrived
    const bool host_src = !targets->bases_on_device;
    const char* hsrc = targets->bases + (nt ? targets->offsets[0] : 0);
    DevArray<char> traw;
    DevArray<int32_t> all_gw, all_ln;
    DevArray<int64_t> all_so;
    std::vector<std::unique_ptr<clast_index>> shells;
    cudaStream_t cs = host_src ? ctx->st_copy : st;
    if (host_src) {
      g_alloc_stream = ctx->st_copy;
      traw.alloc((size_t)tbytes + 1);
      g_alloc_stream = st;
      traw.st = st;  // freed in the compute stream's order, after the builds
    }
    const char* src = host_src ? traw.p : hsrc;
    CLAST_CK(cudaEventRecord(T->ev_start, cs));
    if (!host_src) CLAST_CK(cudaEventRecord(T->ev_up, cs));  // nothing to upload
    int64_t copied = 0;  // source bytes already queued for upload
    std::vector<cudaEvent_t> win_ev;
    // a call that fails part-way frees its blocks on the compute stream, which
    // does not wait for the builds and copies that still use them (declared
    // after what it guards)
    UnwindSync unwind{ctx->st_copy, ctx->st_build[0], ctx->st_build[1], st};
    static_assert(kBuildStreams == 2, "the streams that unwind waits for");
    // the windows are indexed back to back on the stream with no host
    // synchronisation; the table-overflow count is read by the first clast_map
    unsigned long long* failed = T->failed.p;
    CLAST_CK(cudaMemsetAsync(failed, 0, sizeof(unsigned long long), st));
    const int64_t k0 = g_kernel_launches;
    const int64_t base0 = nt ? targets->offsets[0] : 0;
    // the windows of every load (moveTargetWindow, CHostSchedular.cu:25-35) and
    // their sequence tables, planned on the host and uploaded in one go: a copy
    // from pageable memory waits for the stream, so none happens per window
    struct Plan { int32_t load, first, nseqs; int64_t n, meta; };
    std::vector<Plan> plan;
    std::vector<int32_t> gw, ln;
    std::vector<int64_t> so;
    int64_t rec = 0;
    for (int32_t k = 0; k < n_loads; ++k) {
      const int64_t r0 = rec, r1 = rec + load_sizes[k];
      rec = r1;
      // load-relative gateway: prefix sums of len + l - 1 (CHostSeqList_target.cu:8-33)
      std::vector<int64_t> lg(r1 - r0 + 1, 0);
      for (int64_t i = r0; i < r1; ++i)
        lg[i - r0 + 1] = lg[i - r0] + (targets->offsets[i + 1] - targets->offsets[i]) + (l - 1);
      const int64_t tEnd = r1 - r0;
      for (int64_t tb = 0, te = 1; tb < tEnd; tb = te++) {
        while (te < tEnd && lg[te + 1] - lg[tb] < (int64_t)t_vram) ++te;
        const int64_t wn = lg[te] - lg[tb];
        if (wn >= (int64_t)INT32_MAX) throw std::invalid_argument("target window larger than 2^31 bases");
        plan.push_back(Plan{k, (int32_t)tb, (int32_t)(te - tb), wn, (int64_t)gw.size()});
        for (int64_t i = r0 + tb; i < r0 + te; ++i) {
          gw.push_back((int32_t)(lg[i - r0] - lg[tb]));
          ln.push_back((int32_t)(targets->offsets[i + 1] - targets->offsets[i]));
          so.push_back(targets->offsets[i] - base0);
        }
      }
    }
    all_gw.alloc(gw.size());
    all_ln.alloc(ln.size());
    all_so.alloc(so.size());
    if (!gw.empty()) {
      CLAST_CK(cudaMemcpyAsync(all_gw.p, gw.data(), gw.size() * sizeof(int32_t), cudaMemcpyHostToDevice, st));
      CLAST_CK(cudaMemcpyAsync(all_ln.p, ln.data(), ln.size() * sizeof(int32_t), cudaMemcpyHostToDevice, st));
      CLAST_CK(cudaMemcpyAsync(all_so.p, so.data(), so.size() * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    }
    // Windows are built alternately on the context's build streams, each with
    // its own scratch, so that two builds run at once (a build is a chain of
    // small, latency-bound kernels); every build stream starts after the plan's
    // upload above and the compute stream waits for all of them at the end.
    // Windows searched together (2k and 2k + 1) share their filter memory.
    for (size_t wi = 0; wi < plan.size(); ++wi) shells.emplace_back(new clast_index());
    for (size_t wi = 0; wi < plan.size(); wi += 2) {
      const int n = wi + 1 < plan.size() ? 2 : 1;
      clast_index* two[2] = {shells[wi].get(), n > 1 ? shells[wi + 1].get() : nullptr};
      int fshift = 63;
      for (int k = 0; k < n; ++k) fshift = std::min(fshift, filter_shift(plan[wi + k].n / p->stride));
      alloc_filters(two, n, fshift, st);
    }
    cudaEvent_t planned = ctx->timer.take();
    win_ev.push_back(planned);
    CLAST_CK(cudaEventRecord(planned, st));
    for (int b = 0; b < kBuildStreams; ++b) CLAST_CK(cudaStreamWaitEvent(ctx->st_build[b], planned, 0));
    for (size_t wi = 0; wi < plan.size(); ++wi) {
      const Plan& w = plan[wi];
      const int b = (int)(wi % kBuildStreams);
      cudaStream_t bs = ctx->st_build[b];
      if (host_src) {  // the window's records: source bytes up to the end of its last record
        const int64_t last = so[w.meta + w.nseqs - 1] + ln[w.meta + w.nseqs - 1];
        if (last > copied) {
          CLAST_CK(cudaMemcpyAsync(traw.p + copied, hsrc + copied, (size_t)(last - copied), cudaMemcpyHostToDevice,
                                   cs));
          copied = last;
        }
        win_ev.push_back(ctx->timer.take());
        CLAST_CK(cudaEventRecord(win_ev.back(), cs));
        CLAST_CK(cudaStreamWaitEvent(bs, win_ev.back(), 0));
      }
      g_alloc_stream = bs;
      DevArray<char> padded;
      DevArray<int32_t> dgw, dln;
      padded.alloc((size_t)w.n + 2 * kPad);
      dgw.alloc(w.nseqs);
      dln.alloc(w.nseqs);
      CLAST_CK(cudaMemcpyAsync(dgw.p, all_gw.p + w.meta, w.nseqs * sizeof(int32_t), cudaMemcpyDeviceToDevice, bs));
      CLAST_CK(cudaMemcpyAsync(dln.p, all_ln.p + w.meta, w.nseqs * sizeof(int32_t), cudaMemcpyDeviceToDevice, bs));
      CLAST_CK(cudaMemsetAsync(padded.p, 'N', (size_t)w.n + 2 * kPad, bs));
      build_window(src, all_so.p + w.meta, dgw.p, dln.p, w.nseqs, w.n, padded.p + kPad, bs);
      clast_targets::Win win;
      win.load = w.load;
      win.first = w.first;
      win.ix.reset(make_index_resident(ctx->ws_build[b], bs, p, std::move(padded), w.n, std::move(dgw),
                                       std::move(dln), w.nseqs, w.first, failed, std::move(shells[wi])));
      g_alloc_stream = st;
      // the index is used and finally freed in the compute stream's order
      clast_index& ix = *win.ix;
      ix.bases.st = ix.gateway.st = ix.lengths.st = ix.table.st = ix.entries.st = ix.kept.st = st;
      T->wins.push_back(std::move(win));
    }
    // the builds end on build stream 0 (which waits for the others): ev_done
    // there; the compute stream is not held up (clast_map prepares the query
    // while the builds run and waits for ev_done before its first search), and
    // the buffers the builds read are freed on build stream 0 after them
    cudaStream_t b0 = ctx->st_build[0];
    for (int b = 1; b < kBuildStreams; ++b) {
      win_ev.push_back(ctx->timer.take());
      CLAST_CK(cudaEventRecord(win_ev.back(), ctx->st_build[b]));
      CLAST_CK(cudaStreamWaitEvent(b0, win_ev.back(), 0));
    }
    if (host_src) {
      if (tbytes > copied)
        CLAST_CK(cudaMemcpyAsync(traw.p + copied, hsrc + copied, (size_t)(tbytes - copied), cudaMemcpyHostToDevice,
                                 cs));
      CLAST_CK(cudaEventRecord(T->ev_up, cs));
      CLAST_CK(cudaStreamWaitEvent(b0, T->ev_up, 0));  // the whole upload is done before traw goes
    }
    CLAST_CK(cudaEventRecord(T->ev_done, b0));
    traw.st = all_gw.st = all_ln.st = all_so.st = b0;
    T->launches = g_kernel_launches - k0;
    // a host source must stay readable until its copy has been made
    if (host_src) CLAST_CK(cudaEventSynchronize(T->ev_up));
    for (cudaEvent_t e : win_ev) ctx->timer.pool.push_back(e);
    ctx->stats.index_wall_ms = wall_ms() - w0;
    *out = T.release();
    return CLAST_OK;
  });
}

void clast_targets_free(clast_targets* t) { delete t; }

static int map_impl(clast_ctx* ctx, const clast_targets* T, const clast_params* p, int32_t q_vram,
                    const clast_seqs* reads, int32_t n_loads, const int64_t* load_sizes, clast_map_result* out);

int clast_map(clast_ctx* ctx, const clast_targets* T, const clast_params* p, int32_t q_vram,
              const clast_seqs* reads, int32_t n_loads, const int64_t* load_sizes, clast_map_result* out) {
  if (!ctx || !out) return CLAST_ERR_ARG;
  const double w0 = wall_ms();
  const int rc = map_impl(ctx, T, p, q_vram, reads, n_loads, load_sizes, out);
  ctx->stats.map_call_ms = wall_ms() - w0;
  return rc;
}

static int map_impl(clast_ctx* ctx, const clast_targets* T, const clast_params* p, int32_t q_vram,
                    const clast_seqs* reads, int32_t n_loads, const int64_t* load_sizes, clast_map_result* out) {
  std::memset(out, 0, sizeof(*out));
  return guarded(ctx, [&]() -> int {
    check_params(p);
    if (!T || !reads || n_loads < 0 || (n_loads > 0 && !load_sizes)) throw std::invalid_argument("bad arguments");
    int64_t total = 0;
    for (int32_t k = 0; k < n_loads; ++k) total += load_sizes[k];
    if (total != reads->n_seqs) throw std::invalid_argument("load sizes do not add up to n_seqs");
    for (const auto& w : T->wins)
      if (p->lmer != w.ix->l || p->stride != w.ix->stride || p->cut_repeat != w.ix->cut)
        throw std::invalid_argument("params differ from the ones the targets were built with");
    CLAST_CK(cudaSetDevice(ctx->device));
    g_alloc_stream = ctx->st;
    g_kernel_launches = 0;
    cudaStream_t st = ctx->st;
    clast_stats& S = ctx->stats;
    const double w0 = wall_ms();
    S.map_ms = S.map_upload_ms = 0;
    S.map_launches = S.query_bases = S.query_kmers = S.seeds = S.hits = S.results = S.dp_cells = 0;
    S.dp_warp_hits = 0;
    ctx->timer.reset();
    // Results released since the last map give their device block back before
    // this one's is taken: held until then, the old block cut the free memory
    // from which the next job's tables come, and the pool moved or took memory at
    // every step (medium job in a loop: 11.7 - 14.2 ms a step and stalls of up to
    // a second as the pool grew; 11.7 ms steady so).
    for (auto& a : ctx->arenas)
      if (!a->in_use) a->dev.slab.mem.release();
    const int64_t nreads = reads->n_seqs;
    if (nreads >= ((int64_t)1 << 30)) throw std::invalid_argument("at most 2^30 reads per map (2^31 strands)");
    const int64_t nb = reads->offsets[nreads] - reads->offsets[0];
    // The reads' bases go up first, on the copy stream (allocated there, so
    // nothing waits for the compute stream, which may still be building the
    // target indexes), so that the host preparation below overlaps the
    // transfer; the compute stream waits for the uploads further down and
    // frees the buffers in its order.
    cudaStream_t cs = ctx->st_copy;
    CLAST_CK(cudaEventRecord(ctx->ev0, cs));
    DevArray<char> draw;
    const char* rsrc = reads->bases + reads->offsets[0];
    if (!reads->bases_on_device) {
      g_alloc_stream = cs;
      draw.alloc((size_t)nb + 64);
      g_alloc_stream = st;
      draw.st = st;
      if (nb) CLAST_CK(cudaMemcpyAsync(draw.p, rsrc, nb, cudaMemcpyHostToDevice, cs));
      rsrc = draw.p;
      // the compute stream, which frees draw (also when a check below
      // throws), comes after the copy
      CLAST_CK(cudaEventRecord(ctx->ev3, cs));
      CLAST_CK(cudaStreamWaitEvent(st, ctx->ev3, 0));
    }
    // query windows of every load, in read order
    std::vector<int64_t> wfirst;
    std::vector<int64_t> load_first(n_loads + 1, 0);
    for (int32_t k = 0; k < n_loads; ++k) load_first[k + 1] = load_first[k] + load_sizes[k];
    for (int32_t k = 0; k < n_loads; ++k)
      query_windows(reads->offsets, load_first[k], load_first[k + 1], p->lmer, q_vram, wfirst);
    wfirst.push_back(nreads);
    // read lengths: of a large batch on the device (a pass over a million
    // offsets takes the host 1-2 ms), unless one may exceed 32 bits
    const bool dev_lengths = nreads > kHostLengths && nb <= INT32_MAX;
    int32_t min_len = nreads ? INT32_MAX : 0, max_len = 0;
    for (int64_t r = 0; r < nreads && !dev_lengths; ++r) {
      const int64_t len = reads->offsets[r + 1] - reads->offsets[r];
      if (len > INT32_MAX) throw std::invalid_argument("read longer than 2^31 bases");
      min_len = std::min<int32_t>(min_len, (int32_t)len);
      max_len = std::max<int32_t>(max_len, (int32_t)len);
    }
    // The tables of the batch behind its strands: first reads of the loads,
    // strands where the query windows start, read offsets relative to the first
    // read.  They go up in one copy; the offsets of a large batch come straight
    // from the caller's array.
    const size_t win_at = QueryBatch::al(((size_t)n_loads + 1) * sizeof(int64_t));
    const size_t len_at = win_at + QueryBatch::al(wfirst.size() * sizeof(int32_t));
    const size_t off_at = len_at + QueryBatch::al(2 * sizeof(int32_t));  // shortest, longest read
    const size_t off_bytes = ((size_t)nreads + 1) * sizeof(int64_t);
    const bool offs_staged = off_bytes <= kStageMax / 16 || reads->offsets[0] != 0;
    QueryBatch qb;
    g_alloc_stream = cs;
    qb.alloc(2 * nb, 2 * nreads, off_at + off_bytes);
    g_alloc_stream = st;
    qb.mem.st = st;
    qb.min_len = min_len;
    qb.max_len = max_len;
    qb.nwin = (int32_t)wfirst.size() - 1;
    qb.wstart = reinterpret_cast<const int32_t*>(qb.meta + win_at);
    const int64_t* dlf = reinterpret_cast<const int64_t*>(qb.meta);
    const int64_t* doff = reinterpret_cast<const int64_t*>(qb.meta + off_at);
    const size_t table_bytes = off_at + (offs_staged ? off_bytes : 0);
    HostTables host_tables(ctx, table_bytes);
    char* tables = host_tables.p;
    std::memcpy(tables, load_first.data(), load_first.size() * sizeof(int64_t));
    int32_t* wstart = reinterpret_cast<int32_t*>(tables + win_at);
    for (size_t i = 0; i < wfirst.size(); ++i) wstart[i] = (int32_t)(2 * wfirst[i]);
    const int32_t lens[2] = {min_len, max_len};
    std::memcpy(tables + len_at, lens, sizeof(lens));
    if (offs_staged) {
      int64_t* o = reinterpret_cast<int64_t*>(tables + off_at);
      for (int64_t i = 0; i <= nreads; ++i) o[i] = reads->offsets[i] - reads->offsets[0];
    }
    S.map_prep_ms = wall_ms() - w0;
    host_tables.upload(qb.meta, table_bytes, cs);
    if (!offs_staged)
      CLAST_CK(cudaMemcpyAsync(qb.meta + off_at, reads->offsets, off_bytes, cudaMemcpyHostToDevice, cs));
    CLAST_CK(cudaEventRecord(ctx->ev3, cs));
    CLAST_CK(cudaStreamWaitEvent(st, ctx->ev3, 0));
    CLAST_CK(cudaEventRecord(ctx->ev1, st));  // the reads are resident and the compute stream is free
    build_strands(rsrc, doff, nreads, qb.bases + kPad, qb.start, qb.len, st);
    if (nreads > 0) qb.pack(st);
    int32_t* dlen = reinterpret_cast<int32_t*>(qb.meta + len_at);
    if (dev_lengths) {
      read_lengths(doff, nreads, dlen, dlen + 1, st);
      CLAST_CK(cudaMemcpyAsync(ctx->lens, dlen, sizeof(lens), cudaMemcpyDeviceToHost, st));
    }
    S.query_bases = qb.n;
    // the index builds of clast_targets_create end before the first search
    settle_targets(ctx, T);
    CLAST_CK(cudaStreamWaitEvent(st, T->ev_done, 0));
    QueryRef qr = qb.ref();
    if (dev_lengths) qr.lens = ctx->lens;
    // windows searched per group (CLAST_SEED_WINDOWS, 1..4), as long as the
    // group's slots have 32-bit numbers
    int group = 2;
    if (const char* e = std::getenv("CLAST_SEED_WINDOWS")) group = std::max(1, std::min(kMaxSeedWins, std::atoi(e)));
    while (group > 1 && (int64_t)group * qr.q.nstrands >= INT32_MAX) --group;
    // every target window, in holder order (target load, window)
    std::vector<Group> groups;
    for (size_t g0 = 0; g0 < T->wins.size() && qr.q.nstrands > 0; g0 += (size_t)group) {
      Group g;
      g.reads = true;
      for (size_t w = g0; w < std::min(T->wins.size(), g0 + (size_t)group); ++w) {
        if (T->wins[w].ix->n_keys == 0) continue;
        g.load[g.nw] = T->wins[w].load;
        g.ix[g.nw++] = T->wins[w].ix.get();
      }
      if (g.nw > 0) groups.push_back(g);
    }
    std::vector<std::unique_ptr<SlabSink>> found;
    int64_t F = 0;
    for (size_t k = 0; k < groups.size(); ++k) {
      Group g = groups[k];
      std::unique_ptr<SlabSink> sink(new SlabSink(n_loads, groups.size() > 1));
      g.part_cap = std::max(first_part_cap(ctx, qr.n), ctx->part_hint);
      const clast_stats before = S;
      int64_t f = 0;
      bool split = false;
      try {
        f = search_group(ctx, ctx->ws, p, qr, g, *sink);
      } catch (const std::bad_alloc&) {
        if (g.nw == 1) throw;
        split = true;
      } catch (const TooManyHits&) {
        if (g.nw == 1) throw;
        split = true;
      }
      if (split) {  // the hits of all its windows at once are too many: its windows one by one
        sink.reset();
        S = before;
        CLAST_CK(cudaStreamSynchronize(st));
        ctx->timer.flush();
        ctx->ws.release_all();  // buffers that grew for the whole group
        ctx->part_hint = 0;
        groups.erase(groups.begin() + k);
        for (int w = 0; w < g.nw; ++w) {
          Group one;
          one.reads = g.reads;
          one.nw = 1;
          one.ix[0] = g.ix[w];
          one.load[0] = g.load[w];
          groups.insert(groups.begin() + k + w, one);
        }
        --k;
        continue;
      }
      if (f == 0) continue;
      F += f;
      found.push_back(std::move(sink));
    }
    ResultSlab res_dev;
    const int64_t* roff = nullptr;  // per-read offsets of the result
    if (groups.size() == 1 && found.size() == 1) {
      res_dev = std::move(found[0]->slab);
      roff = found[0]->foff;
    } else {
      // fixResult: stable merge by (read, score desc) over the groups, on the device
      res_dev.alloc(F, n_loads);
      if (F > 0) {
        std::vector<GroupHits> gh;
        int64_t base = 0;
        for (const auto& x : found) {
          GroupHits h{};
          for (int k = 0; k < 10; ++k) h.f[k] = x->slab.f[k];
          h.evalue = x->slab.evalue;
          h.foff = x->offsets.p;
          h.base = base;
          base += x->slab.n;
          gh.push_back(h);
        }
        GroupHits* dgh = ctx->ws.get<GroupHits>("m_groups", gh.size());
        CLAST_CK(cudaMemcpyAsync(dgh, gh.data(), gh.size() * sizeof(GroupHits), cudaMemcpyHostToDevice, st));
        int32_t* mcnt = ctx->ws.get<int32_t>("m_cnt", nreads + 1);
        int64_t* moff = ctx->ws.get<int64_t>("m_off", nreads + 1);
        merge_groups(dgh, (int)gh.size(), F, nreads, mcnt, moff, res_dev.view(), ctx->ws, st);
        roff = moff;
      }
    }
    // per query load offsets
    if (roff) gather_i64(roff, dlf, n_loads + 1, res_dev.load_offsets, st);
    else CLAST_CK(cudaMemsetAsync(res_dev.load_offsets, 0, ((size_t)n_loads + 1) * sizeof(int64_t), st));
    clast_map_result res;
    std::memset(&res, 0, sizeof(res));
    res.n = F;
    // one pinned arena laid out as the device's result: one download
    const size_t need = res_dev.bytes;
    PinnedArena* arena = nullptr;
    for (auto& a : ctx->arenas)
      if (!a->in_use && (arena == nullptr || a->bytes > arena->bytes)) arena = a.get();
    if (!arena) {
      ctx->arenas.emplace_back(new PinnedArena());
      arena = ctx->arenas.back().get();
    }
    if (arena->bytes < need) {
      if (arena->p) CLAST_CK(cudaFreeHost(arena->p));
      arena->p = nullptr;
      arena->bytes = 0;
      const size_t want = need + need / 4;
      if (cudaMallocHost(&arena->p, want) != cudaSuccess) {
        (void)cudaGetLastError();
        throw std::bad_alloc();
      }
      arena->bytes = want;
    }
    arena->in_use = true;
    res.owner = arena;
    CLAST_CK(cudaMemcpyAsync(arena->p, res_dev.mem.p, need, cudaMemcpyDeviceToHost, st));
    {
      char* base = static_cast<char*>(arena->p);
      auto host = [&](const void* dev) { return base + (static_cast<const char*>(dev) - res_dev.mem.p); };
      int32_t** dst[10] = {&res.read, &res.strand, &res.t_load, &res.t_seq, &res.t_idx, &res.q_idx, &res.t_len,
                           &res.q_len, &res.match, &res.score};
      for (int k = 0; k < 10; ++k) *dst[k] = reinterpret_cast<int32_t*>(host(res_dev.f[k]));
      res.evalue = reinterpret_cast<double*>(host(res_dev.evalue));
      res.load_offsets = reinterpret_cast<int64_t*>(host(res_dev.load_offsets));
      // the device copy stays with the arena for clast_format_tsv
      arena->dev.slab = std::move(res_dev);
      arena->dev.n = F;
      arena->dev.n_loads = n_loads;
    }
    CLAST_CK(cudaEventRecord(ctx->ev2, st));
    CLAST_CK(cudaEventSynchronize(ctx->ev2));
    float up = 0, ms = 0;
    CLAST_CK(cudaEventElapsedTime(&up, ctx->ev0, ctx->ev3));
    CLAST_CK(cudaEventElapsedTime(&ms, ctx->ev1, ctx->ev2));
    ctx->timer.flush();
    S.map_upload_ms = up;
    S.map_ms = ms;
    S.map_launches = g_kernel_launches;
    S.seed_ms = ctx->timer.ms[StageTimer::SEED];
    S.seed_launches = ctx->timer.n[StageTimer::SEED];
    S.dp_ms = ctx->timer.ms[StageTimer::DP];
    S.dp_launches = ctx->timer.n[StageTimer::DP];
    S.sort_ms = ctx->timer.ms[StageTimer::SORT];
    S.final_ms = ctx->timer.ms[StageTimer::FINAL];
    S.dp_order_ms = ctx->timer.ms[StageTimer::DPORDER];
    ctx->last_ms = up + ms;
    ctx->last_launches = g_kernel_launches;
    S.map_wall_ms = wall_ms() - w0;
    *out = res;
    return CLAST_OK;
  });
}

void clast_map_result_free(clast_map_result* r) {
  if (!r) return;
  if (r->owner) static_cast<PinnedArena*>(r->owner)->in_use = false;
  std::memset(r, 0, sizeof(*r));
}

int clast_ctx_trim(clast_ctx* ctx) {
  if (!ctx) return CLAST_ERR_ARG;
  return guarded(ctx, [&]() -> int {
    CLAST_CK(cudaSetDevice(ctx->device));
    CLAST_CK(cudaDeviceSynchronize());
    for (auto& a : ctx->arenas)
      if (!a->in_use) a->dev.slab.mem.release();
    ctx->ws.release_all();
    ctx->part_hint = 0;
    ctx->release_staging();
    for (auto& w : ctx->ws_build) w.release_all();
    CLAST_CK(cudaDeviceSynchronize());
    cudaMemPool_t pool;
    CLAST_CK(cudaDeviceGetDefaultMemPool(&pool, ctx->device));
    CLAST_CK(cudaMemPoolTrimTo(pool, 0));
    return CLAST_OK;
  });
}

int clast_int32_peak(clast_ctx* ctx, double* tera_ops) {
  if (!ctx || !tera_ops) return CLAST_ERR_ARG;
  return guarded(ctx, [&]() -> int {
    CLAST_CK(cudaSetDevice(ctx->device));
    int* sink = ctx->ws.get<int>("probe_sink", 1);
    *tera_ops = int32_probe(ctx->st, sink);
    return CLAST_OK;
  });
}

int clast_get_stats(const clast_ctx* ctx, clast_stats* out) {
  if (!ctx || !out) return CLAST_ERR_ARG;
  *out = ctx->stats;
  return CLAST_OK;
}

int clast_last_map_stats(const clast_ctx* ctx, double* device_ms, int64_t* kernel_launches) {
  if (!ctx) return CLAST_ERR_ARG;
  if (device_ms) *device_ms = ctx->last_ms;
  if (kernel_launches) *kernel_launches = ctx->last_launches;
  return CLAST_OK;
}

}  // extern "C"

// ----------------------------------------------------------------------------
// clast_search_noalloc: clast_search on a fixed scratch buffer, allocating
// nothing.  It runs search_group, as clast_search does, with seed partitions
// sized to fit the scratch and every device buffer a slot of it (Workspace arena
// mode); the hits go from scratch slots straight into the caller's host arrays.
// ----------------------------------------------------------------------------
namespace {

constexpr size_t kSearchScratchBytes = (size_t)CLAST_NOALLOC_SCRATCH_BYTES;
static __device__ __align__(256) unsigned char g_search_scratch[kSearchScratchBytes];

constexpr int kMaxScratchDevices = 64;
std::mutex g_scratch_mu;
void* g_scratch_addr[kMaxScratchDevices];           // device address of g_search_scratch, per device
std::atomic<int> g_scratch_busy[kMaxScratchDevices];  // 1 while a call uses that device's scratch

// Address of this device's scratch; the device must be current.  Looked up
// once per device.
char* search_scratch(int device) {
  std::lock_guard<std::mutex> lock(g_scratch_mu);
  if (!g_scratch_addr[device]) {
    void* ptr = nullptr;
    CLAST_CK(cudaGetSymbolAddress((void**)&ptr, g_search_scratch));
    g_scratch_addr[device] = ptr;
  }
  return static_cast<char*>(g_scratch_addr[device]);
}

__global__ void k_widen_i32(const int32_t* __restrict__ in, int64_t n, int64_t* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = in[i];
}

// Bytes of the query-sized buffers, as Workspace::get rounds them.
size_t fixed_scratch_bytes(int64_t n, int64_t ns, int parts) {
  auto r = [](size_t b) { return ((b ? b : 1) + 255) & ~size_t(255); };
  const size_t nb = (size_t)n, s = (size_t)ns;
  return r(nb + 2 * kPad) + r(8 * s) + r(4 * s) + r(4 * s) + r(8) + r(8 * (nb / 32 + 4)) + r(8 * (nb / 64 + 4)) +
         r(8 * (s + 1)) + r(4 * s) + r(4 * s) + r(8 * (2 + 2 * (size_t)parts)) + r(4 * s) + r(8 * (s + 1)) +
         r(16 * s) + (64 << 10);
}

// Bytes of search_group's per-strand tables, as Workspace::get rounds them.
size_t fixed_table_bytes(int64_t ns) {
  auto r = [](size_t b) { return ((b ? b : 1) + 255) & ~size_t(255); };
  const size_t s = (size_t)ns;
  return r(8 * (s + 1)) + 2 * r(4 * s) + r(8 * (2 + 2 * (size_t)kSeedParts));
}

// Clears the busy flag of a device's scratch once the call's stream work has
// ended (also when the call failed after launching work).
struct ScratchClaim {
  int device;
  cudaStream_t st;
  ~ScratchClaim() {
    cudaStreamSynchronize(st);
    (void)cudaGetLastError();
    g_scratch_busy[device].store(0);
  }
};

}  // namespace

extern "C" int clast_search_noalloc(clast_ctx* ctx, const clast_index* ix, const clast_params* p,
                                    const char* q_bases, int64_t n_qbases, const int32_t* q_gateway,
                                    const int32_t* q_lengths, int32_t n_qseqs, int32_t q_begin, int64_t capacity,
                                    clast_hits* out) {
  if (!ctx || !out) return CLAST_ERR_ARG;
  out->n = 0;
  return guarded(ctx, [&]() -> int {
    check_params(p);
    if (!ix) throw std::invalid_argument("index is null");
    if (p->lmer != ix->l || p->stride != ix->stride || p->cut_repeat != ix->cut)
      throw std::invalid_argument("params differ from the ones the index was built with");
    if (n_qseqs < 0 || (n_qseqs & 1) || (q_begin & 1))
      throw std::invalid_argument("query windows hold whole reads: n_qseqs and q_begin must be even");
    if (n_qbases < 0 || (n_qbases > 0 && !q_bases) || (n_qseqs > 0 && (!q_gateway || !q_lengths)))
      throw std::invalid_argument("bad query arrays");
    if (capacity < 0 || (capacity > 0 && (!out->t_id || !out->t_idx || !out->q_id || !out->q_idx ||
                                          !out->t_len || !out->q_len || !out->match || !out->score ||
                                          !out->evalue)))
      throw std::invalid_argument("capacity < 0, or a null output array");
    for (int32_t i = 0; i < n_qseqs; ++i)
      if (q_gateway[i] < 0 || q_lengths[i] < 0 || (int64_t)q_gateway[i] + q_lengths[i] > n_qbases)
        throw std::invalid_argument("query sequence outside the base array");
    if (ctx->device < 0 || ctx->device >= kMaxScratchDevices)
      throw std::invalid_argument("device ordinal beyond the scratch table");
    const size_t fixed = fixed_scratch_bytes(n_qbases, n_qseqs, kSeedParts);
    if (fixed > kSearchScratchBytes)
      throw std::invalid_argument("query window of " + std::to_string(n_qbases) + " bases and " +
                                  std::to_string(n_qseqs) + " sequences needs " + std::to_string(fixed) +
                                  " bytes of scratch before seeding; clast_search_noalloc has " +
                                  std::to_string(kSearchScratchBytes) + " (use clast_search)");
    CLAST_CK(cudaSetDevice(ctx->device));
    int idle = 0;
    if (!g_scratch_busy[ctx->device].compare_exchange_strong(idle, 1))
      throw std::invalid_argument("another clast_search_noalloc call is using this device's scratch");
    cudaStream_t st = ctx->st;
    ScratchClaim claim{ctx->device, st};
    char* base = search_scratch(ctx->device);
    g_kernel_launches = 0;
    Workspace ws;
    ws.arena_begin(base, kSearchScratchBytes);
    const int64_t ns = n_qseqs, n = n_qbases;
    // the query window: padded bases, strand starts and lengths, 2-bit words
    char* qbases = ws.get<char>("q_bases", (size_t)n + 2 * kPad);
    CLAST_CK(cudaMemsetAsync(qbases, 'N', (size_t)n + 2 * kPad, st));
    if (n > 0) CLAST_CK(cudaMemcpyAsync(qbases + kPad, q_bases, (size_t)n, cudaMemcpyHostToDevice, st));
    int64_t* qstart = ws.get<int64_t>("q_start", ns);
    int32_t* qlen = ws.get<int32_t>("q_len", ns);
    int32_t* qgw = ws.get<int32_t>("q_gw32", ns);
    int32_t* wstart = ws.get<int32_t>("q_wstart", 2);
    if (ns > 0) {
      CLAST_CK(cudaMemcpyAsync(qgw, q_gateway, ns * sizeof(int32_t), cudaMemcpyHostToDevice, st));
      CLAST_CK(cudaMemcpyAsync(qlen, q_lengths, ns * sizeof(int32_t), cudaMemcpyHostToDevice, st));
      k_widen_i32<<<(unsigned)((ns + 255) / 256), 256, 0, st>>>(qgw, ns, qstart);
      CLAST_LAUNCHED();
    }
    const int32_t ws2[2] = {0, n_qseqs};
    CLAST_CK(cudaMemcpyAsync(wstart, ws2, sizeof(ws2), cudaMemcpyHostToDevice, st));
    uint64_t* packed = ws.get<uint64_t>("q_packed", (size_t)(n / 32 + 4));
    uint64_t* nmask = ws.get<uint64_t>("q_nmask", (size_t)(n / 64 + 4));
    pack_bases(qbases + kPad, n, packed, nmask, st);
    QueryView q;
    q.bases = qbases + kPad;
    q.n = n;
    q.packed = packed;
    q.nmask = nmask;
    q.start = qstart;
    q.len = qlen;
    q.nstrands = n_qseqs;
    auto finish = [&](int64_t F) {
      CLAST_CK(cudaStreamSynchronize(st));
      ctx->last_launches = g_kernel_launches;
      out->n = F;
      return CLAST_OK;
    };
    if (ns == 0 || ix->n_keys == 0) return finish(0);
    int32_t lmin = INT32_MAX, lmax = 0;
    for (int32_t i = 0; i < n_qseqs; ++i) {
      lmin = std::min(lmin, q_lengths[i]);
      lmax = std::max(lmax, q_lengths[i]);
    }
    QueryRef qr;
    qr.q = q;
    qr.n = n;
    qr.wstart = wstart;
    qr.nwin = 1;
    qr.min_len = lmin;
    qr.max_len = lmax;
    // the search is clast_search's, on the fixed scratch; the seed partitions
    // take at most half of what is free behind the seed tables (offsets,
    // counts, counters); the hits go to slots of the scratch, then to the
    // caller's arrays
    Group g;
    g.nw = 1;
    g.ix[0] = ix;
    const size_t tables = ws.arena_used + fixed_table_bytes(ns);
    const size_t left = tables < ws.arena_cap ? ws.arena_cap - tables : 0;
    g.part_fit = (int64_t)(left / 2 / (12 * (size_t)kSeedParts)) - 256;
    g.part_cap = std::max<int64_t>(1, std::min(first_part_cap(ctx, n), g.part_fit));
    struct ArenaSink : HitSink {
      Workspace& ws;
      int64_t capacity;
      clast_hits* out;
      OutView fo{};
      int32_t q_first = 0;
      ArenaSink(Workspace& w, int64_t cap, clast_hits* o) : ws(w), capacity(cap), out(o) {}
      OutView take(int64_t F, const int64_t*, int64_t, cudaStream_t) override {
        if (F > capacity) {
          out->n = F;
          throw std::invalid_argument("window has " + std::to_string(F) + " hits, capacity is " +
                                      std::to_string(capacity));
        }
        fo.t_seq = ws.get<int32_t>("o_tid", F);
        fo.t_idx = ws.get<int32_t>("o_tidx", F);
        fo.q_id = ws.get<int32_t>("o_qid", F);
        fo.q_idx = ws.get<int32_t>("o_qidx", F);
        fo.t_len = ws.get<int32_t>("o_tlen", F);
        fo.q_len = ws.get<int32_t>("o_qlen", F);
        fo.match = ws.get<int32_t>("o_match", F);
        fo.score = ws.get<int32_t>("o_score", F);
        fo.evalue = ws.get<double>("o_e", F);
        fo.q_first = q_first;
        return fo;
      }
    } sink(ws, capacity, out);
    sink.q_first = q_begin;
    const int64_t F = search_group(ctx, ws, p, qr, g, sink);
    if (F == 0) return finish(0);
    const OutView& fo = sink.fo;
    int32_t* const dst[8] = {out->t_id, out->t_idx, out->q_id, out->q_idx, out->t_len, out->q_len, out->match,
                             out->score};
    const int32_t* const src[8] = {fo.t_seq, fo.t_idx, fo.q_id, fo.q_idx, fo.t_len, fo.q_len, fo.match, fo.score};
    for (int k = 0; k < 8; ++k)
      CLAST_CK(cudaMemcpyAsync(dst[k], src[k], F * sizeof(int32_t), cudaMemcpyDeviceToHost, st));
    CLAST_CK(cudaMemcpyAsync(out->evalue, fo.evalue, F * sizeof(double), cudaMemcpyDeviceToHost, st));
    return finish(F);
  });
}

