// clast_engine.h -- internal types shared by the host-side translation units of
// libclast_b200.so (engine, TSV formatting, serving loop): the context, the
// resident index of a target window, the resident targets, and the stream-
// ordered device arrays they are built from.  Not part of the C ABI.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <cstdint>
#include <map>
#include <memory>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/clast_gpu.h"
#include "clast_device.cuh"
#include "clast_kernels.cuh"
#include "clast_workspace.h"

namespace clast {

inline double wall_ms() {
  return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

// Stream used for the stream-ordered allocations of the current API call.
extern thread_local cudaStream_t g_alloc_stream;

// Owning device allocation from the device's stream-ordered memory pool
// (cudaMallocAsync / cudaFreeAsync on the owning context's stream), so
// steady-state calls reuse pool memory instead of calling cudaMalloc.
template <class T>
struct DevArray {
  T* p = nullptr;
  size_t n = 0;
  cudaStream_t st = nullptr;
  DevArray() = default;
  DevArray(const DevArray&) = delete;
  DevArray& operator=(const DevArray&) = delete;
  DevArray(DevArray&& o) noexcept : p(o.p), n(o.n), st(o.st) { o.p = nullptr; o.n = 0; }
  DevArray& operator=(DevArray&& o) noexcept {
    if (this != &o) {
      release();
      p = o.p;
      n = o.n;
      st = o.st;
      o.p = nullptr;
      o.n = 0;
    }
    return *this;
  }
  void alloc(size_t count) {
    release();
    n = count;
    st = g_alloc_stream;
    if (cudaMallocAsync(reinterpret_cast<void**>(&p), (count ? count : 1) * sizeof(T), st) != cudaSuccess) {
      // blocks freed on other streams become reusable once their frees have
      // run: wait for the device, then try once more
      (void)cudaGetLastError();
      cudaDeviceSynchronize();
      (void)cudaGetLastError();
      if (cudaMallocAsync(reinterpret_cast<void**>(&p), (count ? count : 1) * sizeof(T), st) != cudaSuccess) {
        (void)cudaGetLastError();
        p = nullptr;
        n = 0;
        throw std::bad_alloc();
      }
    }
  }
  void release() {
    if (p) cudaFreeAsync(p, st);
    p = nullptr;
    n = 0;
  }
  ~DevArray() { release(); }
};

inline void check_params(const clast_params* p) {
  if (!p) throw std::invalid_argument("params is null");
  if (p->lmer < 1 || p->lmer > 31) throw std::invalid_argument("lmer must be in 1..31");
  if (p->stride < 1) throw std::invalid_argument("stride must be >= 1");
  if (p->gap < 2 || p->gap > 16) throw std::invalid_argument("gap must be in 2..16");
}

// Device copy of a base array with kPad 'N' bytes on both sides.
inline void upload_padded(const char* host, int64_t n, DevArray<char>& dev, cudaStream_t st) {
  dev.alloc((size_t)n + 2 * kPad);
  CLAST_CK(cudaMemsetAsync(dev.p, 'N', (size_t)n + 2 * kPad, st));
  if (n > 0) CLAST_CK(cudaMemcpyAsync(dev.p + kPad, host, (size_t)n, cudaMemcpyHostToDevice, st));
}

// CUDA-event timing of device stages on one stream: begin()/end() bracket
// launches, flush() (after a stream synchronisation) adds up the intervals.
struct StageTimer {
  enum Stage { SEED = 0, DP = 1, SORT = 2, FINAL = 3, DPORDER = 4, N_STAGES = 5 };
  std::vector<cudaEvent_t> pool;
  struct Pending { int stage; cudaEvent_t a, b; };
  std::vector<Pending> pending;
  double ms[N_STAGES] = {0, 0, 0, 0, 0};
  int64_t n[N_STAGES] = {0, 0, 0, 0, 0};
  cudaEvent_t cur_a = nullptr;

  cudaEvent_t take() {
    if (pool.empty()) {
      cudaEvent_t e;
      CLAST_CK(cudaEventCreate(&e));
      return e;
    }
    cudaEvent_t e = pool.back();
    pool.pop_back();
    return e;
  }
  void begin(cudaStream_t st) {
    if (!cur_a) cur_a = take();  // else of a stage that ended by an exception
    CLAST_CK(cudaEventRecord(cur_a, st));
  }
  void end(int stage, cudaStream_t st, int launches = 1) {
    cudaEvent_t b = take();
    CLAST_CK(cudaEventRecord(b, st));
    pending.push_back({stage, cur_a, b});
    cur_a = nullptr;
    n[stage] += launches;
  }
  void flush() {
    for (auto& p : pending) {
      float t = 0;
      CLAST_CK(cudaEventElapsedTime(&t, p.a, p.b));
      ms[p.stage] += t;
      pool.push_back(p.a);
      pool.push_back(p.b);
    }
    pending.clear();
  }
  void reset() {
    flush();
    for (int i = 0; i < N_STAGES; ++i) { ms[i] = 0; n[i] = 0; }
  }
  ~StageTimer() {
    for (auto e : pool) cudaEventDestroy(e);
    if (cur_a) cudaEventDestroy(cur_a);
    for (auto& p : pending) { cudaEventDestroy(p.a); cudaEventDestroy(p.b); }
  }
};

// One search's results in one device allocation: per-load offsets, the ten
// int32 fields read strand t_load t_seq t_idx q_idx t_len q_len match score,
// and the E-values, each from a 256-byte boundary.
struct ResultSlab {
  DevArray<char> mem;
  int64_t n = 0;
  size_t bytes = 0;
  int64_t* load_offsets = nullptr;
  int32_t* f[10] = {};
  double* evalue = nullptr;
  void alloc(int64_t count, int32_t n_loads) {
    auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
    const size_t lo = al(((size_t)n_loads + 1) * sizeof(int64_t));
    const size_t w = al((size_t)(count ? count : 1) * sizeof(int32_t));
    n = count;
    bytes = lo + 10 * w + al((size_t)(count ? count : 1) * sizeof(double));
    mem.alloc(bytes);
    load_offsets = reinterpret_cast<int64_t*>(mem.p);
    for (int k = 0; k < 10; ++k) f[k] = reinterpret_cast<int32_t*>(mem.p + lo + k * w);
    evalue = reinterpret_cast<double*>(mem.p + lo + 10 * w);
  }
  OutView view() const {
    OutView v{};
    v.read = f[0]; v.strand = f[1]; v.t_load = f[2]; v.t_seq = f[3]; v.t_idx = f[4];
    v.q_idx = f[5]; v.t_len = f[6]; v.q_len = f[7]; v.match = f[8]; v.score = f[9];
    v.evalue = evalue;
    return v;
  }
};

// Pinned host buffer that holds one clast_map result; reused once released.
struct PinnedArena {
  void* p = nullptr;
  size_t bytes = 0;
  std::atomic<bool> in_use{false};  // released by the result's owner, possibly on another thread
  // The result on the device, kept until the first map after its release (so
  // that its text can be formatted on the GPU).
  struct Device {
    ResultSlab slab;
    int64_t n = 0;
    int32_t n_loads = 0;
  } dev;
};

// Reads of a batch up to which the host looks at every length itself.
constexpr int64_t kHostLengths = 1 << 15;
// Largest pinned staging buffer of a context.
constexpr size_t kStageMax = (size_t)16 << 20;
constexpr int kBuildStreams = 2;  // target windows indexed at once by clast_targets_create

}  // namespace clast

struct clast_ctx {
  using StageTimer = clast::StageTimer;
  using PinnedArena = clast::PinnedArena;
  using Workspace = clast::Workspace;
  std::vector<std::unique_ptr<PinnedArena>> arenas;      // clast_map results
  std::vector<std::unique_ptr<PinnedArena>> tsv_arenas;  // clast_format_tsv texts
  int device = 0;
  cudaStream_t st = nullptr;
  cudaStream_t st_copy = nullptr;  // query uploads, overlapping index builds still running
  cudaStream_t st_build[clast::kBuildStreams] = {};  // index builds of clast_targets_create
  Workspace ws_build[clast::kBuildStreams];          // their scratch
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr, ev3 = nullptr;
  Workspace ws;
  std::string err;
  double last_ms = 0;
  int64_t last_launches = 0;
  clast_stats stats{};
  StageTimer timer;
  int64_t seed_hint = 0;  // seed buffer capacity that sufficed before
  int64_t part_hint = 0;  // fullest seed partition of a window that overflowed before
  clast::GroupCtl* ctl = nullptr;  // pinned copy of a group's counters
  int32_t* lens = nullptr;         // pinned, behind it: shortest and longest read, when the device looks at them
  // Pinned buffer of up to kStageMax bytes for small tables on their way up and
  // small results on their way down.  stage() waits for the copy made from it
  // last (staged()).
  char* staging = nullptr;
  size_t staging_bytes = 0;
  cudaEvent_t ev_stage = nullptr;
  bool stage_pending = false;
  char* stage(size_t bytes) {
    if (stage_pending) CLAST_CK(cudaEventSynchronize(ev_stage));
    stage_pending = false;
    if (staging_bytes < bytes) {
      if (staging) CLAST_CK(cudaFreeHost(staging));
      staging = nullptr;
      staging_bytes = 0;
      const size_t want = std::max(bytes, std::min(bytes + bytes / 2 + (64 << 10), clast::kStageMax));
      if (cudaMallocHost(reinterpret_cast<void**>(&staging), want) != cudaSuccess) {
        (void)cudaGetLastError();
        staging = nullptr;
        throw std::bad_alloc();
      }
      staging_bytes = want;
    }
    return staging;
  }
  void staged(cudaStream_t s) {
    CLAST_CK(cudaEventRecord(ev_stage, s));
    stage_pending = true;
  }
  void release_staging() {
    if (stage_pending) CLAST_CK(cudaEventSynchronize(ev_stage));
    stage_pending = false;
    if (staging) CLAST_CK(cudaFreeHost(staging));
    staging = nullptr;
    staging_bytes = 0;
  }
  // the DP's one-hit-per-warp kernel runs on st_dp beside the one-per-thread
  // kernels on st (forked and joined by these events)
  cudaStream_t st_dp = nullptr;
  cudaEvent_t ev_dp_fork = nullptr, ev_dp_join = nullptr;
  // the DP's warp / thread split when CLAST_DP_WARP does not set it: a
  // server's lanes run every hit one per thread (under load, other lanes'
  // work shares the SMs, and one-per-warp hits lost more than they gained)
  int dp_warp = clast::kDpWarpAuto;
};

struct clast_index {
  int l = 0, stride = 0, cut = 0;
  int32_t t_begin = 0;
  int64_t n = 0;
  int32_t nseqs = 0;
  clast::DevArray<char> bases;  // padded
  clast::DevArray<int32_t> gateway, lengths;
  // blocked Bloom filter, 2^(64 - fshift) words of stride fstride from `filter`;
  // windows that are searched together share the memory, their words alternating
  std::shared_ptr<clast::DevArray<uint32_t>> filter_mem;
  uint32_t* filter = nullptr;
  int fstride = 1;
  clast::DevArray<ulonglong2> table;    // 2 * nbuckets records {key, payload}
  clast::DevArray<int2> entries;
  int64_t n_unique = 0, n_keys = 0, n_entries = 0;
  clast::DevArray<int64_t> kept;  // [0]: distinct keys kept after the repeat cut (written by the build)
  uint32_t nbuckets = 1;
  int64_t n_records = 2;
  int fshift = 63;

  clast::IndexView view() const {
    clast::IndexView v;
    v.l = l;
    v.fshift = fshift;
    v.fstride = fstride;
    v.filter = filter;
    v.table = table.p;
    v.nbuckets = nbuckets;
    v.n_records = n_records;
    v.entries = entries.p;
    v.n_keys = n_keys;
    return v;
  }
  clast::TargetView tview() const {
    clast::TargetView t;
    t.bases = bases.p + clast::kPad;
    t.n = n;
    t.gateway = gateway.p;
    t.lengths = lengths.p;
    t.nseqs = nseqs;
    return t;
  }
};

namespace clast {

// Words of the filter of a window of ns samples: about 24 bits per sample,
// between 2^12 and 2^F bits; F = 27 (16 MB: the filters of the two windows a
// group searches stay in L2 beside the streams that pass through it) unless
// CLAST_FILTER_BITS says otherwise (16..32).  Returns fshift.
int filter_shift(int64_t ns);
// Zeroed filter memory for n windows (1 or 2, the words of two alternating).
void alloc_filters(clast_index* const* ix, int n, int fshift, cudaStream_t st);

}  // namespace clast

struct clast_targets {
  clast_ctx* ctx = nullptr;
  struct Win {
    int32_t load, first;  // target load, first record within the load
    std::unique_ptr<clast_index> ix;
  };
  std::vector<Win> wins;
  int32_t n_loads = 0;
  std::vector<int64_t> load_first{0};  // first target record of every load, plus the total
  // The index builds run on the context's stream after clast_targets_create
  // returns; the first clast_map waits for them, reads the overflow count and
  // the build time (events) and reports either.
  clast::DevArray<unsigned long long> failed;
  cudaEvent_t ev_start = nullptr, ev_up = nullptr, ev_done = nullptr;  // from the context's event pool
  mutable bool settled = false;
  int64_t launches = 0;
  ~clast_targets() {
    if (ev_done) cudaEventSynchronize(ev_done);
    for (cudaEvent_t e : {ev_start, ev_up, ev_done})
      if (e) ctx->timer.pool.push_back(e);
  }
};

namespace clast {

// Waits for the index builds of clast_targets_create (once), records their
// time in the context's stats and reports a table overflow.
void settle_targets(clast_ctx* ctx, const clast_targets* T);

inline int fail(clast_ctx* c, int code, const std::string& msg) {
  if (c) c->err = msg;
  return code;
}

// Runs f() and turns every exception into a status code plus message.
template <class F>
int guarded(clast_ctx* ctx, F&& f) {
  try {
    return f();
  } catch (const CudaError& e) {
    return fail(ctx, CLAST_ERR_CUDA, e.what());
  } catch (const std::bad_alloc&) {
    return fail(ctx, CLAST_ERR_NOMEM, "out of memory");
  } catch (const std::invalid_argument& e) {
    return fail(ctx, CLAST_ERR_ARG, e.what());
  } catch (const std::exception& e) {
    return fail(ctx, CLAST_ERR_INTERNAL, e.what());
  }
}

}  // namespace clast
