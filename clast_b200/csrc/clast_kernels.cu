// clast_kernels.cu -- sm_100a kernels of the CLAST seed-and-extend path.
//
// Reference (masayano/CLAST) stages and the kernels that replace them:
//   SRead2bit/SRepelHasOddBase + CDeviceSeqList_query::createHashIndex -> pack_bases, kmer_at
//   CDeviceHashTable (sort_by_key, unique, reduce_by_key, scan, cut)   -> sample_keys,
//       radix_sort_u64, index_place (hash table + Bloom filter for one-probe lookups)
//   createRawSeedList (binarySearch, writeSeedList)                     -> seed_reads, seed_fused
//   deleteSeedsOnSequenceBoundary                                       -> folded into these
//   sortSeeds / deletingIsolateSeeds / deleteDuplicateSeeds             -> seed_reads, seed_filter
//   globalAlign* / localAlign* + calculateEvalue + deleteBadHits        -> banded_dp
//   resultSorting + deleteHits_duplicateResult                          -> final_* (per read)
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <type_traits>
#include <utility>

#include "clast_device.cuh"
#include "clast_kernels.cuh"
#include "clast_workspace.h"

namespace clast {

thread_local int64_t g_kernel_launches = 0;

namespace {

constexpr unsigned kFull = 0xffffffffu;

inline int blocks_for(int64_t n, int threads) { return (int)((n + threads - 1) / threads); }
inline int grid_cap(int64_t want) { return (int)(want < 1 ? 1 : (want > 1048576 ? 1048576 : want)); }

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// ------------------------------------------------------------------------
// exclusive scan
// ------------------------------------------------------------------------
// Exclusive prefix sum over the warp; *total = the warp's sum.
__device__ __forceinline__ int warp_excl_scan(int v, int lane, int* total) {
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  *total = __shfl_sync(kFull, incl, 31);
  return incl - v;
}

constexpr int kScanThreads = 256, kScanItems = 8, kScanTile = kScanThreads * kScanItems;

// Element loader of the scans.
template <class T>
struct ArrayLoad {
  const T* __restrict__ p;
  __device__ __forceinline__ int64_t operator()(int64_t i) const { return (int64_t)p[i]; }
};

// ---- single-pass exclusive scan (decoupled look-back) ----
// Tiles take their index from a counter in launch order, so a tile only waits
// for tiles that have already started.  Each tile publishes its aggregate,
// then its first warp walks back over the predecessors' words, 32 at a time
// (flag in the top two bits: aggregate or inclusive prefix), until it meets an
// inclusive prefix.  The walk waits at most kScanSpinLimit polls per step;
// past that the tile sums the inputs before it directly, so no tile can wait
// for ever.  For non-negative inputs (counts and flags) with sums below 2^62.
constexpr uint64_t kScanAgg = 1ull << 62, kScanInc = 2ull << 62, kScanValue = (1ull << 62) - 1;
constexpr int kScanSpinLimit = 1 << 16;

__device__ __forceinline__ void st_relaxed_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

template <class Load>
__global__ void __launch_bounds__(kScanThreads) k_scan_1pass(Load in, int64_t n_in, int64_t n_out,
                                                             int64_t* __restrict__ out,
                                                             unsigned long long* __restrict__ state,
                                                             long long* __restrict__ total) {
  __shared__ int64_t warp_tot[kScanThreads / 32];
  __shared__ int64_t s_prefix;
  __shared__ unsigned long long s_tile;
  __shared__ int s_fallback;
  unsigned long long* status = state + 1;  // state[0]: the tile counter
  if (threadIdx.x == 0) s_tile = atomicAdd(state, 1ull);
  __syncthreads();
  const int64_t t = (int64_t)s_tile;
  const int64_t base = t * kScanTile + (int64_t)threadIdx.x * kScanItems;
  int64_t v[kScanItems];
  int64_t sum = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const int64_t idx = base + i;
    v[i] = (idx < n_in) ? in(idx) : 0;
    sum += v[i];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  int64_t wpre = 0, tot = 0;
#pragma unroll
  for (int w = 0; w < kScanThreads / 32; ++w) {
    const int64_t x = warp_tot[w];
    if (w < warp) wpre += x;
    tot += x;
  }
  if (warp == 0) {
    int64_t run = 0;
    int fallback = 0;
    if (t == 0) {
      if (lane == 0) st_relaxed_u64(status, kScanInc | (unsigned long long)tot);
    } else {
      if (lane == 0) st_relaxed_u64(status + t, kScanAgg | (unsigned long long)tot);
      for (int64_t j = t - 1;; j -= 32) {
        // lane L reads tile j - L; tiles before 0 read as an inclusive 0
        const int64_t jj = j - lane;
        unsigned long long w = jj >= 0 ? ld_relaxed_u64(status + jj) : kScanInc;
        for (int spin = 0; __any_sync(kFull, (w >> 62) == 0) && spin < kScanSpinLimit; ++spin)
          if ((w >> 62) == 0) w = ld_relaxed_u64(status + jj);
        if (__any_sync(kFull, (w >> 62) == 0)) {
          fallback = 1;
          break;
        }
        const unsigned inc = __ballot_sync(kFull, (w & kScanInc) != 0);
        const int last = inc ? __ffs(inc) - 1 : 31;  // nearest inclusive prefix, else the whole step
        int64_t x = lane <= last ? (int64_t)(w & kScanValue) : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
        run += x;
        if (inc) break;
      }
    }
    if (lane == 0) {
      s_prefix = run;
      s_fallback = fallback;
    }
  }
  __syncthreads();
  if (s_fallback) {  // a predecessor never published: sum the inputs before this tile
    int64_t part = 0;
    for (int64_t i = threadIdx.x; i < t * kScanTile && i < n_in; i += kScanThreads) part += in(i);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(kFull, part, o);
    __syncthreads();
    if (lane == 0) warp_tot[warp] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
      int64_t run = 0;
      for (int w = 0; w < kScanThreads / 32; ++w) run += warp_tot[w];
      s_prefix = run;
      st_relaxed_u64(status + t, kScanInc | (unsigned long long)(run + tot));
    }
    __syncthreads();
  } else if (threadIdx.x == 0 && t > 0) {
    st_relaxed_u64(status + t, kScanInc | (unsigned long long)(s_prefix + tot));
  }
  int64_t run = s_prefix + wpre + incl - sum;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    const int64_t idx = base + i;
    if (idx < n_out) out[idx] = run;
    if (idx == n_in && total) *total = run;
    run += v[i];
  }
}

template <class Load>
void scan_1pass(Workspace& ws, Load in, int64_t n, int64_t* out, cudaStream_t st) {
  const int64_t n_out = n + 1;
  const int64_t tiles = (n_out + kScanTile - 1) / kScanTile;
  unsigned long long* state = ws.get<unsigned long long>("scan1_state", tiles + 1);
  CLAST_CK(cudaMemsetAsync(state, 0, (tiles + 1) * sizeof(unsigned long long), st));
  k_scan_1pass<Load><<<(unsigned)tiles, kScanThreads, 0, st>>>(in, n, n_out, out, state, nullptr);
  CLAST_LAUNCHED();
}


// ------------------------------------------------------------------------
// packing and query strands
// ------------------------------------------------------------------------
// 2-bit codes and non-ACGT flags of 8 bases (x: 8 bytes, first base in the
// low byte), eight at a time in 64-bit words.  code = ((b >> 1) ^ (b >> 2)) & 3
// maps A C G T to 0 1 2 3; a byte is A/C/G/T iff it equals "ACGT"[code].
// codes16: first base in bits 15..14; bad8: first base in bit 7.
__device__ __forceinline__ void pack8(uint64_t x, uint32_t& codes16, uint32_t& bad8) {
  const uint64_t c = ((x >> 1) ^ (x >> 2)) & 0x0303030303030303ull;
  const uint32_t clo = (uint32_t)c, chi = (uint32_t)(c >> 32);
  // byte-reverse so that the first base ends in the top bits, then gather the
  // eight 2-bit fields
  uint64_t y = ((uint64_t)__byte_perm(clo, 0, 0x0123) << 32) | __byte_perm(chi, 0, 0x0123);
  y = (y | (y >> 6)) & 0x000F000F000F000Full;
  y = (y | (y >> 12)) & 0x000000FF000000FFull;
  codes16 = (uint32_t)((y | (y >> 24)) & 0xFFFF);
  uint32_t bad = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t ch = h ? chi : clo;
    const uint32_t sel = (ch & 3u) | ((ch >> 4) & 0x30u) | ((ch >> 8) & 0x300u) | ((ch >> 12) & 0x3000u);
    const uint32_t d = __byte_perm(0x54474341u, 0, sel) ^ (uint32_t)(x >> (32 * h));  // "ACGT"[code] ^ byte
    const uint32_t nz = ((((d & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | d) & 0x80808080u) >> 7;  // 1 per nonzero byte
    bad |= ((nz * 0x08040201u) >> 24 & 0xFu) << (4 * (1 - h));                        // first byte -> bit 3
  }
  bad8 = bad;
}

// One 64-base word per thread: 2-bit codes (first base in the top bits, 32
// per word) and the non-ACGT mask (first base in the top bit).  bases must be
// 16-byte aligned with at least 63 readable bytes past n; bases at or past n
// count as 'N'.
__global__ void k_pack(const char* __restrict__ bases, int64_t n, uint64_t* __restrict__ packed,
                       uint64_t* __restrict__ nmask, int64_t nwords) {
  const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= nwords) return;
  const int64_t f0 = w * 64;
  uint64_t m = 0, p0 = 0, p1 = 0;
  if (f0 < n) {
    const uint4* src = reinterpret_cast<const uint4*>(bases + f0);
    uint64_t g[8];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const uint4 q = __ldcs(src + v);
      g[2 * v] = ((uint64_t)q.y << 32) | q.x;
      g[2 * v + 1] = ((uint64_t)q.w << 32) | q.z;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int64_t valid = n - (f0 + 8 * k);  // bytes of this group before n
      if (valid < 8) {
        const uint64_t keep = valid <= 0 ? 0ull : ((1ull << (8 * valid)) - 1);
        g[k] = (g[k] & keep) | (0x4E4E4E4E4E4E4E4Eull & ~keep);  // 'N'
      }
      uint32_t c16, b8;
      pack8(g[k], c16, b8);
      m |= (uint64_t)b8 << (56 - 8 * k);
      if (k < 4) p0 |= (uint64_t)c16 << (48 - 16 * k);
      else p1 |= (uint64_t)c16 << (48 - 16 * (k - 4));
    }
  } else {
    m = ~0ull;
  }
  nmask[w] = m;
  packed[2 * w] = p0;
  packed[2 * w + 1] = p1;
}

__device__ __forceinline__ char complement(char c) {
  switch (c) {
    case 'A': return 'T';
    case 'T': return 'A';
    case 'G': return 'C';
    case 'C': return 'G';
    default: return 'N';
  }
}

// One warp per read: the '+' strand copy and the reverse complement are both
// coalesced (the reversed writes of a warp still cover one contiguous run).
// The read goes in chunks of 8 x 32 bytes whose loads are all issued before
// the first store, so a short read waits for memory once.  The warp also
// writes the two strands' starts and lengths; the first and last ones the
// kPad 'N' bytes before and after the array.
__global__ void k_strands(const char* __restrict__ reads, const int64_t* __restrict__ off, int64_t n_reads,
                          char* __restrict__ out, int64_t* __restrict__ sstart, int32_t* __restrict__ slen) {
  const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= n_reads) return;
  const int64_t a = off[r], len = off[r + 1] - a;
  if (lane < 2) {
    sstart[2 * r + lane] = 2 * a + lane * len;
    slen[2 * r + lane] = (int32_t)len;
  }
  if (r == 0)
    for (int i = lane; i < kPad; i += 32) out[i - kPad] = 'N';
  if (r == n_reads - 1)
    for (int i = lane; i < kPad; i += 32) out[2 * (a + len) + i] = 'N';
  char* const fwd = out + 2 * a;
  char* const rev = out + 2 * a + 2 * len - 1;  // base j of the read -> rev[-j]
  for (int64_t j0 = 0; j0 < len; j0 += 8 * 32) {
    char c[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int64_t j = j0 + u * 32 + lane;
      c[u] = j < len ? reads[a + j] : 'N';
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int64_t j = j0 + u * 32 + lane;
      if (j < len) {
        fwd[j] = c[u];
        rev[-j] = complement(c[u]);
      }
    }
  }
}

// Shortest and longest read.
__global__ void k_read_lengths(const int64_t* __restrict__ off, int64_t n_reads, int* __restrict__ min_len,
                               int* __restrict__ max_len) {
  int lo = INT_MAX, hi = 0;
  for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_reads; r += (int64_t)gridDim.x * blockDim.x) {
    const int len = (int)(off[r + 1] - off[r]);
    lo = min(lo, len);
    hi = max(hi, len);
  }
  lo = __reduce_min_sync(kFull, lo);
  hi = __reduce_max_sync(kFull, hi);
  if ((threadIdx.x & 31) == 0) {
    atomicMin(min_len, lo);
    atomicMax(max_len, hi);
  }
}

// Base array of one target window: every sequence followed by its first l-1
// bases (utilAddSequence.cu:15-46); joint bases past a sequence shorter than
// l-1 are 'N'.
__global__ void k_build_window(const char* __restrict__ src, const int64_t* __restrict__ src_off,
                               const int32_t* __restrict__ gw, const int32_t* __restrict__ len, int nseqs,
                               int64_t n, char* __restrict__ out) {
  // 16 output bytes per thread, written as one 16-byte store (out is 16-byte aligned)
  __shared__ int first_seq;
  const int64_t i0 = (int64_t)blockIdx.x * blockDim.x * 16;
  if (threadIdx.x == 0) {  // sequence of the block's first base; threads walk forward from it
    int lo = 0, hi = nseqs;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if ((int64_t)gw[mid] <= i0) lo = mid;
      else hi = mid;
    }
    first_seq = lo;
  }
  __syncthreads();
  const int64_t b0 = i0 + (int64_t)threadIdx.x * 16;
  if (b0 >= n) return;
  int lo = first_seq;
  while (lo + 1 < nseqs && (int64_t)gw[lo + 1] <= b0) ++lo;
  unsigned char c[16];
  const int64_t j0 = b0 - gw[lo];
  if (b0 + 16 <= n && j0 + 16 <= (int64_t)len[lo]) {
    // inside one sequence's bases: independent loads
    const char* p = src + src_off[lo] + j0;
#pragma unroll
    for (int k = 0; k < 16; ++k) c[k] = (unsigned char)p[k];
  } else {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const int64_t i = b0 + k;
      while (lo + 1 < nseqs && (int64_t)gw[lo + 1] <= i) ++lo;
      const int64_t j = i - gw[lo];
      const int64_t L = len[lo];
      char v = 'N';
      if (i < n) {
        if (j < L) v = src[src_off[lo] + j];
        else if (j - L < L) v = src[src_off[lo] + (j - L)];
      }
      c[k] = (unsigned char)v;
    }
  }
  if (b0 + 16 <= n) {
    uint4 q;
    q.x = c[0] | (c[1] << 8) | (c[2] << 16) | ((uint32_t)c[3] << 24);
    q.y = c[4] | (c[5] << 8) | (c[6] << 16) | ((uint32_t)c[7] << 24);
    q.z = c[8] | (c[9] << 8) | (c[10] << 16) | ((uint32_t)c[11] << 24);
    q.w = c[12] | (c[13] << 8) | (c[14] << 16) | ((uint32_t)c[15] << 24);
    *reinterpret_cast<uint4*>(out + b0) = q;
  } else {
    for (int k = 0; k < 16 && b0 + k < n; ++k) out[b0 + k] = (char)c[k];
  }
}

// ------------------------------------------------------------------------
// index build
// ------------------------------------------------------------------------
// Sample j of the window: its code (4^l for an l-mer with a non-ACGT base).
// pbits > 0: one sortable word code << pbits | j; pbits = 0: the code, with j
// in vals.
__global__ void k_sample_keys(const uint64_t* __restrict__ packed, const uint64_t* __restrict__ nmask,
                              int64_t ns, int stride, int l, int pbits, uint64_t* __restrict__ items,
                              int32_t* __restrict__ vals) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= ns) return;
  uint64_t key;
  const uint64_t c = kmer_at(packed, nmask, j * stride, l, key) ? order_code(key, l) : (1ull << (2 * l));
  if (pbits > 0) {
    items[j] = (c << pbits) | (uint64_t)j;
  } else {
    items[j] = c;
    vals[j] = (int32_t)j;
  }
}

// ---- LSD radix sort of 64-bit words by a bit range, 8 bits per pass ----
// A block takes a tile of kRsTile consecutive words; warp w owns words
// [w * kRsWarpItems, (w + 1) * kRsWarpItems) of it.  Each pass: per-block digit
// counts (k_rs_hist), one scan of the counts laid out digit-major, then
// k_rs_scatter ranks the tile stably in shared memory and writes every
// digit's run out contiguously.  Ranking takes one step per 32 words: the
// lanes holding the same digit are found with eight ballots (one per digit
// bit), the lowest of them adds the group's size to the warp's counter of that
// digit, and each lane's rank is the counter's old value plus the lanes of its
// group below it.
constexpr int kRsThreads = 256, kRsItems = 16, kRsTile = kRsThreads * kRsItems;
constexpr int kRsWarps = kRsThreads / 32, kRsWarpItems = 32 * kRsItems;

__global__ void __launch_bounds__(kRsThreads) k_rs_hist(const uint64_t* __restrict__ keys, int64_t n, int shift,
                                                        uint32_t* __restrict__ hist, int nblocks) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const int64_t base = (int64_t)blockIdx.x * kRsTile;
#pragma unroll 4
  for (int r = 0; r < kRsItems; ++r) {
    const int64_t idx = base + r * kRsThreads + threadIdx.x;
    if (idx < n) atomicAdd(&h[(keys[idx] >> shift) & 255], 1u);
  }
  __syncthreads();
  hist[(int64_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// Lanes of the warp whose 8-bit digit equals this lane's, among the lanes in `among`.
__device__ __forceinline__ unsigned digit_peers(unsigned d, unsigned among) {
  unsigned peers = among;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const unsigned bit = (d >> b) & 1u;
    const unsigned bb = __ballot_sync(kFull, bit);
    peers &= bit ? bb : ~bb;
  }
  return peers;
}

// PAY: a 32-bit value travels with every word (vin -> vout).  Dynamic shared
// memory: the staged tile, kRsTile words (+ kRsTile values).
template <bool PAY>
__global__ void __launch_bounds__(kRsThreads, 3) k_rs_scatter(const uint64_t* __restrict__ kin,
                                                           const int32_t* __restrict__ vin,
                                                           uint64_t* __restrict__ kout, int32_t* __restrict__ vout,
                                                           int64_t n, int shift, const int64_t* __restrict__ offs,
                                                           int nblocks) {
  __shared__ uint32_t wc[kRsWarps][256];  // per-warp digit counters, then the warps' run starts
  __shared__ uint32_t tile_start[256];
  __shared__ uint32_t wsum[kRsWarps];
  __shared__ int64_t goff[256];
  extern __shared__ uint64_t stage[];
  int32_t* stage_v = reinterpret_cast<int32_t*>(stage + kRsTile);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  goff[tid] = offs[(int64_t)tid * nblocks + blockIdx.x];
#pragma unroll
  for (int w = 0; w < kRsWarps; ++w) wc[w][tid] = 0;
  const int64_t base = (int64_t)blockIdx.x * kRsTile + (int64_t)warp * kRsWarpItems;
  const unsigned lt = lanemask_lt();
  uint64_t k[kRsItems];
  int32_t v[PAY ? kRsItems : 1];
#pragma unroll
  for (int r = 0; r < kRsItems; ++r) {
    const int64_t idx = base + r * 32 + lane;
    k[r] = idx < n ? kin[idx] : 0ull;
    if (PAY) v[r] = idx < n ? vin[idx] : 0;
  }
  __syncthreads();
  // stable ranks within the warp's runs, two 16-bit ranks per register
  uint32_t rk[kRsItems / 2];
#pragma unroll
  for (int r = 0; r < kRsItems; ++r) {
    const bool ok = base + r * 32 + lane < n;
    const unsigned d = (unsigned)(k[r] >> shift) & 255u;
    const unsigned peers = digit_peers(d, __ballot_sync(kFull, ok));
    const int leader = __ffs(peers) - 1;  // -1 only for a lane past n
    uint32_t old = 0;
    if (ok && lane == leader) old = atomicAdd(&wc[warp][d], (uint32_t)__popc(peers));
    old = __shfl_sync(kFull, old, leader & 31);
    const uint32_t rank = old + (uint32_t)__popc(peers & lt);
    if (r & 1) rk[r >> 1] |= rank << 16;
    else rk[r >> 1] = rank;
  }
  __syncthreads();
  // digit d = tid: tile-wide start (exclusive scan over digits), then the
  // start of each warp's run of that digit
  uint32_t tot = 0;
#pragma unroll
  for (int w = 0; w < kRsWarps; ++w) tot += wc[w][tid];
  uint32_t incl = tot;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  uint32_t start = incl - tot;
  for (int w = 0; w < warp; ++w) start += wsum[w];
  tile_start[tid] = start;
#pragma unroll
  for (int w = 0; w < kRsWarps; ++w) {
    const uint32_t c = wc[w][tid];
    wc[w][tid] = start;
    start += c;
  }
  __syncthreads();
  // stage the tile in sorted order
#pragma unroll
  for (int r = 0; r < kRsItems; ++r) {
    if (base + r * 32 + lane < n) {
      const unsigned d = (unsigned)(k[r] >> shift) & 255u;
      const uint32_t at = wc[warp][d] + ((rk[r >> 1] >> (16 * (r & 1))) & 0xffffu);
      stage[at] = k[r];
      if (PAY) stage_v[at] = v[r];
    }
  }
  __syncthreads();
  // digit runs out, contiguous
  const int64_t tile0 = (int64_t)blockIdx.x * kRsTile;
  const int valid = (int)min((int64_t)kRsTile, n - tile0);
  for (int i = tid; i < valid; i += kRsThreads) {
    const uint64_t w = stage[i];
    const unsigned d = (unsigned)((w >> shift) & 255);
    const int64_t at = goff[d] + (i - (int)tile_start[d]);
    kout[at] = w;
    if (PAY) vout[at] = stage_v[i];
  }
}

// ---- the index from the sorted samples, in one pass ----
// A tile of kIxTile sorted samples is one block's.  Equal codes form runs; a
// run belongs to the tile that holds its first sample, and the repeat cut
// counts all of its samples.  The kept samples of a run (not cut, not on a
// joint) go to `entries` from the run's first index on, so that no count of
// the kept ones before it is needed.  Every run that keeps a sample is a
// record of the hash table.  The codes arrive ascending, so their home records
// do too, and linear probing puts record u at max(home_u, pos_{u-1} + 1): for a
// tile that starts after the free position x, at u + max(max_{j <= u} (home_j -
// j), x) with u counted within the tile.  A tile that holds C records and ends
// at A for x = 0 therefore maps x to max(A, x + C); x comes from a decoupled
// look-back over those pairs, one word each (flag, C, A).  Tiles take their
// number from a counter in launch order, so a tile waits only for tiles that
// have started, and at most kScanSpinLimit polls per step: past that it counts
// into *failed, which the host reports.
//
// 8 bytes read and 40 written per sample (the table's free half included), and
// one random atomic per code for the filter; bound by instructions (506 per
// sample, half of the issue slots) and the waits at its barriers (38 % of the
// stalls), at a quarter of the memory rate.  The fourteen kernels this replaced
// (heads, two scans, unique codes, kept samples, entries, bucket bounds, a scan
// of the kept codes, a two-level running maximum, placement) wrote and read
// some 120 bytes per sample in between: index of a 250 Mbp window (50 M samples)
// 6.28 to 3.80 ms; with the free records written here too, instead of the whole
// table before, and five blocks per SM (48 registers, 92 bytes spilled; four:
// 3.70) 3.63.
constexpr int kIxThreads = 256, kIxRounds = 4, kIxTile = kIxThreads * kIxRounds;
constexpr int kIxWarps = kIxThreads / 32, kIxWarpItems = 32 * kIxRounds;

template <bool PAIR>
__device__ __forceinline__ uint64_t ix_code(const uint64_t* __restrict__ items, int pbits, int64_t i) {
  return PAIR ? items[i] : items[i] >> pbits;
}
// Sequence and index of the sample at window position pos (onTargetBoundary: a
// sample that reaches into the joint is none, x = -1).
__device__ __forceinline__ int2 ix_resolve(int64_t pos, int l, const int32_t* __restrict__ gw,
                                           const int32_t* __restrict__ len, int nseqs) {
  int lo = 0, hi = nseqs;  // last sequence starting at or before pos
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if ((int64_t)gw[mid] <= pos) lo = mid;
    else hi = mid;
  }
  const int tidx = (int)(pos - gw[lo]);
  return (int64_t)tidx + l > (int64_t)len[lo] ? make_int2(-1, 0) : make_int2(lo, tidx);
}

// Exclusive prefix over the block's warps of v (one value per warp); *total = their sum.
__device__ __forceinline__ int ix_warp_prefix(int v, int* __restrict__ buf, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) buf[warp] = v;
  __syncthreads();
  int before = 0, all = 0;
#pragma unroll
  for (int w = 0; w < kIxWarps; ++w) {
    const int x = buf[w];
    if (w < warp) before += x;
    all += x;
  }
  __syncthreads();
  *total = all;
  return before;
}

// Sets the filter bits of the l-mer of code c.
__device__ __forceinline__ void filter_set(uint32_t* __restrict__ filter, int fshift, int fstride, uint64_t c, int l) {
  const uint64_t key = key_of_code(c, l), rc = key_revcomp(key, l);
  const uint64_t h = filter_hash(key < rc ? key : rc, l);
  atomicOr(filter + (size_t)filter_word(h, fshift) * fstride, filter_mask(h, key > rc));
}

// The filter of a table's keys: as searched, or (FILE) as index files hold it.
template <bool FILE>
__global__ void k_filter_from_table(const ulonglong2* __restrict__ table, int64_t n_records, int l,
                                    uint32_t* __restrict__ filter, int fshift, int fstride) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_records) return;
  const ulonglong2 r = table[i];
  if (r.y == kNoPayload) return;
  if (FILE) {
    const uint64_t h = file_filter_hash(r.x);
    atomicOr(filter + filter_word(h, fshift), file_filter_mask(h));
  } else {
    filter_set(filter, fshift, fstride, r.x, l);
  }
}

// Free records.  Most lie between two records of a tile and are written with
// them, so that a sector of the table is written whole and once.  What a long
// free stretch covers of the table's chunks of kIxChunk records is only marked
// here and filled by k_index_free, which has the whole GPU for it (a window of
// N's is one such stretch).
constexpr int kIxChunkLog = 12, kIxChunk = 1 << kIxChunkLog, kIxOwnFree = 32;

// [from, to) of the table; every lane of the warp takes part.
__device__ __forceinline__ void ix_free(ulonglong2* __restrict__ table, unsigned char* __restrict__ chunk_free,
                                        int64_t from, int64_t to) {
  const int lane = threadIdx.x & 31;
  const ulonglong2 free_rec = make_ulonglong2(~0ull, kNoPayload);
  const int64_t a = (from + kIxChunk - 1) >> kIxChunkLog, z = to >> kIxChunkLog;
  const int64_t head = z > a ? a << kIxChunkLog : to;
  for (int64_t i = from + lane; i < head; i += 32) table[i] = free_rec;
  if (z > a) {
    for (int64_t c = a + lane; c < z; c += 32) chunk_free[c] = 1;
    for (int64_t i = (z << kIxChunkLog) + lane; i < to; i += 32) table[i] = free_rec;
  }
}

__global__ void __launch_bounds__(256) k_index_free(ulonglong2* __restrict__ table,
                                                    const unsigned char* __restrict__ chunk_free, int64_t chunks) {
  for (int64_t c = blockIdx.x; c < chunks; c += gridDim.x) {
    if (!chunk_free[c]) continue;  // the same for the whole block
    for (int i = threadIdx.x; i < kIxChunk; i += 256)
      table[(c << kIxChunkLog) + i] = make_ulonglong2(~0ull, kNoPayload);
  }
}

// The samples at the start of a tile that belong to a run begun in an earlier
// tile.  With the repeat cut off, or above kIxLongRun, such a run can span any
// number of tiles, and whether it has a record at all (samples on joints are
// none) may only show in its last one.  So k_index_leads looks at all tiles'
// before the placement, the tile that holds a run's first sample adds them up,
// a word per tile, and k_index_lead_entries writes their entries after it: no
// tile waits for another one's walk over samples.  Stride 1 without a cut, index
// of a 60 Mbp window of poly-A 4.3 ms, of one with 100 runs of 100 kbp 4.15, of
// 400,000 records of 14 A's 8.7; with one block walking each such run 54.6, 14.7
// and no index (the later tiles' waits ran out).  Windows without such runs pay
// two launches: 1.00 against 0.97 ms for 12 M samples.
struct IndexLead {
  int32_t kept;   // samples of them that no joint holds
  int32_t whole;  // the run goes on past the tile
  int2 first;     // the first kept one
  int64_t to;     // where the kept ones go in the entries; -1: the run is cut
};
// Runs that pass a repeat cut of up to this are seen whole by one step of a block.
constexpr int kIxLongRun = kIxThreads;

struct IndexBuild {
  const uint64_t* items;  // sorted: code << pbits | sample, or codes with the samples in vals (pbits 0)
  const int32_t* vals;
  int64_t ns;
  int pbits;
  uint64_t bound;  // codes from here on are l-mers with a non-ACGT base
  int stride, l, cut;
  const int32_t* gw;
  const int32_t* len;
  int nseqs;
  uint32_t nbuckets;
  int2* entries;
  ulonglong2* table;
  int64_t n_records;
  uint32_t* filter;
  int fshift, fstride;
  unsigned long long* state;  // [0] tile counter, then one word per tile
  unsigned char* chunk_free;  // per whole chunk of the table: no record lies in it
  IndexLead* leads;           // per tile, with the cut off or above kIxLongRun
  unsigned long long* kept;   // records placed
  unsigned long long* failed;
};

template <bool PAIR>
__global__ void __launch_bounds__(kIxThreads) k_index_leads(IndexBuild b) {
  __shared__ int s_first;
  const int64_t t = blockIdx.x, i0 = t * kIxTile;
  const uint64_t c = ix_code<PAIR>(b.items, b.pbits, i0);
  IndexLead* const lead = b.leads + t;
  if (t == 0 || c >= b.bound || ix_code<PAIR>(b.items, b.pbits, i0 - 1) != c) {  // the same for the whole block
    if (threadIdx.x == 0) *lead = IndexLead{0, 0, make_int2(-1, 0), -1};
    return;
  }
  if (threadIdx.x == 0) s_first = kIxTile;
  __syncthreads();
  const uint64_t pmask = PAIR ? 0 : (1ull << b.pbits) - 1;
  int kept = 0, mine = kIxTile;
  int2 r_mine = make_int2(-1, 0);
#pragma unroll
  for (int j = kIxRounds - 1; j >= 0; --j) {
    const int k = j * kIxThreads + (int)threadIdx.x;
    bool keep = false;
    if (i0 + k < b.ns) {
      const uint64_t w = b.items[i0 + k];
      if ((PAIR ? w : w >> b.pbits) == c) {
        const int2 r = ix_resolve((int64_t)(PAIR ? b.vals[i0 + k] : (int)(w & pmask)) * b.stride, b.l, b.gw, b.len, b.nseqs);
        keep = r.x >= 0;
        if (keep) {
          mine = k;
          r_mine = r;
        }
      }
    }
    kept += __syncthreads_count(keep);
  }
  if (mine < kIxTile) atomicMin(&s_first, mine);
  __syncthreads();
  if (kept ? mine == s_first : threadIdx.x == 0) {
    const int64_t next = i0 + kIxTile;
    *lead = IndexLead{kept, next < b.ns && ix_code<PAIR>(b.items, b.pbits, next) == c, r_mine, -1};
  }
}

// LONG: the cut is off or above kIxLongRun (see IndexLead).
template <bool PAIR, bool LONG>
__global__ void __launch_bounds__(kIxThreads, 5) k_index_place(IndexBuild b) {
  __shared__ uint64_t code[kIxTile + 1];
  __shared__ int2 res[kIxTile];
  __shared__ uint16_t start[kIxTile + 1];  // first sample of every run of the tile
  __shared__ uint16_t kpre[kIxTile + 1];   // kept samples before sample k
  __shared__ uint16_t first[kIxTile];      // first kept sample of the run that starts at k
  __shared__ int wbuf[kIxWarps];
  __shared__ int64_t wmax[kIxWarps];
  __shared__ uint64_t s_prev;
  __shared__ unsigned long long s_tile;
  __shared__ int64_t s_x;
  __shared__ int2 s_cross;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = lanemask_lt();
  unsigned long long* status = b.state + 1;
  if (tid == 0) s_tile = atomicAdd(b.state, 1ull);
  __syncthreads();
  const int64_t t = (int64_t)s_tile, i0 = t * kIxTile;
  const int nt = (int)min((int64_t)kIxTile, b.ns - i0);
  const uint64_t pmask = PAIR ? 0 : (1ull << b.pbits) - 1;
  int pos[kIxRounds];
#pragma unroll
  for (int j = 0; j < kIxRounds; ++j) {
    const int k = warp * kIxWarpItems + j * 32 + lane;
    uint64_t c = ~0ull;
    pos[j] = 0;
    if (k < nt) {
      const uint64_t w = b.items[i0 + k];
      c = PAIR ? w : w >> b.pbits;
      pos[j] = PAIR ? b.vals[i0 + k] : (int)(w & pmask);
    }
    code[k] = c;
  }
  if (tid == 0) {
    code[kIxTile] = i0 + kIxTile < b.ns ? ix_code<PAIR>(b.items, b.pbits, i0 + kIxTile) : ~0ull;
    s_prev = i0 > 0 ? ix_code<PAIR>(b.items, b.pbits, i0 - 1) : ~0ull;
  }
  __syncthreads();
  // runs: rid[j] = the run of this thread's sample within the tile (-1: it began before the tile)
  int rid[kIxRounds];
  unsigned started = 0;
  int n_runs;
  {
    unsigned m[kIxRounds];
    int n = 0;
#pragma unroll
    for (int j = 0; j < kIxRounds; ++j) {
      const int k = warp * kIxWarpItems + j * 32 + lane;
      const bool st = k < nt && (k == 0 ? s_prev : code[k - 1]) != code[k];
      m[j] = __ballot_sync(kFull, st);
      rid[j] = n + __popc(m[j] & lt) + (st ? 1 : 0) - 1;
      started |= (st ? 1u : 0u) << j;
      n += __popc(m[j]);
    }
    const int before = ix_warp_prefix(n, wbuf, &n_runs);
#pragma unroll
    for (int j = 0; j < kIxRounds; ++j) {
      rid[j] += before;
      if ((started >> j) & 1u) start[rid[j]] = (uint16_t)(warp * kIxWarpItems + j * 32 + lane);
    }
    if (tid == 0) start[n_runs] = (uint16_t)nt;
  }
  __syncthreads();
  // the last run may go on past the tile
  const uint64_t last_code = n_runs > 0 ? code[start[n_runs - 1]] : ~0ull;
  const bool cross = n_runs > 0 && nt == kIxTile && last_code < b.bound && code[kIxTile] == last_code;
  bool cross_pass = false;  // it passes the cut: codes ascend, so it has `cut` samples if the one cut - 1 on is its own
  if (cross) {
    const int64_t at_cut = i0 + start[n_runs - 1] + b.cut - 1;
    cross_pass = b.cut == -1 ||
                 (b.cut > 0 && !(at_cut < b.ns && ix_code<PAIR>(b.items, b.pbits, at_cut) == last_code));
  }
  // kept samples
  unsigned kept = 0;
  {
    unsigned m[kIxRounds];
    int n = 0;
#pragma unroll
    for (int j = 0; j < kIxRounds; ++j) {
      const int k = warp * kIxWarpItems + j * 32 + lane;
      bool keep = false;
      const bool last = cross && rid[j] == n_runs - 1;
      if (k < nt && code[k] < b.bound && rid[j] >= 0 && (LONG || !last)) {
        const int cnt = start[rid[j] + 1] - start[rid[j]];
        if (LONG && last ? cross_pass : b.cut == -1 || cnt < b.cut) {  // removeRepeatedSequence
          const int2 r = ix_resolve((int64_t)pos[j] * b.stride, b.l, b.gw, b.len, b.nseqs);
          keep = r.x >= 0;
          res[k] = r;
        }
      }
      m[j] = __ballot_sync(kFull, keep);
      kept |= (keep ? 1u : 0u) << j;
      n += __popc(m[j]);
    }
    int total;
    int at = ix_warp_prefix(n, wbuf, &total);
#pragma unroll
    for (int j = 0; j < kIxRounds; ++j) {
      kpre[warp * kIxWarpItems + j * 32 + lane] = (uint16_t)(at + __popc(m[j] & lt));
      at += __popc(m[j]);
    }
    if (tid == 0) kpre[kIxTile] = (uint16_t)total;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kIxRounds; ++j)
    if ((kept >> j) & 1u) {
      const int k = warp * kIxWarpItems + j * 32 + lane, h = start[rid[j]];
      const int rank = kpre[k] - kpre[h];
      b.entries[i0 + h + rank] = res[k];
      if (rank == 0) first[h] = (uint16_t)k;
    }
  // A run that goes on past the tile: its samples from there on that are kept.
  // A run that passes a cut of up to kIxLongRun ends within one step of the block.
  int cross_kept = 0;
  if (cross_pass && !LONG) {
    const int64_t h = i0 + start[n_runs - 1], i = h + tid;
    int2 r = make_int2(-1, 0);
    if (i < b.ns) {
      const uint64_t w = b.items[i];
      if ((PAIR ? w : w >> b.pbits) == last_code)
        r = ix_resolve((int64_t)(PAIR ? b.vals[i] : (int)(w & pmask)) * b.stride, b.l, b.gw, b.len, b.nseqs);
    }
    const unsigned m = __ballot_sync(kFull, r.x >= 0);
    const int at = ix_warp_prefix(__popc(m), wbuf, &cross_kept) + __popc(m & lt);
    if (r.x >= 0) {
      b.entries[h + at] = r;
      if (at == 0) s_cross = r;
    }
  }
  int own = 0;  // kept samples of that run within the tile
  if (cross_pass && LONG) {
    own = kpre[kIxTile] - kpre[start[n_runs - 1]];
    const int64_t h = i0 + start[n_runs - 1] + own;
    for (int64_t u = t + 1;; u += kIxThreads) {
      IndexLead* const lead = b.leads + u + tid;
      const bool in = u + tid < (int64_t)gridDim.x;
      const int k0 = in ? lead->kept : 0;
      const unsigned ends = __ballot_sync(kFull, !in || !lead->whole);
      if (lane == 0) wbuf[warp] = ends ? 1 : 0;
      __syncthreads();
      bool part = !(ends & lt), done = false;  // the run's tiles: up to the first one that it does not fill
#pragma unroll
      for (int w = 0; w < kIxWarps; ++w) {
        if (w < warp && wbuf[w]) part = false;
        if (wbuf[w]) done = true;
      }
      __syncthreads();
      int all;
      const int k = part ? k0 : 0, before = warp_excl_scan(k, lane, &all);
      const int at = ix_warp_prefix(all, wbuf, &all) + before;
      if (k > 0) {
        lead->to = h + cross_kept + at;
        if (own == 0 && cross_kept + at == 0) s_cross = lead->first;
      }
      cross_kept += all;
      if (done) break;
    }
    if (own > 0 && tid == 0) s_cross = res[first[start[n_runs - 1]]];
    cross_kept += own;
  }
  __syncthreads();
  // records: u = rank within the tile, slack = home - u, the maximum of the records before
  unsigned rec = 0;
  int u[kIxRounds], kc[kIxRounds];
  int64_t run[kIxRounds], home[kIxRounds];
  int n_rec;
  int64_t tile_max = INT64_MIN;
  {
    unsigned m[kIxRounds];
    int n = 0;
#pragma unroll
    for (int j = 0; j < kIxRounds; ++j) {
      const int k = warp * kIxWarpItems + j * 32 + lane;
      kc[j] = 0;
      home[j] = 0;
      if ((started >> j) & 1u) {
        const bool c = cross && rid[j] == n_runs - 1;
        kc[j] = c ? cross_kept : kpre[start[rid[j] + 1]] - kpre[k];
        if (kc[j] > 0) home[j] = record_home(code[k], b.l, b.nbuckets);
      }
      m[j] = __ballot_sync(kFull, kc[j] > 0);
      u[j] = n + __popc(m[j] & lt);
      rec |= (kc[j] > 0 ? 1u : 0u) << j;
      n += __popc(m[j]);
    }
    const int before = ix_warp_prefix(n, wbuf, &n_rec);
    int64_t carry = INT64_MIN;
#pragma unroll
    for (int j = 0; j < kIxRounds; ++j) {
      u[j] += before;
      int64_t v = (rec >> j) & 1u ? home[j] - u[j] : INT64_MIN;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(kFull, v, o);
        if (lane >= o && y > v) v = y;
      }
      int64_t y = __shfl_up_sync(kFull, v, 1);
      if (lane == 0) y = INT64_MIN;
      run[j] = y > carry ? y : carry;
      y = __shfl_sync(kFull, v, 31);
      if (y > carry) carry = y;
    }
    if (lane == 0) wmax[warp] = carry;
    __syncthreads();
    int64_t pre = INT64_MIN;
#pragma unroll
    for (int w = 0; w < kIxWarps; ++w) {
      const int64_t x = wmax[w];
      if (w < warp && x > pre) pre = x;
      if (x > tile_max) tile_max = x;
    }
#pragma unroll
    for (int j = 0; j < kIxRounds; ++j) run[j] = run[j] > pre ? run[j] : pre;
  }
  // x: the position after the records of all earlier tiles
  if (warp == 0) {
    const int64_t A = n_rec > 0 ? n_rec + tile_max : 0;
    int64_t x = 0;
    if (t > 0) {
      if (lane == 0) st_relaxed_u64(status + t, kScanAgg | ((unsigned long long)n_rec << 50) | (unsigned long long)A);
      int64_t after = 0;  // records of the tiles walked over
      for (int64_t j = t - 1;; j -= 32) {
        const int64_t jj = j - lane;
        unsigned long long w = jj >= 0 ? ld_relaxed_u64(status + jj) : kScanInc;
        for (int spin = 0; __any_sync(kFull, (w >> 62) == 0) && spin < kScanSpinLimit; ++spin)
          if ((w >> 62) == 0) w = ld_relaxed_u64(status + jj);
        if (__any_sync(kFull, (w >> 62) == 0)) {
          if (lane == 0) atomicAdd(b.failed, 1ull);
          break;
        }
        const unsigned inc = __ballot_sync(kFull, (w & kScanInc) != 0);
        const int last = inc ? __ffs(inc) - 1 : 31;
        const bool whole = (w & kScanInc) != 0;  // an inclusive position, else a pair
        const int64_t C = lane <= last && !whole ? (int64_t)((w >> 50) & 0xfff) : 0;
        int64_t incl = C;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int64_t y = __shfl_up_sync(kFull, incl, o);
          if (lane >= o) incl += y;
        }
        int64_t v = lane <= last ? (int64_t)(whole ? w & kScanValue : w & ((1ull << 50) - 1)) + after + incl - C : 0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const int64_t y = __shfl_xor_sync(kFull, v, o);
          v = y > v ? y : v;
        }
        x = v > x ? v : x;
        after += __shfl_sync(kFull, incl, 31);
        if (inc) break;
      }
    }
    if (lane == 0) {
      const int64_t end = A > x + n_rec ? A : x + n_rec;
      st_relaxed_u64(status + t, kScanInc | (unsigned long long)end);
      s_x = x;
      if (n_rec) atomicAdd(b.kept, (unsigned long long)n_rec);
    }
    if (t == (int64_t)gridDim.x - 1) ix_free(b.table, b.chunk_free, A > x + n_rec ? A : x + n_rec, b.n_records);
  }
  __syncthreads();
  const int64_t x = s_x;
#pragma unroll
  for (int j = 0; j < kIxRounds; ++j) {
    // the free records between the record before this one and this one: [from, at)
    const int64_t from = u[j] + (run[j] > x ? run[j] : x);
    int64_t at = from;
    if ((rec >> j) & 1u) {
      const int k = warp * kIxWarpItems + j * 32 + lane;
      const uint64_t c = code[k];
      filter_set(b.filter, b.fshift, b.fstride, c, b.l);
      uint64_t payload;
      if (kc[j] == 1) {
        const int2 e = cross && rid[j] == n_runs - 1 ? s_cross : res[first[k]];
        payload = ((uint64_t)(uint32_t)e.x << 32) | (uint32_t)e.y;
      } else {
        payload = kMulti | ((uint64_t)(i0 + k) << 32) | (uint32_t)kc[j];
      }
      if (home[j] > from) at = home[j];
      if (from >= 0 && at < b.n_records) {
        if (at - from <= kIxOwnFree)
          for (int64_t i = from; i < at; ++i) b.table[i] = make_ulonglong2(~0ull, kNoPayload);
        b.table[at] = make_ulonglong2(c, payload);
      } else {  // unreachable: positions rise to the last one, which the table holds
        atomicAdd(b.failed, 1ull);
        at = from;
      }
    }
    for (unsigned far = __ballot_sync(kFull, at - from > kIxOwnFree); far; far &= far - 1) {
      const int src = __ffs(far) - 1;
      ix_free(b.table, b.chunk_free, __shfl_sync(kFull, from, src), __shfl_sync(kFull, at, src));
    }
  }
}

// The entries of the leads (see IndexLead) whose run has a record.
template <bool PAIR>
__global__ void __launch_bounds__(kIxThreads) k_index_lead_entries(IndexBuild b, int64_t tiles) {
  __shared__ int wbuf[kIxWarps];
  const int tid = threadIdx.x, lane = tid & 31;
  const uint64_t pmask = PAIR ? 0 : (1ull << b.pbits) - 1;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const int64_t i0 = t * kIxTile;
    int64_t to = b.leads[t].to;
    if (b.leads[t].kept == 0 || to < 0) continue;  // the same for the whole block
    const uint64_t c = ix_code<PAIR>(b.items, b.pbits, i0);
    for (int j = 0; j < kIxRounds; ++j) {
      const int64_t i = i0 + j * kIxThreads + tid;
      int2 r = make_int2(-1, 0);
      if (i < b.ns) {
        const uint64_t w = b.items[i];
        if ((PAIR ? w : w >> b.pbits) == c)
          r = ix_resolve((int64_t)(PAIR ? b.vals[i] : (int)(w & pmask)) * b.stride, b.l, b.gw, b.len, b.nseqs);
      }
      const unsigned m = __ballot_sync(kFull, r.x >= 0);
      int all;
      const int at = ix_warp_prefix(__popc(m), wbuf, &all) + __popc(m & lanemask_lt());
      if (r.x >= 0) b.entries[to + at] = r;
      to += all;
    }
  }
}

// ------------------------------------------------------------------------
// seeds
// ------------------------------------------------------------------------
// Seeding in one pass, one warp per strand.  The strand's l-mers go in rounds
// of 32 * kSeedPerLane; in a round lane L takes the kSeedPerLane consecutive
// l-mers from L * kSeedPerLane, so it reads their 2-bit words and N flags once
// and shifts each key out of them.  The lookups of a round are issued
// together, level by level (2-bit words and N flags → filter words → home
// buckets), so a strand waits about one latency per level.  Round 0's results
// are staged for the write pass while the range reservation is in flight (one
// round covers 160 l-mers: a 164 bp strand); later rounds are looked up again
// when written.  The strand's seeds get one
// contiguous range from an atomic cursor; if the range would pass `cap`,
// nothing is written and the host reruns with a larger buffer (the cursor then
// holds the exact total).  Seeds are written in l-mer order, so the seeds of a
// strand on one diagonal arrive already sorted.
constexpr int kSeedPerLane = 5;
constexpr int kSeedRound = 32 * kSeedPerLane;

// Both records of a home bucket: one 256-bit streaming load (sm_100), the
// address 32-byte aligned (home records are even, the table 256-byte aligned).
__device__ __forceinline__ void ld_bucket(const ulonglong2* a, uint64_t& c0, uint64_t& p0, uint64_t& c1,
                                          uint64_t& p1) {
  asm volatile("ld.global.cs.v4.u64 {%0, %1, %2, %3}, [%4];" : "=l"(c0), "=l"(p0), "=l"(c1), "=l"(p1) : "l"(a));
}

// (hi << s) | (lo >> (64 - s)) for s in [0, 63]: the 64 bits from bit s of hi:lo
__device__ __forceinline__ uint64_t funnel64(uint64_t hi, uint64_t lo, int s) {
  return (hi << s) | ((lo >> 1) >> (63 - s));
}

// Payloads of the l-mers qi = r0 + lane * P + i (i < P) of a strand; invalid or
// absent ones get kNoPayload (the key search of krnlBinarySearch.cu:3-33 and
// the bucket read of writeSeedList).  Returns the number of valid l-mers.
template <bool SMALL>
__device__ __forceinline__ int round_lookup(const QueryView& q, const IndexView& ix, int64_t st, int nk, int r0,
                                            int lane, uint64_t (&pl)[kSeedPerLane]) {
  constexpr int P = kSeedPerLane;
  const int q0 = r0 + lane * P;
  const int nv = max(0, min(P, nk - q0));  // valid l-mer slots of this lane
  uint64_t code[P];
  uint32_t vmask = 0;
  if (nv > 0) {
    const int64_t f = st + q0;
    // The lane's P l-mers span P - 1 + l <= 35 bases from f: their 2-bit words
    // and non-ACGT flags are read in one batch.  An l-mer with a non-ACGT base
    // is not looked up (SRepelHasOddBase).
    vmask = (1u << nv) - 1;
    if (SMALL) {
      // 16-base units j0 .. j0 + 2 of the codes, 32-base units k0, k0 + 1 of
      // the flags (unit j = 32-bit element j ^ 1)
      const uint32_t* p32 = reinterpret_cast<const uint32_t*>(q.packed);
      const uint32_t* n32 = reinterpret_cast<const uint32_t*>(q.nmask);
      const int64_t j0 = f >> 4, k0 = f >> 5;
      const uint32_t u0 = __ldcs(p32 + (j0 ^ 1)), u1 = __ldcs(p32 + ((j0 + 1) ^ 1)),
                     u2 = __ldcs(p32 + ((j0 + 2) ^ 1));
      const uint32_t m0 = __ldcs(n32 + (k0 ^ 1)), m1 = __ldcs(n32 + ((k0 + 1) ^ 1));
      const uint32_t nflag = __funnelshift_l(m1, m0, (int)(f & 31));  // base f in the top bit
      const int o = 2 * (int)(f & 15);
      const uint32_t mask = (2 * ix.l == 32) ? ~0u : ((1u << (2 * ix.l)) - 1);
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const int bo = o + 2 * i;
        const uint32_t x = bo < 32 ? __funnelshift_l(u1, u0, bo) : __funnelshift_l(u2, u1, bo - 32);
        const uint32_t key = x >> (32 - 2 * ix.l);
        code[i] = (uint32_t)(key * (uint32_t)0x6659FD93u) & mask;  // order_code for l <= 16
        if ((nflag << i) >> (32 - ix.l)) vmask &= ~(1u << i);
      }
    } else {
      // 32-base words w0 .. w0 + 2 of the codes, 64-base words k0, k0 + 1 of the flags
      const int64_t w0 = f >> 5, k0 = f >> 6;
      const uint64_t u0 = ld_stream(q.packed + w0), u1 = ld_stream(q.packed + w0 + 1),
                     u2 = ld_stream(q.packed + w0 + 2);
      const uint64_t nflag = funnel64(ld_stream(q.nmask + k0), ld_stream(q.nmask + k0 + 1), (int)(f & 63));
      const int o = 2 * (int)(f & 31);
#pragma unroll
      for (int i = 0; i < P; ++i) {
        const int bo = o + 2 * i;  // < 2 * (31 + P)
        const uint64_t x = bo < 64 ? funnel64(u0, u1, bo) : funnel64(u1, u2, bo - 64);
        code[i] = order_code(x >> (64 - 2 * ix.l), ix.l);
        if ((nflag << i) >> (64 - ix.l)) vmask &= ~(1u << i);
      }
    }
  }
  uint32_t fw[P], fm[P];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const uint64_t key = key_of_code(code[i], ix.l), rc = key_revcomp(key, ix.l);
    const uint64_t h = filter_hash(key < rc ? key : rc, ix.l);
    fm[i] = filter_mask(h, key > rc);
    fw[i] = ((vmask >> i) & 1u) ? __ldg(ix.filter + (size_t)filter_word(h, ix.fshift) * ix.fstride) : 0u;
  }
  // The home bucket (records home and home + 1, one aligned 32-byte sector)
  // in one load; only keys displaced past it probe further.
  uint64_t c0[P], p0[P], c1[P], p1[P];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const bool pass = ((vmask >> i) & 1u) && (fw[i] & fm[i]) == fm[i];
    c0[i] = 0ull;
    p0[i] = kNoPayload;
    c1[i] = 0ull;
    p1[i] = kNoPayload;
    if (pass)
      ld_bucket(ix.table + (SMALL ? record_home16((uint32_t)code[i], ix.l, ix.nbuckets)
                                  : record_home(code[i], ix.l, ix.nbuckets)),
                c0[i], p0[i], c1[i], p1[i]);
  }
#pragma unroll
  for (int i = 0; i < P; ++i) {
    if (c0[i] == code[i] || p0[i] == kNoPayload) pl[i] = p0[i];
    else if (c1[i] == code[i] || p1[i] == kNoPayload) pl[i] = p1[i];
    else pl[i] = table_probe(ix, code[i], record_home(code[i], ix.l, ix.nbuckets) + 2);
  }
  return __popc(vmask);
}

// Writes the seed of entry e (sequence within window, index within sequence)
// for l-mer qi at w; tlen = length of sequence e.x (global mode only).
__device__ __forceinline__ void seed_store(int2 e, int qi, int tlen, int gap, int local, int qlen, int64_t w,
                                           int& valid, uint64_t* __restrict__ skey, uint32_t* __restrict__ sq) {
  const int s0 = e.y - qi;  // tHitStartIdx, is_onCorner
  const bool drop = !local && ((s0 + gap < 0) || (s0 + qlen - gap > tlen));
  // streaming stores: the seeds must not evict the filter from L2
  __stcs(reinterpret_cast<unsigned long long*>(skey + w),
         drop ? kDroppedSeed : (((uint64_t)(uint32_t)e.x << 32) | ((uint32_t)s0 ^ 0x80000000u)));
  __stcs(sq + w, (uint32_t)qi);
  valid += drop ? 0 : 1;
}

// Writes the c = payload_count(pl) seeds of l-mer qi at w onwards.
__device__ __forceinline__ void seed_put(const IndexView& ix, const TargetView& t, int gap, int local, int qlen,
                                         int qi, uint64_t pl, int64_t w, int& valid, uint64_t* __restrict__ skey,
                                         uint32_t* __restrict__ sq) {
  const int c = payload_count(pl);
  const bool multi = (pl & kMulti) != 0;
  const int us = (int)(pl >> 32) & 0x7fffffff;
  for (int i = 0; i < c; ++i) {
    const int2 e = multi ? __ldcs(ix.entries + us + i) : make_int2((int)(pl >> 32), (int)(uint32_t)pl);
    seed_store(e, qi, local ? 0 : t.lengths[e.x], gap, local, qlen, w + i, valid, skey, sq);
  }
}

// Writes a round's seeds (lane L's l-mers r0 + L*P .. in order, lanes in
// order) from w onwards and advances w past them.  When every l-mer of the
// round has at most one entry, the payloads go through the warp's slice of
// shared memory (stage_pl / stage_qi, kSeedRound entries) so that lane j
// writes seed j; otherwise each lane writes its own.
__device__ __forceinline__ void round_emit(const IndexView& ix, const TargetView& t, int gap, int local, int qlen,
                                           int r0, int lane, const uint64_t (&pl)[kSeedPerLane], int64_t& w,
                                           int& valid, uint64_t* __restrict__ skey, uint32_t* __restrict__ sq,
                                           uint64_t* stage_pl, int32_t* stage_qi) {
  int cnt = 0;
  bool multi = false;
#pragma unroll
  for (int i = 0; i < kSeedPerLane; ++i) {
    const int c = payload_count(pl[i]);
    cnt += c;
    multi |= c > 1;
  }
  int round_total;
  const int excl = warp_excl_scan(cnt, lane, &round_total);
  if (!__any_sync(kFull, multi)) {
    int k = excl;
#pragma unroll
    for (int i = 0; i < kSeedPerLane; ++i)
      if (pl[i] != kNoPayload) {
        stage_pl[k] = pl[i];
        stage_qi[k] = r0 + lane * kSeedPerLane + i;
        ++k;
      }
    __syncwarp();
    for (int j = lane; j < round_total; j += 32) seed_put(ix, t, gap, local, qlen, stage_qi[j], stage_pl[j], w + j,
                                                         valid, skey, sq);
    __syncwarp();
  } else {
    int64_t wl = w + excl;
#pragma unroll
    for (int i = 0; i < kSeedPerLane; ++i)
      if (pl[i] != kNoPayload) {
        seed_put(ix, t, gap, local, qlen, r0 + lane * kSeedPerLane + i, pl[i], wl, valid, skey, sq);
        wl += payload_count(pl[i]);
      }
  }
  w += round_total;
}

constexpr int kSeedFusedThreads = 64;  // two strands per block: blocks retire at a finer grain than with four
constexpr int kSeedPrefetchBlocks = 2048;

// The seed buffer is split into kSeedParts partitions of part_cap seeds, each
// with its own cursor; strand s takes its range in partition s % kSeedParts, so
// the range reservations of neighbouring warps hit different counters.
// SMALL: l <= 16, keys read with 32-bit funnel shifts.
template <bool SMALL>
__global__ void __launch_bounds__(kSeedFusedThreads, SMALL ? 16 : 12) k_seed_fused(QueryView q, IndexView ix, TargetView t, int gap,
                                                                   int local, unsigned long long* __restrict__ cursor,
                                                                   unsigned long long* __restrict__ n_kmers,
                                                                   int64_t* __restrict__ off, int32_t* __restrict__ cnt,
                                                                   int32_t* __restrict__ nvalid,
                                                                   uint64_t* __restrict__ skey,
                                                                   uint32_t* __restrict__ sq, int64_t part_cap) {
  constexpr int P = kSeedPerLane;
  __shared__ uint64_t stage_pl[kSeedFusedThreads / 32][kSeedRound];
  __shared__ int32_t stage_qi[kSeedFusedThreads / 32][kSeedRound];
  const int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  if (s >= q.nstrands) return;
  const int64_t st = q.start[s];
  const int qlen = q.len[s];
  const int nk = qlen - ix.l + 1;
  // L2 prefetch for the block kSeedPrefetchBlocks later: its strand table
  // entries and, estimated from this strand's start and the mean strand
  // length, its 2-bit words and N flags, so that its first loads hit L2.
  // Every address stays inside its array.
  if (wib == 0 && lane < 5) {
    const int64_t sp = ((int64_t)blockIdx.x + kSeedPrefetchBlocks) * (kSeedFusedThreads / 32);
    if (sp < q.nstrands && q.n > 0) {
      const int64_t f = min(q.n - 1, st + (sp - s) * (q.n / q.nstrands));
      const void* a = lane == 0 ? (const void*)(q.start + sp)
                    : lane == 1 ? (const void*)(q.len + sp)
                    : lane == 4 ? (const void*)(q.nmask + (f >> 6))
                                : (const void*)(q.packed + min((f >> 5) + 16 * (lane - 2), q.n / 32 + 3));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
    }
  }
  uint64_t pl0[P];
  int valid_kmers = round_lookup<SMALL>(q, ix, st, nk, 0, lane, pl0);
  int lane_cnt = 0;
  bool multi0 = false;
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const int c = payload_count(pl0[i]);
    lane_cnt += c;
    multi0 |= c > 1;
  }
  // Round 0 is staged before its range is known: in the single-entry case
  // lane j takes seed j of the round and reads its sequence length now, so
  // that the load overlaps the range reservation below.
  int rt0;
  const int excl0 = warp_excl_scan(lane_cnt, lane, &rt0);
  const bool simple0 = !__any_sync(kFull, multi0);
  uint64_t* const spl = stage_pl[wib];
  int32_t* const sqi = stage_qi[wib];
  uint64_t pl_j = kNoPayload;
  int qi_j = 0, tl_j = 0;
  if (simple0) {
    int k = excl0;
#pragma unroll
    for (int i = 0; i < P; ++i)
      if (pl0[i] != kNoPayload) {
        spl[k] = pl0[i];
        sqi[k] = lane * P + i;
        ++k;
      }
    __syncwarp();
    if (lane < rt0) {
      pl_j = spl[lane];
      qi_j = sqi[lane];
      if (!local) tl_j = t.lengths[(int)(pl_j >> 32)];
    }
  } else {
    // the payloads wait in the lane's own stage slots
#pragma unroll
    for (int i = 0; i < P; ++i) spl[lane * P + i] = pl0[i];
  }
  for (int r0 = kSeedRound; r0 < nk; r0 += kSeedRound) {
    uint64_t pl[P];
    valid_kmers += round_lookup<SMALL>(q, ix, st, nk, r0, lane, pl);
#pragma unroll
    for (int i = 0; i < P; ++i) lane_cnt += payload_count(pl[i]);
  }
  const int total = (int)__reduce_add_sync(kFull, (unsigned)lane_cnt);
  valid_kmers = (int)__reduce_add_sync(kFull, (unsigned)valid_kmers);
  const int part = (int)(s % kSeedParts);
  unsigned long long rel = 0;
  if (lane == 0) {
    if (valid_kmers) atomicAdd(n_kmers + part, (unsigned long long)valid_kmers);
    rel = total ? atomicAdd(&cursor[part], (unsigned long long)total) : 0ull;
  }
  rel = __shfl_sync(kFull, rel, 0);
  const unsigned long long base = (unsigned long long)part * (unsigned long long)part_cap + rel;
  if (lane == 0) {
    off[s] = (int64_t)base;
    cnt[s] = total;
  }
  const int64_t cap = (int64_t)(part + 1) * part_cap;
  if (total == 0 || (int64_t)(base + total) > cap) {
    if (lane == 0) nvalid[s] = 0;
    return;
  }
  int valid = 0;
  int64_t w = (int64_t)base;
  if (simple0) {
    if (lane < rt0)
      seed_store(make_int2((int)(pl_j >> 32), (int)(uint32_t)pl_j), qi_j, tl_j, gap, local, qlen, w + lane, valid,
                 skey, sq);
    for (int j = lane + 32; j < rt0; j += 32) seed_put(ix, t, gap, local, qlen, sqi[j], spl[j], w + j, valid, skey, sq);
  } else {
    int64_t wl = w + excl0;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const uint64_t pl = spl[lane * P + i];
      if (pl != kNoPayload) {
        seed_put(ix, t, gap, local, qlen, lane * P + i, pl, wl, valid, skey, sq);
        wl += payload_count(pl);
      }
    }
  }
  __syncwarp();
  w += rt0;
  for (int r0 = kSeedRound; r0 < nk; r0 += kSeedRound) {
    uint64_t pl[P];
    round_lookup<SMALL>(q, ix, st, nk, r0, lane, pl);
    round_emit(ix, t, gap, local, qlen, r0, lane, pl, w, valid, skey, sq, spl, sqi);
  }
  valid = (int)__reduce_add_sync(kFull, (unsigned)valid);
  if (lane == 0) nvalid[s] = valid;
}

// ---- sorting networks (ascending compare-exchange, safe with a ragged tail) ----
template <class K2>
__device__ __forceinline__ bool less2(uint64_t a1, K2 a2, uint64_t b1, K2 b2) {
  return a1 < b1 || (a1 == b1 && a2 < b2);
}

template <class K2>
__device__ __forceinline__ void cta_network(uint64_t* s1, K2* s2, int n) {
  int np = 1;
  while (np < n) np <<= 1;
  for (int size = 2; size <= np; size <<= 1) {
    for (int i = threadIdx.x; i < np / 2; i += blockDim.x) {  // flip stage
      const int blk = i / (size / 2), r = i % (size / 2);
      const int a = blk * size + r, b = blk * size + size - 1 - r;
      if (b < n && less2(s1[b], s2[b], s1[a], s2[a])) {
        const uint64_t t1 = s1[a]; s1[a] = s1[b]; s1[b] = t1;
        const K2 t2 = s2[a]; s2[a] = s2[b]; s2[b] = t2;
      }
    }
    __syncthreads();
    for (int stride = size >> 2; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < np / 2; i += blockDim.x) {
        const int blk = i / stride, r = i % stride;
        const int a = blk * 2 * stride + r, b = a + stride;
        if (b < n && less2(s1[b], s2[b], s1[a], s2[a])) {
          const uint64_t t1 = s1[a]; s1[a] = s1[b]; s1[b] = t1;
          const K2 t2 = s2[a]; s2[a] = s2[b]; s2[b] = t2;
        }
      }
      __syncthreads();
    }
  }
}

// Compare-exchange of a network step held one element per lane: the lower
// lane of the pair keeps the smaller element.
template <class K2>
__device__ __forceinline__ void warp_cx(uint64_t& a1, K2& a2, int lane, int partner) {
  const uint64_t b1 = __shfl_sync(kFull, a1, partner);
  const K2 b2 = __shfl_sync(kFull, a2, partner);
  const bool b_less = less2(b1, b2, a1, a2);
  if (lane < partner ? b_less : !b_less && (b1 != a1 || b2 != a2)) { a1 = b1; a2 = b2; }
}
// Sorts every group of N lanes (N a power of two up to 32).
template <int N, class K2>
__device__ __forceinline__ void lanes_sort(uint64_t& a1, K2& a2, int lane) {
#pragma unroll
  for (int size = 2; size <= N; size <<= 1) {
    warp_cx(a1, a2, lane, lane ^ (size - 1));
#pragma unroll
    for (int stride = size >> 2; stride > 0; stride >>= 1) warp_cx(a1, a2, lane, lane ^ stride);
  }
}

constexpr int kCtaSortCap = 2048;

// is "s" near its predecessor "p" (hasNotNearPair / hasNearPair, same strand)
__device__ __forceinline__ bool near_pred(int tid, int tidx, int diag, int ptid, int ptidx, int pdiag,
                                          int width, int gap) {
  return tid == ptid && width >= tidx - ptidx && width >= ptidx - tidx && gap >= pdiag - diag;
}


constexpr int kWarpSmemCap = 256;

// ------------------------------------------------------------------------
// Seeding of whole reads in a group of target windows
// ------------------------------------------------------------------------
// One warp per read looks the l-mers of both its strands up in all NW windows:
// the l-mer at position i of the '+' strand and its reverse complement, at
// position len - l - i of the '-' strand, come from the same words of the '+'
// strand and share their filter word, and the words of two windows lie side by
// side, so one 8-byte load answers four look-ups.  The (l-mer, strand, window)
// that pass a filter are listed in the warp's shared memory, and the lanes
// share the bucket reads, two in flight each.  Seeds gather by slot (strand,
// window) in shared memory; with at most kSlotSeeds per slot, which most reads
// stay under, the warp sorts and filters them there (four slots of up to eight
// seeds at once), so that only the hits reach memory.  A read of more than
// kFastRounds rounds of kSeedRound l-mers, or with a fuller slot, is left to
// k_seed_reads_long, which writes its seeds for the tiers of the seed filter.
//
// Bound by issue (0.66 per cycle and scheduler, some 1,900 warp instructions per
// read of 150 bp) with the latency of the filter and bucket reads.  One warp per
// strand with a load per strand, l-mer and window, and every seed through
// memory into the filters, took on a million reads against two windows 4.17 ms
// for the seeds and 1.00 ms for the filters, against 3.05 and 0.46 ms now; on
// 10,000 reads of 100 - 5,000 bp 0.85 against 0.56 ms, on 300 bp reads 0.50
// against 0.36 ms.  (The same with the long reads in this kernel ran out of the
// instruction cache: 5.45 ms.)
constexpr int kSlotSeeds = 32;
constexpr int kFastRounds = 3;  // reads of up to 480 l-mers may stay in shared memory

template <bool SMALL>
struct SeedKey {
  typedef uint64_t K;
};
template <>
struct SeedKey<true> {
  typedef uint32_t K;
};

template <bool SMALL, int NW>
struct ListSmem {
  static constexpr int kList = 2 * NW * kSeedRound;
  typename SeedKey<SMALL>::K code[kList];
  uint16_t tag[kList];  // l-mer within the round << 3 | slot
};

// Keys of the lane's l-mers q0 .. q0 + P - 1 (from strand position st + q0) and
// of their reverse complements; bit i of the result: l-mer i has bases A/C/G/T
// only.
template <bool SMALL>
__device__ __forceinline__ uint32_t lane_keys(const QueryView& q, int64_t f, int nv, int l,
                                              typename SeedKey<SMALL>::K (&kf)[kSeedPerLane],
                                              typename SeedKey<SMALL>::K (&kr)[kSeedPerLane]) {
  constexpr int P = kSeedPerLane;
  uint32_t vmask = (1u << nv) - 1;
  if constexpr (SMALL) {
    // 16-base units j0 .. j0 + 2 of the codes, 32-base units k0, k0 + 1 of
    // the flags (unit j = 32-bit element j ^ 1)
    const uint32_t* p32 = reinterpret_cast<const uint32_t*>(q.packed);
    const uint32_t* n32 = reinterpret_cast<const uint32_t*>(q.nmask);
    const int64_t j0 = f >> 4, k0 = f >> 5;
    const uint32_t u0 = __ldcs(p32 + (j0 ^ 1)), u1 = __ldcs(p32 + ((j0 + 1) ^ 1)), u2 = __ldcs(p32 + ((j0 + 2) ^ 1));
    const uint32_t m0 = __ldcs(n32 + (k0 ^ 1)), m1 = __ldcs(n32 + ((k0 + 1) ^ 1));
    const uint32_t nflag = __funnelshift_l(m1, m0, (int)(f & 31));  // base f in the top bit
    const int o = 2 * (int)(f & 15);
    const uint32_t mask = l == 16 ? ~0u : (1u << (2 * l)) - 1;
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int bo = o + 2 * i;
      const uint32_t x = bo < 32 ? __funnelshift_l(u1, u0, bo) : __funnelshift_l(u2, u1, bo - 32);
      const uint32_t y = __brev(~x);
      kf[i] = x >> (32 - 2 * l);
      kr[i] = (((y >> 1) & 0x55555555u) | ((y & 0x55555555u) << 1)) & mask;
      if ((nflag << i) >> (32 - l)) vmask &= ~(1u << i);
    }
  } else {
    // 32-base words w0 .. w0 + 2 of the codes, 64-base words k0, k0 + 1 of the flags
    const int64_t w0 = f >> 5, k0 = f >> 6;
    const uint64_t u0 = ld_stream(q.packed + w0), u1 = ld_stream(q.packed + w0 + 1), u2 = ld_stream(q.packed + w0 + 2);
    const uint64_t nflag = funnel64(ld_stream(q.nmask + k0), ld_stream(q.nmask + k0 + 1), (int)(f & 63));
    const int o = 2 * (int)(f & 31);
#pragma unroll
    for (int i = 0; i < P; ++i) {
      const int bo = o + 2 * i;  // < 2 * (31 + P)
      const uint64_t x = bo < 64 ? funnel64(u0, u1, bo) : funnel64(u1, u2, bo - 64);
      kf[i] = x >> (64 - 2 * l);
      kr[i] = key_revcomp(kf[i], l);
      if ((nflag << i) >> (64 - l)) vmask &= ~(1u << i);
    }
  }
  return vmask;
}

// Lists the (l-mer, slot) of a round that pass the windows' filters, in l-mer
// order; returns their number.  *valid is raised by the lane's valid l-mers.
template <bool SMALL, int NW>
__device__ __forceinline__ int round_list(const QueryView& q, const SeedWins& W, int64_t st, int nk, int r0, int lane,
                                          ListSmem<SMALL, NW>& sm, int& valid) {
  typedef typename SeedKey<SMALL>::K K;
  constexpr int P = kSeedPerLane, NS = 2 * NW;
  const int l = W.w[0].ix.l;
  const int q0 = r0 + lane * P;
  const int nv = max(0, min(P, nk - q0));
  K kf[P], kr[P];
  uint32_t vmask = 0;
#pragma unroll
  for (int i = 0; i < P; ++i) kf[i] = kr[i] = 0;
  if (nv > 0) vmask = lane_keys<SMALL>(q, st + q0, nv, l, kf, kr);
  valid += __popc(vmask);
  // the filter words of every window, all in flight together
  uint32_t fw[P][NW], low[P];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const K smaller = kf[i] < kr[i] ? kf[i] : kr[i];
    const uint64_t h = SMALL ? filter_hash16((uint32_t)smaller) : filter_hash((uint64_t)smaller, l);
    low[i] = (uint32_t)h;
    const bool on = (vmask >> i) & 1u;
#pragma unroll
    for (int w = 0; w < NW; ++w) fw[i][w] = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      const IndexView& ix = W.w[w].ix;
      if (w % 2 == 1 && W.w[w].paired) continue;
      const uint32_t* a = ix.filter + (size_t)filter_word(h, ix.fshift) * ix.fstride;
      if (w + 1 < NW && W.w[w + 1 < NW ? w + 1 : w].paired) {
        if (on) {
          const uint2 x = __ldg(reinterpret_cast<const uint2*>(a));
          fw[i][w] = x.x;
          fw[i][w + 1 < NW ? w + 1 : w] = x.y;
        }
      } else if (on) {
        fw[i][w] = __ldg(a);
      }
    }
  }
  typedef std::conditional_t<(P * NS <= 32), uint32_t, uint64_t> Mask;
  Mask pass = 0;  // bit i * NS + slot
#pragma unroll
  for (int i = 0; i < P; ++i) {
    if (!((vmask >> i) & 1u)) continue;
    const uint32_t ms = filter_bits3(low[i]), ml = filter_bits3(low[i] >> 15);
    const uint32_t mf = kf[i] > kr[i] ? ml : ms, mr = kr[i] > kf[i] ? ml : ms;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      if ((fw[i][w] & mf) == mf) pass |= (Mask)1 << (i * NS + 2 * w);
      if ((fw[i][w] & mr) == mr) pass |= (Mask)1 << (i * NS + 2 * w + 1);
    }
  }
  int total;
  int k = warp_excl_scan(__popcll(pass), lane, &total);
  const K mult = SMALL ? (K)0x6659FD93u : (K)0xD6E8FEB86659FD93ull;  // order_code
  const K mask = 2 * l == 8 * (int)sizeof(K) ? ~(K)0 : ((K)1 << (2 * l)) - 1;
#pragma unroll
  for (int i = 0; i < P; ++i) {
    uint32_t m = (uint32_t)(pass >> (i * NS)) & ((1u << NS) - 1);
    while (m) {
      const int x = __ffs(m) - 1;
      m &= m - 1;
      sm.code[k] = ((x & 1 ? kr[i] : kf[i]) * mult) & mask;
      sm.tag[k] = (uint16_t)((lane * P + i) << 3 | x);
      ++k;
    }
  }
  __syncwarp();
  return total;
}

// The home buckets of list entries j (kNoPayload past the list) and their tags:
// two per lane in flight.
template <bool SMALL, int NW>
__device__ __forceinline__ void list_payloads(const SeedWins& W, const ListSmem<SMALL, NW>& sm, int c0, int lane,
                                              int total, uint64_t (&pl)[2], int (&tag)[2]) {
  const int l = W.w[0].ix.l;
  uint64_t b0[2], b1[2], b2[2], b3[2];
  int64_t home[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int j = c0 + 32 * u + lane;
    const bool in = j < total;
    tag[u] = in ? sm.tag[j] : 0;
    b0[u] = b2[u] = 0;
    b1[u] = b3[u] = kNoPayload;
    home[u] = 0;
    if (in) {
      const IndexView& ix = W.w[(tag[u] & 7) >> 1].ix;
      home[u] = SMALL ? record_home16((uint32_t)sm.code[j], l, ix.nbuckets) : record_home(sm.code[j], l, ix.nbuckets);
      ld_bucket(ix.table + home[u], b0[u], b1[u], b2[u], b3[u]);
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int j = c0 + 32 * u + lane;
    pl[u] = kNoPayload;
    if (j < total) {
      const uint64_t c = sm.code[j];
      if (b0[u] == c || b1[u] == kNoPayload) pl[u] = b1[u];
      else if (b2[u] == c || b3[u] == kNoPayload) pl[u] = b3[u];
      else pl[u] = table_probe(W.w[(tag[u] & 7) >> 1].ix, c, home[u] + 2);
    }
  }
}

// Index of the l-mer of `tag` within its strand.
__device__ __forceinline__ int tag_qidx(int tag, int r0, int nk) {
  const int i = r0 + (tag >> 3);
  return tag & 1 ? nk - 1 - i : i;
}
// The seed of entry e of l-mer qi: its key, kDroppedSeed for is_onCorner.
__device__ __forceinline__ uint64_t seed_key(const SeedWins& W, int slot, int2 e, int qi, int gap, int local, int qlen) {
  const int s0 = e.y - qi;  // tHitStartIdx
  if (!local && ((s0 + gap < 0) || (s0 + qlen - gap > W.w[slot >> 1].t.lengths[e.x]))) return kDroppedSeed;
  return ((uint64_t)(uint32_t)e.x << 32) | ((uint32_t)s0 ^ 0x80000000u);
}
// Entry i of payload pl.
__device__ __forceinline__ int2 payload_entry(const SeedWins& W, int slot, uint64_t pl, int i) {
  if (pl & kMulti) return __ldcs(W.w[slot >> 1].ix.entries + ((int)(pl >> 32) & 0x7fffffff) + i);
  return make_int2((int)(pl >> 32), (int)(uint32_t)pl);
}
// The lane whose items (the warp's, lane after lane; lane L's first is number
// first_L) hold item t.
__device__ __forceinline__ int item_lane(int first, int t) {
  int src = 0;
#pragma unroll
  for (int step = 16; step > 0; step >>= 1)
    if (__shfl_sync(kFull, first, src + step) <= t) src += step;
  return src;
}

// A seed as one sortable word, (sequence, diagonal, l-mer), for sequences below
// 2^20 and l-mers below 2^12.
constexpr int kWordQBits = 12;
__device__ __forceinline__ uint64_t seed_word(uint64_t key, int qi) {
  return ((key >> 32) << (32 + kWordQBits)) | ((uint64_t)(uint32_t)key << kWordQBits) | (uint32_t)qi;
}
__device__ __forceinline__ int word_seq(uint64_t k) { return (int)(k >> (32 + kWordQBits)); }
__device__ __forceinline__ uint32_t word_diag(uint64_t k) { return (uint32_t)(k >> kWordQBits); }
__device__ __forceinline__ int word_q(uint64_t k) { return (int)(k & ((1u << kWordQBits) - 1)); }
__device__ __forceinline__ uint64_t word_key(uint64_t k) { return ((uint64_t)word_seq(k) << 32) | word_diag(k); }

// One slot's seed words, one per lane of a group of G lanes (a power of two; n
// of them, the j-th in lane j): sorts them and applies the isolate and
// duplicate filters as filter_chunk does, the slot not being its query window's
// first.  Returns whether this lane's seed is a hit; near = whether the group's
// first seed that survives the isolate filter is near the slot's first seed
// (k_window_first).
__device__ __forceinline__ bool slot_filter(uint64_t& k, int n, int G, unsigned group, int width, int gap, bool& near) {
  const int lane = threadIdx.x & 31, j = lane & (G - 1);
  const uint64_t n1 = __shfl_down_sync(kFull, k, 1);
  if (__any_sync(kFull, j + 1 < n && n1 < k)) {
#pragma unroll 1
    for (int size = 2; size <= G; size <<= 1)
#pragma unroll 1
      for (int m = size - 1; m > 0; m = m == size - 1 ? size >> 2 : m >> 1) {
        const uint64_t o = __shfl_xor_sync(kFull, k, m);
        if ((lane & m) < ((lane ^ m) & m) ? o < k : o > k) k = o;
      }
  }
  const int tid = word_seq(k), diag = (int)(word_diag(k) ^ 0x80000000u), tidx = diag + word_q(k);
  const int ptid = __shfl_up_sync(kFull, tid, 1), ptidx = __shfl_up_sync(kFull, tidx, 1);
  const int pdiag = __shfl_up_sync(kFull, diag, 1);
  const bool keep8 = j > 0 && j < n && near_pred(tid, tidx, diag, ptid, ptidx, pdiag, width, gap);
  const unsigned kept = __ballot_sync(kFull, keep8);
  near = false;
  if (kept == 0) return false;
  const unsigned below = kept & group & lanemask_lt();
  // the previous survivor, or for the first one the slot's first seed
  const int src = below ? 31 - __clz(below) : lane & ~(G - 1);
  const int stid = __shfl_sync(kFull, tid, src), stidx = __shfl_sync(kFull, tidx, src);
  const int sdiag = __shfl_sync(kFull, diag, src);
  const bool dup = keep8 && near_pred(tid, tidx, diag, stid, stidx, sdiag, width, gap);
  near = (__ballot_sync(kFull, dup && !below) & group) != 0;
  return keep8 && !(dup && below);
}

template <bool SMALL, int NW>
struct ReadSmem {
  uint64_t word[2 * NW][kSlotSeeds];  // valid seeds per slot, then hits
  int n[2 * NW];                      // their counts
  ListSmem<SMALL, NW> list;
};

template <bool SMALL, int NW>
__global__ void __launch_bounds__(kSeedFusedThreads, NW <= 2 ? 18 : 8) k_seed_reads(QueryView q, SeedWins W, int width,
                                                                                  int gap, int local) {
  constexpr int NS = 2 * NW;                           // the read's slots
  constexpr int kG = NW == 1 ? 16 : NW == 2 ? 8 : 4;   // lanes per slot when all are filtered at once
  __shared__ ReadSmem<SMALL, NW> smem[kSeedFusedThreads / 32];
  const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int64_t n_reads = q.nstrands / 2;
  if (r >= n_reads) return;
  ReadSmem<SMALL, NW>& sm = smem[wib];
  const int64_t st = q.start[2 * r];
  const int qlen = q.len[2 * r];
  const int nk = qlen - W.w[0].ix.l + 1;
  const int64_t v0 = r * NS;
  const unsigned lt = lanemask_lt();
  // L2 prefetch for the block kSeedPrefetchBlocks later: its strand table
  // entries and, estimated from this read's start and the mean strand length,
  // its 2-bit words and N flags.  Every address stays inside its array.
  if (wib == 0 && lane < 4) {
    const int64_t rp = ((int64_t)blockIdx.x + kSeedPrefetchBlocks) * (kSeedFusedThreads / 32);
    if (rp < n_reads && q.n > 0) {
      const int64_t f = min(q.n - 1, st + (rp - r) * 2 * (q.n / q.nstrands));
      const void* a = lane == 0 ? (const void*)(q.start + 2 * rp)
                    : lane == 1 ? (const void*)(q.len + 2 * rp)
                    : lane == 2 ? (const void*)(q.nmask + (f >> 6))
                                : (const void*)(q.packed + min(f >> 5, q.n / 32 + 3));
      asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
    }
  }
  if (nk <= 0) {
    if (lane < NS) W.nvalid[v0 + lane] = W.cnt[v0 + lane] = W.hcnt[v0 + lane] = 0;
    return;
  }
  bool fast = nk <= kFastRounds * kSeedRound && W.words;
  int valid_kmers = 0;
  int seeds[NW];  // entries found per window, the ones on a corner among them
#pragma unroll
  for (int w = 0; w < NW; ++w) seeds[w] = 0;
  if (lane < NS) sm.n[lane] = 0;
#pragma unroll 1
  for (int r0 = 0; r0 < nk && fast; r0 += kSeedRound) {
    __syncwarp();
    const int total = round_list<SMALL, NW>(q, W, st, nk, r0, lane, sm.list, valid_kmers);
#pragma unroll 1
    for (int c0 = 0; c0 < total && fast; c0 += 64) {
      uint64_t pl2[2];
      int tag2[2];
      list_payloads(W, sm.list, c0, lane, total, pl2, tag2);
#pragma unroll 1
      for (int u = 0; u < 2; ++u) {
        const uint64_t pl = u ? pl2[1] : pl2[0];
        const int tag = u ? tag2[1] : tag2[0];
        const int c = payload_count(pl);
        const unsigned found = __ballot_sync(kFull, c > 0);
        if (!found) continue;
#pragma unroll
        for (int w = 0; w < NW; ++w) seeds[w] += ((tag & 7) >> 1) == w ? c : 0;
        const unsigned multi = __ballot_sync(kFull, c > 1);
        int all, first = 0;
        if (multi) {
          first = warp_excl_scan(c, lane, &all);
          if (all > NS * kSlotSeeds) {  // too many for the slots
            fast = false;
            break;
          }
        } else {
          all = 32;  // an entry per lane, as they lie
        }
#pragma unroll 1
        for (int t0 = 0; t0 < all; t0 += 32) {
          int tg = tag, i = 0;
          uint64_t p = pl;
          bool in = c > 0;
          if (multi) {
            const int t = t0 + lane, src = item_lane(first, t);
            in = t < all;
            p = __shfl_sync(kFull, pl, src);
            tg = __shfl_sync(kFull, tag, src);
            i = t - __shfl_sync(kFull, first, src);
          }
          const int slot = tg & 7, qi = tag_qidx(tg, r0, nk);
          uint64_t key = kDroppedSeed;
          if (in) key = seed_key(W, slot, payload_entry(W, slot, p, i), qi, gap, local, qlen);
          const bool ok = key != kDroppedSeed;
          const unsigned peers = __match_any_sync(kFull, ok ? slot : 8);
          const int leader = __ffs(peers) - 1;
          int at = 0;
          if (ok && lane == leader) at = atomicAdd(&sm.n[slot], __popc(peers));
          at = __shfl_sync(kFull, at, leader) + __popc(peers & lt);
          if (ok && at < kSlotSeeds) sm.word[slot][at] = seed_word(key, qi);
        }
      }
      __syncwarp();
      if (__any_sync(kFull, sm.n[lane < NS ? lane : 0] > kSlotSeeds)) fast = false;
    }
  }
  if (!fast) {  // k_seed_reads_long's: reads of one round from the list's start, longer ones from its end
    if (lane == 0) {
      if (nk <= kSeedRound) W.long_reads[atomicAdd(W.n_long, 1)] = (uint32_t)r;
      else W.long_reads[n_reads - 1 - atomicAdd(W.n_long + 1, 1)] = (uint32_t)r;
    }
    return;
  }
  const int part = (int)(r % kSeedParts);
  const int64_t cap = W.part_cap * NW;  // the group's windows share a partition
  valid_kmers = (int)__reduce_add_sync(kFull, (unsigned)valid_kmers);
#pragma unroll
  for (int w = 0; w < NW; ++w) {
    const int n = (int)__reduce_add_sync(kFull, (unsigned)seeds[w]);
    if (lane == w) {
      if (valid_kmers) atomicAdd(W.w[w].n_kmers + part, 2ull * (unsigned long long)valid_kmers);
      if (n) atomicAdd(W.w[w].n_seeds + part, (unsigned long long)n);
    }
  }
  const int n_slot = lane < NS ? sm.n[lane < NS ? lane : 0] : 0;  // lane x < NS: valid seeds of slot x
  if (lane < NS) {
    W.nvalid[v0 + lane] = n_slot;
    W.cnt[v0 + lane] = 0;  // nothing left to filter
  }
  if (!__any_sync(kFull, n_slot > 0)) {
    if (lane < NS) W.hcnt[v0 + lane] = 0;
    return;
  }
  // every slot of up to kG seeds at once, a group of lanes each; then each fuller one with the whole warp
  unsigned todo = __ballot_sync(kFull, n_slot > kG);
  int h_slot = 0;  // lane x < NS: hits of slot x
  int x = lane / kG, G = kG;
  unsigned group = ((1u << kG) - 1) << (lane & ~(kG - 1));
  int n = __shfl_sync(kFull, n_slot, x < NS ? x : 0);
  if (x >= NS || n > kG) n = 0;
#pragma unroll 1
  for (bool groups = true;; groups = false) {
    if (!groups) {
      if (!todo) break;
      x = __ffs(todo) - 1;
      todo &= todo - 1;
      G = 32;
      group = kFull;
      n = __shfl_sync(kFull, n_slot, x);
    }
    const int j = lane & (G - 1);
    uint64_t k = j < n ? sm.word[x][j] : ~0ull;
    bool near;
    const bool hit = slot_filter(k, n, G, group, width, gap, near);
    if (j == 0 && n > 0) {  // the slot's hit if it is its query window's first
      W.first_key[v0 + x] = word_key(k);
      W.first_q[v0 + x] = (uint32_t)word_q(k) | (near ? 0x80000000u : 0u);
    }
    const unsigned m = __ballot_sync(kFull, hit);
    if (hit) sm.word[x][__popc(m & group & lt)] = k;  // the slot's hits, in order, wait for their place
    if (groups) {
      if (lane < NS) h_slot = __popc(m & (((1u << kG) - 1) << (lane * kG)));
    } else if (lane == x) {
      h_slot = __popc(m);
    }
    __syncwarp();
  }
  int all;
  const int before = warp_excl_scan(h_slot, lane, &all);
  unsigned long long rel = 0;
  if (all > 0) {
    if (lane == 0) rel = atomicAdd(W.cursor + part, (unsigned long long)all);
    rel = __shfl_sync(kFull, rel, 0);
    if ((int64_t)rel + all > cap) {  // the partition is full: the search runs again with larger ones
      if (lane < NS) W.hcnt[v0 + lane] = W.nvalid[v0 + lane] = 0;
      return;
    }
  }
  const int64_t base = part * cap + (int64_t)rel;
  if (lane < NS) {
    W.off[v0 + lane] = base + before;
    W.hcnt[v0 + lane] = h_slot;
  }
  for (unsigned m = __ballot_sync(kFull, h_slot > 0); m; m &= m - 1) {
    const int y = __ffs(m) - 1;
    const int ny = __shfl_sync(kFull, h_slot, y), by = __shfl_sync(kFull, before, y);
    if (lane < ny) {
      const uint64_t k = sm.word[y][lane];
      W.skey[base + by + lane] = word_key(k);
      W.sq[base + by + lane] = (uint32_t)word_q(k);
    }
  }
}

// The reads k_seed_reads leaves: their seeds go to memory.  Counts of every
// slot, then a range for the read, then the seeds, the entries of a chunk of
// l-mers shared by the lanes.  TEAM warps take a read, the rounds of it in
// equal runs: one for reads of one round, which keep their payloads in shared
// memory in between, a block of four (two for three or four windows) for longer ones, which are looked up
// again.  Teams take reads from a counter, as they finish.  The '-' strand's
// l-mers come from its end to its start, so its slots are filled from their
// end: all slots are in l-mer order.
template <bool SMALL, int NW, int TEAM>
struct LongSmem {
  ListSmem<SMALL, NW> list;
  uint64_t pl[TEAM == 1 ? ListSmem<SMALL, NW>::kList : 1];
};
template <int NW>
constexpr int kLongTeam = NW <= 2 ? 4 : 2;
template <bool SMALL, int NW, int TEAM>
__global__ void __launch_bounds__(TEAM == 1 ? kSeedFusedThreads : 32 * TEAM)
    k_seed_reads_long(QueryView q, SeedWins W, int gap, int local) {
  constexpr int NS = 2 * NW;
  constexpr int kWarps = TEAM == 1 ? kSeedFusedThreads / 32 : TEAM;
  __shared__ LongSmem<SMALL, NW, TEAM> smem[kWarps];
  __shared__ int team_n[TEAM][NS];    // entries per warp and slot
  __shared__ int team_valid[NS];      // valid seeds per slot
  __shared__ int team_kmers, team_li;
  __shared__ unsigned long long team_rel;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  LongSmem<SMALL, NW, TEAM>& sm = smem[warp];
  const int n_long = W.n_long[TEAM == 1 ? 0 : 1];
  int* const next = W.n_long + (TEAM == 1 ? 2 : 3);
  const int64_t n_reads = q.nstrands / 2;
  for (;;) {
    int li = 0;
    if (TEAM == 1) {
      if (lane == 0) li = atomicAdd(next, 1);
      li = __shfl_sync(kFull, li, 0);
    } else {
      __syncthreads();
      if (threadIdx.x == 0) {
        team_li = atomicAdd(next, 1);
        team_kmers = 0;
      }
      if (threadIdx.x < NS) team_valid[threadIdx.x] = 0;
      __syncthreads();
      li = team_li;
    }
    if (li >= n_long) break;
    const int64_t r = W.long_reads[TEAM == 1 ? (int64_t)li : n_reads - 1 - li];
    const int64_t st = q.start[2 * r];
    const int qlen = q.len[2 * r];
    const int nk = qlen - W.w[0].ix.l + 1;
    const int64_t v0 = r * NS;
    const int part = (int)(r % kSeedParts);
    const int64_t cap = W.part_cap * NW;
    const bool one_round = TEAM == 1;
    // this warp's rounds
    const int rounds = (nk + kSeedRound - 1) / kSeedRound;
    const int r_from = TEAM == 1 ? 0 : (int)((int64_t)rounds * warp / TEAM) * kSeedRound;
    const int r_to = TEAM == 1 ? nk : (int)((int64_t)rounds * (warp + 1) / TEAM) * kSeedRound;
    int n_all = 0;  // lane x < NS: entries of slot x
    int valid_kmers = 0, total = 0;
    for (int r0 = r_from; r0 < r_to; r0 += kSeedRound) {
      total = round_list<SMALL, NW>(q, W, st, nk, r0, lane, sm.list, valid_kmers);
#pragma unroll 1
      for (int c0 = 0; c0 < total; c0 += 64) {
        uint64_t pl[2];
        int tag[2];
        list_payloads(W, sm.list, c0, lane, total, pl, tag);
#pragma unroll
        for (int u = 0; u < 2; ++u)
          if (one_round && c0 + 32 * u + lane < total) sm.pl[c0 + 32 * u + lane] = pl[u];
        const int ca = payload_count(pl[0]), cb = payload_count(pl[1]);
#pragma unroll
        for (int x = 0; x < NS; ++x) {
          const int n = (int)__reduce_add_sync(kFull, (unsigned)(((tag[0] & 7) == x ? ca : 0) + ((tag[1] & 7) == x ? cb : 0)));
          if (lane == x) n_all += n;
        }
      }
      __syncwarp();
    }
    valid_kmers = (int)__reduce_add_sync(kFull, (unsigned)valid_kmers);
    int done = 0;  // lane x < NS: entries of slot x written, or before this warp's
    if (TEAM > 1) {
      if (lane < NS) team_n[warp][lane] = n_all;
      if (lane == 0) atomicAdd(&team_kmers, valid_kmers);
      __syncthreads();
      n_all = 0;
      if (lane < NS)
#pragma unroll
        for (int w = 0; w < TEAM; ++w) {
          if (w == warp) done = n_all;
          n_all += team_n[w][lane];
        }
      valid_kmers = team_kmers;
    }
    int64_t all = 0, before = 0;
#pragma unroll
    for (int x = 0; x < NS; ++x) {
      const int n = __shfl_sync(kFull, n_all, x);
      if (x < lane) before += n;
      all += n;
    }
    unsigned long long rel = 0;
    if (TEAM == 1 || warp == 0) {
      if (lane == 0 && all > 0) rel = atomicAdd(W.cursor + part, (unsigned long long)all);
      rel = __shfl_sync(kFull, rel, 0);
#pragma unroll
      for (int w = 0; w < NW; ++w) {
        const int n = __shfl_sync(kFull, n_all, 2 * w) + __shfl_sync(kFull, n_all, 2 * w + 1);
        if (lane == w) {
          if (valid_kmers) atomicAdd(W.w[w].n_kmers + part, 2ull * (unsigned long long)valid_kmers);
          if (n) atomicAdd(W.w[w].n_seeds + part, (unsigned long long)n);
        }
      }
    }
    if (TEAM > 1) {
      if (threadIdx.x == 0) team_rel = rel;
      __syncthreads();
      rel = team_rel;
    }
    if (all == 0 || (int64_t)rel + all > cap) {
      if ((TEAM == 1 || warp == 0) && lane < NS) W.nvalid[v0 + lane] = W.cnt[v0 + lane] = W.hcnt[v0 + lane] = 0;
      continue;
    }
    const int64_t base = part * cap + (int64_t)rel + before;  // lane x < NS: of slot x
    int valid[NS];  // this lane's valid seeds per slot
#pragma unroll
    for (int x = 0; x < NS; ++x) valid[x] = 0;
    for (int r0 = r_from; r0 < r_to; r0 += kSeedRound) {
      int dummy = 0;
      if (!one_round) total = round_list<SMALL, NW>(q, W, st, nk, r0, lane, sm.list, dummy);
#pragma unroll 1
      for (int c0 = 0; c0 < total; c0 += 64) {
        uint64_t pl2[2];
        int tag2[2];
        if (one_round) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const int j = c0 + 32 * u + lane;
            tag2[u] = j < total ? sm.list.tag[j] : 0;
            pl2[u] = j < total ? sm.pl[j] : kNoPayload;
          }
        } else {
          list_payloads(W, sm.list, c0, lane, total, pl2, tag2);
        }
#pragma unroll 1
        for (int u = 0; u < 2; ++u) {
          const uint64_t pl = u ? pl2[1] : pl2[0];
          const int tag = u ? tag2[1] : tag2[0];
          const int c = payload_count(pl);
          // this lane's first entry among its slot's, and among the chunk's
          int64_t at = 0;
          int first = 0, chunk = 0;
#pragma unroll
          for (int x = 0; x < NS; ++x) {
            int n;
            const int mine = warp_excl_scan((tag & 7) == x ? c : 0, lane, &n);
            const int d = __shfl_sync(kFull, done, x), size = __shfl_sync(kFull, n_all, x);
            const int64_t b = __shfl_sync(kFull, base, x);
            if ((tag & 7) == x) at = x & 1 ? b + size - (d + mine) - c : b + d + mine;
            if (lane == x) done += n;
            chunk += n;
          }
          int sum;
          first = warp_excl_scan(c, lane, &sum);
#pragma unroll 1
          for (int t0 = 0; t0 < chunk; t0 += 32) {
            const int t = t0 + lane, src = item_lane(first, t);
            const uint64_t p = __shfl_sync(kFull, pl, src);
            const int tg = __shfl_sync(kFull, tag, src), i = t - __shfl_sync(kFull, first, src);
            const int64_t to = __shfl_sync(kFull, at, src) + i;
            const int slot = tg & 7, qi = tag_qidx(tg, r0, nk);
            bool ok = false;
            if (t < chunk) {
              const uint64_t key = seed_key(W, slot, payload_entry(W, slot, p, i), qi, gap, local, qlen);
              __stcs(reinterpret_cast<unsigned long long*>(W.skey + to), key);
              __stcs(W.sq + to, (uint32_t)qi);
              ok = key != kDroppedSeed;
            }
#pragma unroll
            for (int x = 0; x < NS; ++x) valid[x] += ok && slot == x;
          }
        }
      }
      __syncwarp();
    }
    int n_slot = 0;
#pragma unroll
    for (int x = 0; x < NS; ++x) {
      const int n = (int)__reduce_add_sync(kFull, (unsigned)valid[x]);
      if (lane == x) n_slot = n;
    }
    if (TEAM > 1) {
      if (lane < NS && n_slot) atomicAdd(&team_valid[lane], n_slot);
      __syncthreads();
      if (warp == 0 && lane < NS) n_slot = team_valid[lane];
    }
    if ((TEAM == 1 || warp == 0) && lane < NS) {
      const int64_t v = v0 + lane;
      W.off[v] = base;
      W.cnt[v] = n_all;
      W.nvalid[v] = n_slot;
      if (n_slot > 0) {
        const int t = n_all <= kWarpSmemCap ? 0 : n_all <= kCtaSortCap ? 1 : 2;
        W.lists[t * (int64_t)NW * q.nstrands + atomicAdd(W.n_listed + t, 1)] = (uint32_t)v;
      } else {
        W.hcnt[v] = 0;
      }
    }
    __syncwarp();
  }
}

// The first strand of every (target window, query window) with a valid seed:
// its seed count is stored complemented, for the isolate filter keeps the first
// seed of a query window.  Where the seeding kernel filtered the slot itself
// (cnt 0), as one that is not first, that seed is a hit more, and the slot's
// first other hit is none if it lies near that seed (first_q's top bit).
__global__ void k_window_first(int32_t* __restrict__ nvalid, const int32_t* __restrict__ wstart, int nwin, int nw,
                               const int32_t* __restrict__ cnt, const uint32_t* __restrict__ first_q,
                               int32_t* __restrict__ hcnt, int64_t part_cap, GroupCtl* __restrict__ ctl) {
  if (blockIdx.x == 0 && threadIdx.x < kSeedParts && (int64_t)ctl->cursor[threadIdx.x] > part_cap) ctl->full = 1;
  const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= nwin * nw) return;
  const int w = i / nwin, qw = i % nwin;
  const int a = wstart[qw], b = wstart[qw + 1];
  for (int c = a; c < b; c += 32) {
    const int s = c + lane;
    const int64_t v = strand_slot(s, w, nw);
    const int n = s < b ? nvalid[v] : 0;
    const unsigned m = __ballot_sync(kFull, n > 0);
    if (m) {
      if (lane == __ffs(m) - 1) {
        nvalid[v] = ~n;
        if (first_q && cnt[v] == 0) hcnt[v] += 1 - (int)(first_q[v] >> 31);
      }
      return;
    }
  }
}

// ---- seed sort fused with the isolate / duplicate filters ----
// Slots (strand, target window) of a group; nvalid as k_window_first leaves it.
struct SeedFilterCtx {
  const int64_t* off;
  const int32_t* cnt;
  const int32_t* nvalid;
  int width, gap;
  int32_t* hcnt;
  const int* full;  // GroupCtl::full
};
__device__ __forceinline__ int valid_seeds(int nvalid) { return nvalid < 0 ? ~nvalid : nvalid; }

// State carried from one 32-seed chunk of a strand to the next.
struct FilterState {
  int ptid = 0, ptidx = 0, pdiag = 0;  // last seed of the previous chunk
  bool have_surv = false;
  int stid = 0, stidx = 0, sdiag = 0;  // last isolate-filter survivor so far
  int64_t out = 0;                     // next hit slot
};

// deletingIsolateSeeds then deleteDuplicateSeeds on the chunk of sorted seeds
// j = c0 + lane (valid when j < n); survivors are written at f.out onwards.
__device__ __forceinline__ void filter_chunk(int c0, int n, uint64_t k, uint32_t qi, bool wf, int width, int gap,
                                             FilterState& f, uint64_t* __restrict__ skey,
                                             uint32_t* __restrict__ sq) {
  const int lane = threadIdx.x & 31;
  const unsigned lt = lanemask_lt();
  const int j = c0 + lane;
  const bool in = j < n;
  const int tid = (int)(k >> 32);
  const int diag = (int)((uint32_t)k ^ 0x80000000u);
  const int tidx = diag + (int)qi;
  int ptid_l = __shfl_up_sync(kFull, tid, 1);
  int ptidx_l = __shfl_up_sync(kFull, tidx, 1);
  int pdiag_l = __shfl_up_sync(kFull, diag, 1);
  if (lane == 0) { ptid_l = f.ptid; ptidx_l = f.ptidx; pdiag_l = f.pdiag; }
  bool keep8 = false;
  if (in) keep8 = (j == 0) ? wf : near_pred(tid, tidx, diag, ptid_l, ptidx_l, pdiag_l, width, gap);
  const unsigned b8 = __ballot_sync(kFull, keep8);
  const unsigned below = b8 & lt;
  const int src = below ? 31 - __clz(below) : 0;
  const int qtid = __shfl_sync(kFull, tid, src);
  const int qtidx = __shfl_sync(kFull, tidx, src);
  const int qdiag = __shfl_sync(kFull, diag, src);
  bool keep9 = keep8;
  if (keep8) {
    if (below) keep9 = !near_pred(tid, tidx, diag, qtid, qtidx, qdiag, width, gap);
    else if (f.have_surv) keep9 = !near_pred(tid, tidx, diag, f.stid, f.stidx, f.sdiag, width, gap);
  }
  const unsigned b9 = __ballot_sync(kFull, keep9);
  if (keep9) {
    const int64_t w = f.out + __popc(b9 & lt);
    skey[w] = k;
    sq[w] = qi;
  }
  f.out += __popc(b9);
  f.ptid = __shfl_sync(kFull, tid, 31);
  f.ptidx = __shfl_sync(kFull, tidx, 31);
  f.pdiag = __shfl_sync(kFull, diag, 31);
  if (b8) {
    const int last = 31 - __clz(b8);
    f.stid = __shfl_sync(kFull, tid, last);
    f.stidx = __shfl_sync(kFull, tidx, last);
    f.sdiag = __shfl_sync(kFull, diag, last);
    f.have_surv = true;
  }
}

// Seed-sort tiers by a slot's seed count: <= kThreadSortCap (one thread,
// registers; most slots hold a few chance seeds), <= kWarpSmemCap (one warp:
// up to 32 in registers, more in its slice of shared memory), longer (one CTA:
// up to kCtaSortCap in shared memory, more in global memory).  The first tier
// runs over all slots and lists the others' slots; so four launches do what
// a classification and five tiers did, for every window of the group at once.
constexpr int kThreadSortCap = 8;

// 1..kThreadSortCap seeds: one thread per slot.  The seeds (padded with
// keys above every seed) go through an odd-even transposition network in
// registers unless they already ascend; the slot's valid seeds then
// come first (seeds the boundary filters dropped hold kDroppedSeed, above
// every valid key) and only they are filtered, in seed order, as
// filter_chunk applies the filters to a warp's chunk:
// a seed survives the isolate filter when it is near its predecessor (the
// strand's first seed only when the strand is its window's first), and the
// duplicate filter then drops it when it is near the previous seed that
// survived the isolate filter.
__global__ void k_seed_filter_small(uint64_t* __restrict__ skey, uint32_t* __restrict__ sq, SeedFilterCtx c, int64_t nv,
                                    uint32_t* __restrict__ lists, GroupCtl* __restrict__ ctl) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int x = s < nv ? c.nvalid[s] : 0;
  const int nvalid = *c.full ? 0 : valid_seeds(x);
  const int n = nvalid > 0 ? c.cnt[s] : 0;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int t = 0; t < 3; ++t) {
    const bool in = t == 0   ? n > kThreadSortCap && n <= kWarpSmemCap
                    : t == 1 ? n > kWarpSmemCap && n <= kCtaSortCap
                             : n > kCtaSortCap;
    const unsigned m = __ballot_sync(kFull, in);
    if (!m) continue;
    int base = 0;
    if (lane == __ffs(m) - 1) base = atomicAdd(&ctl->n_seeds[t], __popc(m));
    base = __shfl_sync(kFull, base, __ffs(m) - 1);
    if (in) lists[t * nv + base + __popc(m & lanemask_lt())] = (uint32_t)s;
  }
  if (s >= nv || n > kThreadSortCap) return;
  if (n == 0) {
    c.hcnt[s] = 0;
    return;
  }
  const int64_t o = c.off[s];
  const int nv_s = nvalid;
  uint64_t k[kThreadSortCap];
  uint32_t q[kThreadSortCap];
  bool sorted = true;
#pragma unroll
  for (int i = 0; i < kThreadSortCap; ++i) {
    k[i] = i < n ? skey[o + i] : ~0ull;
    q[i] = i < n ? sq[o + i] : ~0u;
    if (i > 0 && less2(k[i], q[i], k[i - 1], q[i - 1])) sorted = false;
  }
  if (!sorted) {
#pragma unroll
    for (int pass = 0; pass < kThreadSortCap; ++pass)
#pragma unroll
      for (int i = pass & 1; i + 1 < kThreadSortCap; i += 2)
        if (less2(k[i + 1], q[i + 1], k[i], q[i])) {
          const uint64_t tk = k[i]; k[i] = k[i + 1]; k[i + 1] = tk;
          const uint32_t tq = q[i]; q[i] = q[i + 1]; q[i + 1] = tq;
        }
  }
  const bool wf = x < 0;
  int ptid = 0, ptidx = 0, pdiag = 0;  // previous seed
  int stid = 0, stidx = 0, sdiag = 0;  // previous isolate-filter survivor
  bool have = false;
  int64_t out = o;
#pragma unroll
  for (int j = 0; j < kThreadSortCap; ++j) {
    if (j < nv_s) {
      const int tid = (int)(k[j] >> 32);
      const int diag = (int)((uint32_t)k[j] ^ 0x80000000u);
      const int tidx = diag + (int)q[j];
      const bool k8 = (j == 0) ? wf : near_pred(tid, tidx, diag, ptid, ptidx, pdiag, c.width, c.gap);
      const bool k9 = k8 && !(have && near_pred(tid, tidx, diag, stid, stidx, sdiag, c.width, c.gap));
      if (k9) {
        skey[out] = k[j];
        sq[out] = q[j];
        ++out;
      }
      if (k8) { stid = tid; stidx = tidx; sdiag = diag; have = true; }
      ptid = tid; ptidx = tidx; pdiag = diag;
    }
  }
  c.hcnt[s] = (int32_t)(out - o);
}

// Bitonic network over n <= np elements in shared memory, run by one warp.
__device__ __forceinline__ void warp_smem_network(uint64_t* s1, uint32_t* s2, int n) {
  const int lane = threadIdx.x & 31;
  int np = 64;
  while (np < n) np <<= 1;
  for (int size = 2; size <= np; size <<= 1) {
    for (int i = lane; i < np / 2; i += 32) {  // flip stage
      const int blk = i / (size / 2), r = i % (size / 2);
      const int a = blk * size + r, b = blk * size + size - 1 - r;
      if (b < n && less2(s1[b], s2[b], s1[a], s2[a])) {
        const uint64_t t1 = s1[a]; s1[a] = s1[b]; s1[b] = t1;
        const uint32_t t2 = s2[a]; s2[a] = s2[b]; s2[b] = t2;
      }
    }
    __syncwarp();
    for (int stride = size >> 2; stride > 0; stride >>= 1) {
      for (int i = lane; i < np / 2; i += 32) {
        const int blk = i / stride, r = i % stride;
        const int a = blk * 2 * stride + r, b = a + stride;
        if (b < n && less2(s1[b], s2[b], s1[a], s2[a])) {
          const uint64_t t1 = s1[a]; s1[a] = s1[b]; s1[b] = t1;
          const uint32_t t2 = s2[a]; s2[a] = s2[b]; s2[b] = t2;
        }
      }
      __syncwarp();
    }
  }
}

constexpr int kWarpSmemThreads = 128;

// kThreadSortCap + 1 .. kWarpSmemCap seeds: one warp per slot, sorting in
// registers up to 32 (a network sized to the count) and in its own slice of
// shared memory above; skipped when the seeds already ascend.
__global__ void __launch_bounds__(kWarpSmemThreads) k_seed_filter_mid(uint64_t* __restrict__ skey,
                                                                      uint32_t* __restrict__ sq, SeedFilterCtx c,
                                                                      const uint32_t* __restrict__ list,
                                                                      const int* __restrict__ count) {
  __shared__ uint64_t sh1[kWarpSmemThreads / 32][kWarpSmemCap];
  __shared__ uint32_t sh2[kWarpSmemThreads / 32][kWarpSmemCap];
  const int lane = threadIdx.x & 31;
  uint64_t* s1 = sh1[threadIdx.x >> 5];
  uint32_t* s2 = sh2[threadIdx.x >> 5];
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int total = *count;
  for (int64_t li = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; li < total; li += nwarps) {
    const int64_t s = list[li];
    if (*c.full) {
      if (lane == 0) c.hcnt[s] = 0;
      continue;
    }
    const int64_t o = c.off[s];
    const int n = c.cnt[s];
    const int x = c.nvalid[s];
    const int nv = valid_seeds(x);
    FilterState f;
    f.out = o;
    if (n <= 32) {
      uint64_t a1 = ~0ull;
      uint32_t a2 = ~0u;
      if (lane < n) {
        a1 = skey[o + lane];
        a2 = sq[o + lane];
      }
      const uint64_t n1 = __shfl_down_sync(kFull, a1, 1);
      const uint32_t n2 = __shfl_down_sync(kFull, a2, 1);
      if (__any_sync(kFull, lane + 1 < n && less2(n1, n2, a1, a2))) {
        if (n <= 16) lanes_sort<16>(a1, a2, lane);
        else lanes_sort<32>(a1, a2, lane);
      }
      filter_chunk(0, nv, a1, a2, x < 0, c.width, c.gap, f, skey, sq);
    } else {
      for (int i = lane; i < n; i += 32) {
        s1[i] = skey[o + i];
        s2[i] = sq[o + i];
      }
      __syncwarp();
      bool unsorted = false;
      for (int i = lane; i + 1 < n; i += 32) unsorted |= less2(s1[i + 1], s2[i + 1], s1[i], s2[i]);
      if (__any_sync(kFull, unsorted)) warp_smem_network(s1, s2, n);
      for (int c0 = 0; c0 < nv; c0 += 32) {
        const int j = c0 + lane;
        filter_chunk(c0, nv, j < nv ? s1[j] : 0ull, j < nv ? s2[j] : 0u, x < 0, c.width, c.gap, f, skey, sq);
      }
      __syncwarp();
    }
    if (lane == 0) c.hcnt[s] = (int32_t)(f.out - o);
  }
}

// Longer: one CTA per slot sorts and warp 0 filters from there.  Slots of up
// to kCtaSortCap seeds are sorted in shared memory by 256 threads (1,024
// threads, which the longer ones need, took 1.73 against 0.95 ms for the whole
// stage on a repeat-rich genome), more in global memory by 1,024.
template <bool SMEM>
__global__ void __launch_bounds__(SMEM ? 256 : 1024) k_seed_filter_big(uint64_t* __restrict__ skey,
                                                                       uint32_t* __restrict__ sq, SeedFilterCtx c,
                                                                       const uint32_t* __restrict__ list,
                                                                       const int* __restrict__ count) {
  __shared__ uint64_t s1[SMEM ? kCtaSortCap : 1];
  __shared__ uint32_t s2[SMEM ? kCtaSortCap : 1];
  const int total = *count;
  for (int li = blockIdx.x; li < total; li += gridDim.x) {
    const int64_t s = list[li];
    if (*c.full) {  // the same for the whole block
      if (threadIdx.x == 0) c.hcnt[s] = 0;
      continue;
    }
    const int64_t o = c.off[s];
    const int n = c.cnt[s];
    if (SMEM) {
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        s1[i] = skey[o + i];
        s2[i] = sq[o + i];
      }
      __syncthreads();
      cta_network(s1, s2, n);
    } else {
      cta_network(skey + o, sq + o, n);
      __syncthreads();
    }
    if (threadIdx.x < 32) {
      const int x = c.nvalid[s];
      const int nv = valid_seeds(x);
      FilterState f;
      f.out = o;
      for (int c0 = 0; c0 < nv; c0 += 32) {
        const int j = c0 + (int)threadIdx.x;
        uint64_t k = 0;
        uint32_t qv = 0;
        if (j < nv) {
          k = SMEM ? s1[j] : skey[o + j];
          qv = SMEM ? s2[j] : sq[o + j];
        }
        filter_chunk(c0, nv, k, qv, x < 0, c.width, c.gap, f, skey, sq);
      }
      if (threadIdx.x == 0) c.hcnt[s] = (int32_t)(f.out - o);
    }
    __syncthreads();
  }
}

__global__ void k_gather_hits(const uint64_t* __restrict__ skey, const uint32_t* __restrict__ sq,
                              const int64_t* __restrict__ off, const int32_t* __restrict__ hcnt,
                              const int64_t* __restrict__ hoff, int64_t nv, int nw, uint64_t* __restrict__ hk,
                              int32_t* __restrict__ hq, uint32_t* __restrict__ hs, const int32_t* __restrict__ qlen,
                              int l, int band, FirstSeeds first, GroupCtl* __restrict__ ctl) {
  const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int n = (v < nv) ? hcnt[v] : 0;
  // every hit of the strand fills band * (qlen - l) cells: backward rows + forward rows
  unsigned long long c =
      n ? (unsigned long long)n * (unsigned long long)band * (unsigned long long)(qlen[slot_strand((uint32_t)v, nw)] - l) : 0;
#pragma unroll
  for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(&ctl->cells, c);
  if (v >= nv) return;
  if (n == 0) return;
  int64_t a = off[v], b = hoff[v];
  int i = 0;
  if (first.key && first.nvalid[v] < 0 && first.cnt[v] == 0) {  // see k_window_first
    const uint32_t q0 = first.q[v];
    hk[b] = first.key[v];
    hq[b] = (int32_t)(q0 & 0x7fffffffu);
    hs[b] = (uint32_t)v;
    a += (int)(q0 >> 31) - 1;
    i = 1;
  }
  for (; i < n; ++i) {
    hk[b + i] = skey[a + i];
    hq[b + i] = (int32_t)sq[a + i];
    hs[b + i] = (uint32_t)v;
  }
}

// ------------------------------------------------------------------------
// banded DP
// ------------------------------------------------------------------------
// POINT_MATRIX / MATCH_COUNTER (krnlMatrix.cuh:11-67) depend only on seven
// letter classes: A, C, G, T, any other scored letter (B D H K M N R S U V W Y),
// a '-1' letter (E F I J L O P Q Z) and the bad-area letter X.  Bytes outside
// 'A'..'Z' score as 'N'.
constexpr int kClassX = 6;

__host__ __device__ constexpr int class_of_letter(int i) {  // i = letter - 'A'
  return i == 0 ? 0 : i == 2 ? 1 : i == 6 ? 2 : i == 19 ? 3 : i == 23 ? kClassX
       : (i == 4 || i == 5 || i == 8 || i == 9 || i == 11 || i == 14 || i == 15 || i == 16 || i == 25) ? 5 : 4;
}
// (point, match increment) for target class t, query class q.
__device__ __forceinline__ int2 cell_score(int t, int q) {
  if (t == kClassX || q == kClassX) return make_int2(-1000, -1000);
  if (t == 5 || q == 5) return make_int2(-1, -1);
  if (t == q && t < 4) return make_int2(1, 1);
  return make_int2(-3, 0);
}

// Scores of the band are kept as potentials: after row r (from 0) of a pass,
// column c holds S + 4 (r + 1) + 2 c (likewise for V and H).  A vertical step
// (r - 1, c + 1) -> (r, c) and a horizontal one (r, c - 1) -> (r, c) both raise
// 4 (r + 1) + 2 c by 2, which cancels the gap extension, so that extending a
// gap costs nothing and opening one costs 5 from either side:
//   V = max(s_up - 5, v_up)   H = max(s_left - 5, h_left)   diagonal: s_diag + POINT + 4
// (calcutlateCell, krnlAlignment.cu:42-77, with every difference unchanged, so
// every comparison and tie is too).  With P = max(diagonal, V), S = max(P, H)
// and S - 5 <= max(P - 5, H), the horizontal state is a running maximum along
// the row, H' = max(P - 5, H): one operation per cell on the row's dependent
// chain.  H wins iff H >= P (it wins ties over V, and both win them over the
// diagonal); otherwise V wins iff V >= diagonal.
constexpr int kStepRow = 4, kStepCol = 2;
constexpr int kOpenPot = kGapOpen + kGapExtend + kStepCol;  // -5
// The integer kernel takes kStepRow * kDpRebaseRows out of its potentials every
// kDpRebaseRows rows, and starts that much below zero, so that they stay below
// S + 200 whatever the number of rows: without it a matching read's potentials
// rise by 5 per row and pass 2^31 at row 429,496,729.  Half a dozen subtractions
// per 4,096 rows; short enough that reads of some kbp go through several.
constexpr int kDpRebaseRows = 4096;

// Shared memory of a DP block: the letter-pair table (POINT + 4, match
// increment) by class, and the classes' byte offsets into it by letter byte
// (target offset in the low byte, query offset in the high half).  The four
// bases of target and query take the table's first 16 entries, which are the
// 32 banks once: lanes that look up different base pairs never conflict.
template <class T2>
struct DpTab {
  T2 w[128];
  uint16_t q_off[256];
  uint8_t t_off[256];
};
__host__ __device__ constexpr int dp_t_class_off(int c) { return 32 * c; }                          // < 256
__host__ __device__ constexpr int dp_q_class_off(int c) { return c < 4 ? 8 * c : 256 * (c - 3); }

__device__ __forceinline__ int2 dp_pair_of(int2, int x, int y) { return make_int2(x, y); }
__device__ __forceinline__ float2 dp_pair_of(float2, int x, int y) { return make_float2((float)x, (float)y); }

template <class T2>
__device__ __forceinline__ void dp_table_init(DpTab<T2>& tab) {
  for (int i = threadIdx.x; i < 49; i += blockDim.x) {
    const int t = i / 7, q = i % 7;
    const int2 w = cell_score(t, q);
    tab.w[(dp_t_class_off(t) + dp_q_class_off(q)) / 8] = dp_pair_of(T2(), w.x + kStepRow, w.y);
  }
  for (int i = threadIdx.x; i < 256; i += blockDim.x) {
    const int c = class_of_letter(base_class((char)i));
    tab.t_off[i] = (uint8_t)dp_t_class_off(c);
    tab.q_off[i] = (uint16_t)dp_q_class_off(c);
  }
}
template <class T2>
__device__ __forceinline__ uint32_t dp_t_off(const DpTab<T2>& tab, char b) {
  return tab.t_off[(unsigned char)b];
}
template <class T2>
__device__ __forceinline__ uint32_t dp_q_off(const DpTab<T2>& tab, char b) {
  return tab.q_off[(unsigned char)b];
}
template <class T2>
__device__ __forceinline__ T2 dp_pair(const DpTab<T2>& tab, uint32_t off) {
  return *reinterpret_cast<const T2*>(reinterpret_cast<const char*>(tab.w) + off);
}

// initTempNodeArray, krnlAlignment.cu:6-38 (band rows 1..W): state of column c
// before row 0.  u is the vertical state the column hands to the row below.
template <int GAP>
__device__ __forceinline__ void dp_init_col(int c, int& s, int& u, int& m) {
  const int sc = c < GAP ? kMarginScore : c == GAP ? 0 : (c - GAP) * kGapExtend + kGapOpen;
  s = sc + kStepCol * c;
  u = c < GAP ? s : s + kOpenPot;  // max(S - 5, V): V is the margin itself left of the middle, S - 5 elsewhere
  m = c < GAP ? kMarginScore : 0;
}
// Left margin's H and the fixed band row's V (below the last column) of row 0;
// both rise by kStepRow per row.
template <int GAP>
constexpr int kDpLeftH = kMarginScore + kGapExtend + kStepRow;
template <int GAP>
constexpr int kDpBottomV =
    (GAP + 1) * kGapExtend + kGapOpen + kGapOpen + kGapExtend + kStepRow + kStepCol * 2 * GAP;

__device__ __forceinline__ float max3_f32(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Banded DP of one hit, backward pass then forward pass, in ONE row loop of
// rows_b + rows_f iterations: every hit of a read has qLen - l rows in total,
// so the threads of a warp stay converged although each switches from the
// backward to the forward pass at its own row.
//
// Bound by the ALU pipe (79 % busy on 2 kbp reads), where a warp instruction
// takes two cycles and where maxima, compares and selects run whatever their
// type.  So the whole numbers are held in floats (exact: see kDpMaxThreadRows):
// their additions run on the FMA pipe instead, at twice the rate, and a cell's
// ALU work is one three-way and two two-way maxima, two compares and two
// selects.  The columns' letters are packed four to a word, one dp4a makes a
// table address of them, and each pair is looked up well ahead of its use
// (without that, a lone hit waits 2.1 against 0.96 ms on 5 kbp).  Measured
// against the integer form with a spread table that this replaced: 1,172 to
// 2,045 GCUPS on uneven reads of 50 bp - 10 kbp (28.7 to 16.4 ms), 1,185 to
// 1,740 on a million reads of 150 bp (4.55 to 3.09 ms), 599 to 1,200 at gap 16.
// FMA: the second select is a saturated difference times the two values'
// difference (whole numbers, so exact), on the FMA pipe; faster only where
// four blocks share an SM (see kDpBlocksFull).  (Tried: packed f32x2
// additions, both selects so; slower.)
template <int GAP>
struct Band {
  static constexpr int W = 2 * GAP + 1;
  static constexpr int kWords = (W + 3) / 4;
  float2 sm[W];         // score potential, matches
  float u[W];           // the vertical state each column hands to the row below
  uint32_t tw[kWords];  // the columns' target letters: byte c = class offset in the table

  // The band before row 0, and the first W target bases of a pass: index ib0 +
  // step * c, 'X' outside [lo, hi).
  __device__ __forceinline__ void init(const DpTab<float2>& tab, const char* __restrict__ tb, int64_t tstart,
                                       int64_t ib0, int step, int64_t lo, int64_t hi) {
#pragma unroll
    for (int i = 0; i < kWords; ++i) tw[i] = 0;
#pragma unroll
    for (int c = 0; c < W; ++c) {
      int s, v, m;
      dp_init_col<GAP>(c, s, v, m);
      sm[c] = make_float2((float)s, (float)m);
      u[c] = (float)v;
      const int64_t ib = ib0 + (int64_t)step * c;
      tw[c / 4] |= dp_t_off(tab, (ib < lo || ib >= hi) ? 'X' : tb[tstart + ib]) << (8 * (c % 4));
    }
  }
  __device__ __forceinline__ void shift_in(uint32_t t) {
#pragma unroll
    for (int i = 0; i + 1 < kWords; ++i) tw[i] = __funnelshift_r(tw[i], tw[i + 1], 8);
    tw[kWords - 1] = (tw[kWords - 1] >> 8) | (t << (8 * ((W - 1) % 4)));
  }
  // select end node (global mode) after `rows` rows, krnlAlignment.cu:170-185
  __device__ __forceinline__ void end_node(int rows, int& best, int& best_m, int& ep) const {
    best = kMarginScore;
    best_m = kMarginScore;
    ep = -1;
#pragma unroll
    for (int c = 0; c < W; ++c) {
      const int sc = (int)sm[c].x - kStepRow * rows - kStepCol * c;
      if (best < sc) { best = sc; best_m = (int)sm[c].y; ep = c; }
    }
  }
};

template <int GAP, bool LOCAL, bool FMA>
__device__ __forceinline__ void banded_hit(const DpTab<float2>& tab, const char* __restrict__ tb, int64_t tstart,
                                           int tlen, const char* __restrict__ qb, int64_t qstart, int qlen, int tidx,
                                           int qidx, int l, int& t_hl, int& q_hl, int& match, int& score,
                                           int& o_tidx, int& o_qidx) {
  constexpr int W = Band<GAP>::W;
  constexpr int kNoLow = INT_MIN / 2, kNoHigh = INT_MAX / 2;
  constexpr float kOpen = (float)kOpenPot;
  const int rows_b = qlen - (qidx + l);  // alignmentSize of the backward pass
  const int rows_f = qidx;              // rows of the forward pass
  const int rows = rows_b + rows_f;
  Band<GAP> bd;
  // backward pass (globalAlignBackward / localAlignBackward): target bases
  // tIdx + l - gap + q + c ('X' at or past tLen), query bases qIdx + l + q.
  // tp, qp: letters of the row after the next; they hold while r < t_end, q_end.
  int64_t step = 1;
  const char* __restrict__ tp = tb + tstart + tidx + l + GAP + 1;
  const char* __restrict__ qp = qb + qstart + qidx + l;
  int t_end = tlen - (tidx + l + GAP + 1), q_end = rows_b;
  // The row's letter pairs come in K parts through two buffers: a part is
  // looked up before the cells of the part ahead of it run, the first one
  // during the row before.  (With one buffer of W pairs, each reloaded right
  // after its use, the compiler copies nearly every pair into another register
  // first.  At gap 2 the five pairs stay in place all the same: K = 1.)
  constexpr int K = GAP <= 2 ? 1 : GAP >= 10 && GAP <= 14 ? 4 : 2, CH = (W + K - 1) / K;
  float2 w[K == 1 ? 1 : 2][CH];
  uint32_t qo = 0;   // the row's query letter
  char t_n, q_n;     // letters of the next row
  auto pair = [&](int c) { return dp_pair(tab, __dp4a(bd.tw[c / 4], 1u << (8 * (c % 4)), qo)); };
  auto look_up = [&](int k) {
#pragma unroll
    for (int c = k * CH; c < W && c < (k + 1) * CH; ++c) w[k & 1][c - k * CH] = pair(c);
  };
  // r0: the pass's first row
  auto enter = [&](int r0) {
    const char q0 = r0 < q_end ? *qp : 'N';
    qp += step;
    qo = dp_q_off(tab, q0);
    look_up(0);
    t_n = r0 < t_end ? *tp : 'X';
    q_n = r0 + 1 < q_end ? *qp : 'N';
    tp += step;
    qp += step;
    --t_end;
    q_end -= 2;
  };
  bd.init(tab, tb, tstart, (int64_t)tidx + l - GAP, 1, kNoLow, tlen);
  enter(0);
  int bs = 0, bm = 0, calc = -1, ep = GAP;
  int pass = 0;
  float lift = kStepRow;  // potential of the row's column 0: kStepRow * (row of the pass + 1)
  auto finish = [&](int pass_rows) {  // result of the pass that just ended
    int move, best, best_m, e;
    if (LOCAL) { best = bs; best_m = bm; e = ep; move = calc + 1; }
    else { bd.end_node(pass_rows, best, best_m, e); move = pass_rows; }
    e -= GAP;
    if (pass_rows != 0) {
      if (pass == 1) {  // forward: the hit's start moves
        o_tidx -= move + e;
        o_qidx -= move;
      }
      t_hl += move + e;
      q_hl += move;
      match += best_m;
      score += best;
    }
  };
#pragma unroll 1
  for (int r = 0; r < rows; ++r) {
    if (r == rows_b) {  // switch to the forward pass (globalAlignForward / localAlignForward)
      finish(rows_b);
      pass = 1;
      step = -1;
      qp = qb + qstart + qidx - 1;           // query bases qIdx - q - 1
      tp = tb + tstart + tidx - GAP - 2;     // target bases tIdx + gap - 1 - q - c ('X' below 0)
      t_end = r + tidx - GAP - 1;
      q_end = rows;
      bd.init(tab, tb, tstart, (int64_t)tidx + GAP - 1, -1, 0, kNoHigh);
      enter(r);
      bs = 0; bm = 0; calc = -1; ep = GAP;
      lift = kStepRow;
    }
    // letters two rows ahead go out first
    const char t_nn = r < t_end ? *tp : 'X', q_nn = r < q_end ? *qp : 'N';
    tp += step;
    qp += step;
    float h = lift + (float)(kDpLeftH<GAP> - kStepRow), mh = kMarginScore;  // row 0 of the band (left margin)
    float top = -3e38f;                                                     // highest score of the row + lift (local)
    const float vbot = lift + (float)(kDpBottomV<GAP> - kStepRow);
    auto cell = [&](int c, float2 w) {
      const float v = (c + 1 < W) ? bd.u[(c + 1) % W] : vbot;
      const float vm = (c + 1 < W) ? bd.sm[(c + 1) % W].y : 0.0f;
      const float2 d = make_float2(bd.sm[c].x + w.x, bd.sm[c].y + w.y);
      const float S = max3_f32(d.x, v, h);
      const float open = S + kOpen;
      const float Q = FMA ? fmaf(__saturatef(S - v), d.y - vm, vm) : S == v ? vm : d.y;
      const float M = S == h ? mh : Q;
      bd.sm[c] = make_float2(S, M);
      bd.u[c] = fmaxf(open, v);
      h = fmaxf(open, h);
      mh = M;
      if (LOCAL) top = fmaxf(S - (float)(kStepCol * c), top);
    };
#pragma unroll
    for (int k = 0; k < K; ++k) {
      if (k + 1 < K) {
        look_up(k + 1);
      } else {
        bd.shift_in(dp_t_off(tab, t_n));  // 'X' is the bad-area letter itself
        qo = dp_q_off(tab, q_n);
        if (K > 1) look_up(0);
      }
#pragma unroll
      for (int c = k * CH; c < W && c < (k + 1) * CH; ++c) {
        cell(c, w[k & 1][c - k * CH]);
        if (K == 1) w[0][c] = pair(c);
      }
    }
    if (LOCAL && top - lift > (float)bs) {  // the first column with the row's highest score
      bs = (int)(top - lift);
      calc = (int)lift / kStepRow - 1;
#pragma unroll
      for (int c = W - 1; c >= 0; --c)
        if (bd.sm[c].x - (float)(kStepCol * c) == top) { bm = (int)bd.sm[c].y; ep = c; }
    }
    t_n = t_nn;
    q_n = q_nn;
    lift += (float)kStepRow;
  }
  if (rows_b == rows) {  // the loop never switched: close the backward pass (rows_f == 0)
    finish(rows_b);
  } else {
    finish(rows_f);
  }
}

// The same extension with one warp per hit, in 32-bit integers: the band's
// anti-diagonal wavefront.  Cell (r, c) of the band needs (r, c-1), (r-1, c+1) and (r-1, c),
// so the cells with equal 2r + c are independent.  Lane j owns band columns 2j
// and 2j + 1 and runs row r - j while lane 0 runs row r: column 2j at the even
// step, taking H and the match count left of it from lane j - 1 (shuffles) and
// the vertical state from its own odd column; column 2j + 1 at the odd step,
// with the vertical state and match count from lane j + 1 (shuffles).  A row's
// dependent chain is two shuffles and four maxima instead of W cells, which is
// what one long hit in a small batch waits for.  Same cell arithmetic as
// banded_hit, same tie rules (the local best is the first maximum in
// row-major order, the global end node the first maximum in column order),
// so every output equals banded_hit's.  Results are returned in every lane.
// A row takes some 210 cycles alone (275 before H became a running maximum and
// the letter pairs were looked up a row ahead): the two shuffles and the selects
// between them.
template <int GAP, bool LOCAL>
__device__ __forceinline__ void banded_hit_warp(const DpTab<int2>& tab, const char* __restrict__ tb,
                                                int64_t tstart, int tlen, const char* __restrict__ qb, int64_t qstart,
                                                int qlen, int tidx, int qidx, int l, int& t_hl, int& q_hl, int& match,
                                                int& score, int& o_tidx, int& o_qidx) {
  constexpr int W = 2 * GAP + 1;
  const int lane = threadIdx.x & 31;
  const int ce = 2 * lane, co = 2 * lane + 1;  // this lane's band columns
  const bool has_e = ce < W, has_o = co < W;
  const int left = (lane + 31) & 31, right = (lane + 1) & 31;
  const char* __restrict__ t_seq = tb + tstart;
  const char* __restrict__ q_seq = qb + qstart;
  const int rows_b = qlen - (qidx + l);
  const int rows_f = qidx;
  for (int pass = 0; pass < 2; ++pass) {
    const int rows_p = pass == 0 ? rows_b : rows_f;
    if (rows_p <= 0) continue;
    // target base of cell (r, c): ib0 + step * (r + c), the bad-area letter
    // outside [lo, hi); query base of row r: qi0 + step * r (banded_hit's
    // indices, pass by pass)
    const int step = pass == 0 ? 1 : -1;
    const int ib0 = pass == 0 ? tidx + l - GAP : tidx + GAP - 1;
    const int lo = pass == 0 ? INT_MIN : 0, hi = pass == 0 ? tlen : INT_MAX;
    const int qi0 = pass == 0 ? qidx + l : qidx - 1;
    auto t_byte = [&](int ib) -> char { return (ib < lo || ib >= hi) ? 'X' : t_seq[ib]; };
    auto q_byte = [&](int r) -> char { return (unsigned)r < (unsigned)rows_p ? q_seq[qi0 + step * r] : 'N'; };
    int se, ue, me, so, uo, mo;  // score, vertical state for the row below, matches of the two columns
    dp_init_col<GAP>(ce, se, ue, me);
    dp_init_col<GAP>(co, so, uo, mo);
    int ho = 0;
    int lift = kStepRow * (1 - lane);  // of the lane's row: kStepRow * (row + 1), less what rebase() took out
    auto rebase = [&]() {
      constexpr int d = kStepRow * kDpRebaseRows;
      se -= d;
      ue -= d;
      so -= d;
      uo -= d;
      ho -= d;
      lift -= d;
    };
    rebase();
    int bs = 0, bm = 0, calc = -1, ep = GAP;
    // Row r of this lane uses the target bases r + 2j (even column; the odd
    // column's base of row r - 1) and r + 2j + 1, and query base r.  Bytes are
    // loaded five rows ahead, turned into table offsets two rows ahead and
    // into pairs one row ahead, so that no load's latency falls inside a row.
    int r = -lane;
    const uint32_t t_a = dp_t_off(tab, t_byte(ib0 + step * (r + ce)));
    const uint32_t t_b = dp_t_off(tab, t_byte(ib0 + step * (r + co)));
    uint32_t t_c = dp_t_off(tab, t_byte(ib0 + step * (r + 1 + co)));  // odd column of row r + 1
    const uint32_t q_a = dp_q_off(tab, q_byte(r));
    uint32_t q_c = dp_q_off(tab, q_byte(r + 1));
    int2 we = dp_pair(tab, t_a + q_a), wo = dp_pair(tab, t_b + q_a);
    uint32_t t_even = t_b;  // even column of row r + 1
    char t2 = t_byte(ib0 + step * (r + 2 + co)), t3 = t_byte(ib0 + step * (r + 3 + co));
    char t4 = t_byte(ib0 + step * (r + 4 + co));
    char q2 = q_byte(r + 2), q3 = q_byte(r + 3), q4 = q_byte(r + 4);
    int tk = ib0 + step * (r + 5 + co);
    // One row.  EDGE: some lanes may be outside the pass's rows and keep their state.
    auto row = [&](auto edge) {
      constexpr bool EDGE = decltype(edge)::value;
      const int hl = __shfl_sync(kFull, ho, left), ml = __shfl_sync(kFull, mo, left);
      const char t5 = t_byte(tk);
      const char q5 = q_byte(r + 5);
      tk += step;
      const int2 we_n = dp_pair(tab, t_even + q_c), wo_n = dp_pair(tab, t_c + q_c);
      const bool on = !EDGE || (unsigned)r < (unsigned)rows_p;
      // even step: column 2j; H from lane j - 1, the vertical state from our
      // odd column (below the last column: the fixed band row)
      const int ve = has_o ? uo : kDpBottomV<GAP> - kStepRow + lift;
      const int Pe = __viaddmax_s32(se, we.x, ve);
      const int Qe = Pe == ve ? (has_o ? mo : 0) : me + we.y;
      const int h = lane == 0 ? kDpLeftH<GAP> - kStepRow + lift : hl;
      const int mh = lane == 0 ? kMarginScore : ml;
      const int Se = max(Pe, h);
      const int Me = Se == h ? mh : Qe;
      const int Ue = __viaddmax_s32(Se, kOpenPot, ve);
      const int he = __viaddmax_s32(Pe, kOpenPot, h);
      if (on) {
        se = Se;
        ue = Ue;
        me = Me;
      }
      // odd step: column 2j + 1; the vertical state from lane j + 1
      const int vo = __shfl_sync(kFull, ue, right), vm = __shfl_sync(kFull, me, right);
      const int Po = __viaddmax_s32(so, wo.x, vo);
      const int Qo = Po == vo ? vm : mo + wo.y;
      const int So = max(Po, he);
      const int Mo = So == he ? Me : Qo;
      if (on) {
        so = So;
        uo = __viaddmax_s32(So, kOpenPot, vo);
        mo = Mo;
        ho = __viaddmax_s32(Po, kOpenPot, he);
        if (LOCAL) {
          const int xe = Se - lift - kStepCol * ce, xo = So - lift - kStepCol * co;
          if (has_e && xe > bs) { bs = xe; bm = Me; calc = r; ep = ce; }
          if (has_o && xo > bs) { bs = xo; bm = Mo; calc = r; ep = co; }
        }
      }
      we = we_n;
      wo = wo_n;
      t_even = t_c;
      t_c = dp_t_off(tab, t2);
      q_c = dp_q_off(tab, q2);
      t2 = t3;
      t3 = t4;
      t4 = t5;
      q2 = q3;
      q3 = q4;
      q4 = q5;
      lift += kStepRow;
      ++r;
    };
    // lane GAP starts GAP rows after lane 0 and ends GAP rows after it
    const int n_ramp = min(GAP, rows_p);
    for (int it = 0; it < n_ramp; ++it) row(std::true_type());
    for (int it = n_ramp; it < rows_p;) {
      const int stop = rows_p - it > kDpRebaseRows ? it + kDpRebaseRows : rows_p;
#pragma unroll 2
      for (; it < stop; ++it) row(std::false_type());
      rebase();  // every lane at once, whatever row it is in: the lanes' states stay comparable
    }
    for (int it = 0; it < GAP; ++it) row(std::true_type());
    int best, best_m, e, move;
    if (LOCAL) {  // first maximum in row-major order: (score desc, row asc, column asc)
#pragma unroll
      for (int off = 16; off; off >>= 1) {
        const int xs = __shfl_xor_sync(kFull, bs, off), xm = __shfl_xor_sync(kFull, bm, off);
        const int xc = __shfl_xor_sync(kFull, calc, off), xe = __shfl_xor_sync(kFull, ep, off);
        if (xs > bs || (xs == bs && (xc < calc || (xc == calc && xe < ep)))) { bs = xs; bm = xm; calc = xc; ep = xe; }
      }
      best = bs;
      best_m = bm;
      e = ep;
      move = calc + 1;
    } else {  // end node: the first column of the last row with the highest score above the margin
      int sc = INT_MIN, c = W, m = 0;
      const int top = lift - kStepRow * (GAP - lane + 1);  // the last row's lift: lane j ended GAP - j rows ago
      if (has_e) { sc = se - top - kStepCol * ce; c = ce; m = me; }
      const int sco = so - top - kStepCol * co;
      if (has_o && sco > sc) { sc = sco; c = co; m = mo; }
#pragma unroll
      for (int off = 16; off; off >>= 1) {
        const int xs = __shfl_xor_sync(kFull, sc, off), xc = __shfl_xor_sync(kFull, c, off);
        const int xm = __shfl_xor_sync(kFull, m, off);
        if (xs > sc || (xs == sc && xc < c)) { sc = xs; c = xc; m = xm; }
      }
      if (sc > kMarginScore) { best = sc; best_m = m; e = c; }
      else { best = kMarginScore; best_m = kMarginScore; e = -1; }
      move = rows_p;
    }
    e -= GAP;
    if (pass == 1) {
      o_tidx -= move + e;
      o_qidx -= move;
    }
    t_hl += move + e;
    q_hl += move;
    match += best_m;
    score += best;
  }
}

struct DpKernelArgs {
  TargetView t[kMaxSeedWins];
  int nw;
  QueryView q;
  const uint64_t* hk;
  const int32_t* hq;
  const uint32_t* hs;
  const uint64_t* order;
  int64_t n;
  DpParams p;
  DpOut o;
  // the first n_warp hits of the order run one per warp (k_banded_dp_warp),
  // the others one per thread: n_warp = *warp_n when given, else warp_fixed
  const long long* warp_n;
  long long warp_fixed;
  int* bad;  // see DpLaunch::bad
};

// A hit whose target sequence or strand lies outside the window cannot come
// from the seeding stages; it is flagged and given empty outputs instead of
// being read past the window.
__device__ __forceinline__ bool dp_hit_outside(const DpKernelArgs& a, const TargetView& t, int tid, int64_t s) {
  return (unsigned)tid >= (unsigned)t.nseqs || s >= (int64_t)a.q.nstrands;
}

__device__ __forceinline__ int64_t dp_warp_hits(const DpKernelArgs& a) {
  const int64_t w = a.warp_n ? (int64_t)*a.warp_n : (int64_t)a.warp_fixed;
  return w < a.n ? w : a.n;
}

// calculateEvalue (krnlCalculateEvalue.cu:21, same operation order) and the
// two hit filters of deleteBadHits, then the hit's outputs at its own index.
__device__ __forceinline__ void dp_store(const DpKernelArgs& a, int64_t h, int qlen, int o_tidx, int o_qidx, int t_hl,
                                         int q_hl, int match, int score) {
  const double e = a.p.K * a.p.total_db * (double)qlen * exp(-a.p.lambda * (double)score);
  const bool keep = !(a.p.cutoff != -1.0 && a.p.cutoff < e) && !(a.p.l + a.p.stride > q_hl);
  a.o.t_idx[h] = o_tidx;
  a.o.q_idx[h] = o_qidx;
  a.o.t_len[h] = t_hl;
  a.o.q_len[h] = q_hl;
  a.o.match[h] = match;
  a.o.score[h] = score;
  a.o.evalue[h] = e;
  a.o.keep[h] = keep ? 1 : 0;
}

__device__ __forceinline__ void dp_skip(const DpKernelArgs& a, int64_t h) {
  a.o.t_idx[h] = a.o.q_idx[h] = a.o.t_len[h] = a.o.q_len[h] = a.o.match[h] = a.o.score[h] = 0;
  a.o.evalue[h] = 0.0;
  a.o.keep[h] = 0;
  if (a.bad) atomicExch(a.bad, 1);
}

// Extension of the hit at position i of the order (alignmentHits +
// calculateEvalue + the two hit filters of deleteBadHits).
template <int GAP, bool LOCAL, bool FMA>
__device__ __forceinline__ void dp_one(const DpKernelArgs& a, const DpTab<float2>& tab, int64_t i) {
  const int64_t h = a.order ? (int64_t)(uint32_t)a.order[i] : i;
  const uint64_t k = a.hk[h];
  const int qidx = a.hq[h];
  const int64_t s = slot_strand(a.hs[h], a.nw);
  const TargetView& t = a.t[slot_window(a.hs[h], a.nw)];
  const int tid = (int)(k >> 32);
  if (dp_hit_outside(a, t, tid, s)) {
    dp_skip(a, h);
    return;
  }
  const int tidx = (int)((uint32_t)k ^ 0x80000000u) + qidx;
  const int64_t tstart = t.gateway[tid];
  const int tlen = t.lengths[tid];
  const int64_t qstart = a.q.start[s];
  const int qlen = a.q.len[s];
  const int l = a.p.l;
  int t_hl = l, q_hl = l, match = l, score = l;  // CDeviceHitList.cu:283-286
  int o_tidx = tidx, o_qidx = qidx;
  banded_hit<GAP, LOCAL, FMA>(tab, t.bases, tstart, tlen, a.q.bases, qstart, qlen, tidx, qidx, l, t_hl, q_hl, match,
                         score, o_tidx, o_qidx);
  dp_store(a, h, qlen, o_tidx, o_qidx, t_hl, q_hl, match, score);
}

// A block extends kDpThreads * rounds consecutive hits of the order.  With
// `by_rows` (hits of equal length, in no order of their own) it first sorts
// them by the rows of the forward pass, so that the lanes of a warp leave the
// backward pass at the same row: the switch (end node, new band, its letters)
// is some 350 instructions that every lane leaving at a row of its own would
// run alone (3.63 to 3.44 ms on a million reads of 150 bp).
constexpr int kDpThreads = 128, kDpMaxRounds = 4;
// Blocks per SM by the registers the band takes (natural: 90 at gap 2, 145 at
// gap 8, 227 at gap 16).  Where the reads are long and uneven, three blocks of
// up to 168 registers are the better ones at gap 8: 2.69 ms against 2.93 for
// four of 128 on 10,000 reads of 100 - 5,000 bp, the same on 30,000.  At gaps
// 10 - 14 three blocks (with the letter pairs in four parts) take 9.4 ms
// against 10.4 for the two that the whole row's pairs left room for.
// kDpBlocksFull: hits of equal length, more of them than those blocks hold, run
// four to an SM at gaps 5 - 8 (a million reads of 150 bp at gap 8: 3.25 to 3.09
// ms; 60,000 local ones: 1.05 to 0.89).
template <int GAP>
constexpr int kDpBlocksPerSm = GAP <= 4 ? 4 : GAP <= 14 ? 3 : 2;
template <int GAP>
constexpr int kDpBlocksFull = GAP >= 5 && GAP <= 8 ? 4 : kDpBlocksPerSm<GAP>;

template <int GAP, bool LOCAL, int BLOCKS>
__global__ void __launch_bounds__(kDpThreads, BLOCKS)
    k_banded_dp(DpKernelArgs a, int rounds, int by_rows) {
  __shared__ DpTab<float2> tab;
  __shared__ uint32_t key[kDpThreads * kDpMaxRounds];  // forward rows << 16 | hit within the block
  dp_table_init(tab);
  const int64_t base = dp_warp_hits(a) + (int64_t)blockIdx.x * (kDpThreads * rounds);
  const int n = kDpThreads * rounds;  // a power of two
  if (by_rows) {
    for (int i = threadIdx.x; i < n; i += kDpThreads)
      key[i] = base + i < a.n ? ((uint32_t)min(a.hq[base + i], 0xfffe) << 16) | (uint32_t)i : ~0u;
    for (int size = 2; size <= n; size <<= 1)
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        __syncthreads();
        for (int i = threadIdx.x; i < n / 2; i += kDpThreads) {
          const int lo = 2 * i - (i & (stride - 1)), hi = lo + stride;
          const uint32_t x = key[lo], y = key[hi];
          if ((x > y) == ((lo & size) == 0)) {
            key[lo] = y;
            key[hi] = x;
          }
        }
      }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += kDpThreads) {
    const int64_t at = base + (by_rows ? (int64_t)(key[i] & 0xffffu) : (int64_t)i);
    if (at < a.n && !(by_rows && key[i] == ~0u)) dp_one<GAP, LOCAL, !LOCAL && (BLOCKS > kDpBlocksPerSm<GAP>)>(a, tab, at);
  }
}

// One hit per warp (banded_hit_warp) for the first n_warp hits of the order,
// the longest ones: a grid-stride loop over them, one warp each.
template <int GAP, bool LOCAL>
__global__ void __launch_bounds__(128) k_banded_dp_warp(DpKernelArgs a) {
  __shared__ DpTab<int2> tab;
  dp_table_init(tab);
  __syncthreads();
  const int64_t nw = dp_warp_hits(a);
  const int lane = threadIdx.x & 31;
  const int64_t wpb = blockDim.x >> 5;
  for (int64_t i = (int64_t)blockIdx.x * wpb + (threadIdx.x >> 5); i < nw; i += (int64_t)gridDim.x * wpb) {
    const int64_t h = a.order ? (int64_t)(uint32_t)a.order[i] : i;
    const uint64_t k = a.hk[h];
    const int qidx = a.hq[h];
    const int64_t s = slot_strand(a.hs[h], a.nw);
    const TargetView& t = a.t[slot_window(a.hs[h], a.nw)];
    const int tid = (int)(k >> 32);
    if (dp_hit_outside(a, t, tid, s)) {  // the same for every lane of the warp
      if (lane == 0) dp_skip(a, h);
      continue;
    }
    const int tidx = (int)((uint32_t)k ^ 0x80000000u) + qidx;
    const int64_t tstart = t.gateway[tid];
    const int tlen = t.lengths[tid];
    const int64_t qstart = a.q.start[s];
    const int qlen = a.q.len[s];
    const int l = a.p.l;
    int t_hl = l, q_hl = l, match = l, score = l;  // CDeviceHitList.cu:283-286
    int o_tidx = tidx, o_qidx = qidx;
    banded_hit_warp<GAP, LOCAL>(tab, t.bases, tstart, tlen, a.q.bases, qstart, qlen, tidx, qidx, l, t_hl, q_hl,
                                match, score, o_tidx, o_qidx);
    if (lane == 0) dp_store(a, h, qlen, o_tidx, o_qidx, t_hl, q_hl, match, score);
  }
}

// Length buckets of the hits for the warp / thread split: 16 buckets per power of two of
// the row count (rows within a bucket differ by at most 1/16), numbered so
// that ascending bucket = longest first.
constexpr int kDpBuckets = 16 * 33;
__device__ __forceinline__ int dp_bucket(int rows) {
  if (rows < 16) return kDpBuckets - 1 - rows;  // exact below 16
  const int e = 31 - __clz(rows);                // rows in [2^e, 2^(e+1))
  const int sub = (rows >> (e - 4)) & 15;
  return kDpBuckets - 1 - (16 * (e - 3) + sub);
}

__global__ void k_dp_bucket_count(const uint32_t* __restrict__ hs, int nw, const int32_t* __restrict__ q_len, int64_t n,
                                  int l,
                                  unsigned int* __restrict__ count, unsigned long long* __restrict__ rows) {
  __shared__ unsigned int c[kDpBuckets];
  __shared__ unsigned long long sr[kDpBuckets];
  for (int i = threadIdx.x; i < kDpBuckets; i += blockDim.x) {
    c[i] = 0;
    sr[i] = 0;
  }
  __syncthreads();
  for (int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; h < n; h += (int64_t)gridDim.x * blockDim.x) {
    const int r = max(0, q_len[slot_strand(hs[h], nw)] - l);
    const int b = dp_bucket(r);
    atomicAdd(&c[b], 1u);
    atomicAdd(&sr[b], (unsigned long long)r);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kDpBuckets; i += blockDim.x)
    if (c[i]) {
      atomicAdd(&count[i], c[i]);
      atomicAdd(&rows[i], sr[i]);
    }
}

// Rows of bucket b (ascending b = longest first): [dp_bucket_lo(b), dp_bucket_hi(b)].
__host__ __device__ __forceinline__ long long dp_bucket_lo(int b) {
  const int x = kDpBuckets - 1 - b;
  if (x < 16) return x;
  const int e = x / 16 + 3, sub = x % 16;
  return (long long)(16 + sub) << (e - 4);
}
__host__ __device__ __forceinline__ long long dp_bucket_hi(int b) {
  const int x = kDpBuckets - 1 - b;
  if (x < 16) return x;
  return dp_bucket_lo(b) + (1ll << (x / 16 - 1)) - 1;
}

// Cost model of the warp / thread split, in SM clock cycles, fitted on the B200
// at gaps 2 - 16 in both modes to batches of 1 to 13,000 hits of 150 bp - 5 kbp,
// equal and uneven, every hit one way or the other.
// Thread mode: a row takes dp_thread_row_cycles where the hit's warp has the SM
// sub-partition to itself (a row is W dependent cells; below some twenty of them
// it waits for the letters of the warp's other hits, and a local one also keeps
// its best cell), the ends and bands of its two passes dp_thread_band_cycles; a
// full grid runs kDpThreadCellsPerCycle cells per cycle.  Warp mode: a row takes
// kDpWarpRowCycles alone (two wavefront steps); the GPU runs
// dp_warp_rows_per_cycle rows per cycle and a hit kDpWarpHitCycles of its own.
// Two kernels run side by side: with L the longer of the two longest hits' times
// and I the issue time of both kernels' work, the batch takes max(L + I/2, I)
// (measured: a lone hit's rows slow down as other warps share its sub-partition,
// and the GPU cannot issue faster than I), and the second stream kDpForkCycles.
// Only the split depends on these; results do not.  With 26 cycles per cell and 6
// rows per cycle everywhere (as fitted at gap 8, global mode), local batches and
// narrow bands stayed in thread mode too long: 4,000 local reads of 100 - 5,000 bp
// 1.93 to 0.73 ms at gap 3, 1.16 to 0.75 at gap 8; 3,000 of 150 bp at gap 16 0.118
// to 0.077.
constexpr double kDpThreadCellsPerCycle = 1000.0;
constexpr double kDpWarpRowCycles = 217.0;
constexpr double kDpWarpHitCycles = 8.4;
constexpr double kDpForkCycles = 10000.0;
constexpr long long kDpWarpMinRows = 16;
__host__ __device__ __forceinline__ double dp_thread_row_cycles(int W, bool local) {
  return !local ? fmax(480.0, 27.0 * W) : W <= 5 ? 510.0 : 500.0 + 26.0 * W;
}
__host__ __device__ __forceinline__ double dp_thread_band_cycles(int W, bool local) {
  return (local ? 25.0 : 50.0) * W * W;
}
__host__ __device__ __forceinline__ double dp_warp_rows_per_cycle(bool local) { return local ? 4.6 : 5.9; }

// Estimated time of the DP with the `s` longest hits (rows summed: sw, the
// longest r1) one per warp and the rest (rows summed: rest, the longest rn)
// one per thread.
__host__ __device__ __forceinline__ double dp_split_cycles(int W, bool local, long long s, double r1, double sw,
                                                           double rn, double rest) {
  double lat = s > 0 ? r1 * kDpWarpRowCycles : 0.0;
  if (rest > 0) lat = fmax(lat, rn * dp_thread_row_cycles(W, local) + dp_thread_band_cycles(W, local));
  const double issue = sw / dp_warp_rows_per_cycle(local) + (double)s * kDpWarpHitCycles +
                       rest * W / kDpThreadCellsPerCycle;
  return fmax(lat + 0.5 * issue, issue) + (s > 0 && rest > 0 ? kDpForkCycles : 0.0);
}

// The split on the device: the hits of kDpMaxThreadRows rows or more one per
// warp; then, with `split`, every bucket boundary (longest first) is a candidate,
// and the earliest estimated end wins.  One thread; ~500 buckets.
__global__ void k_dp_warp_split(const unsigned int* __restrict__ count, const unsigned long long* __restrict__ rows,
                                int W, bool local, long long cap, bool split, long long* __restrict__ warp_n) {
  if (threadIdx.x != 0) return;
  double total = 0;
  for (int b = 0; b < kDpBuckets; ++b) total += (double)rows[b];
  long long s = 0, best_s = 0;
  double sw = 0, r1 = -1, best = 0;
  bool all_taken = true, any = false;  // any: `best` holds a candidate's time
  for (int b = 0; b < kDpBuckets; ++b) {
    if (!count[b]) continue;
    const double rn = (double)dp_bucket_hi(b);
    if (r1 < 0) r1 = rn;
    if (dp_bucket_lo(b) < kDpMaxThreadRows) {
      // candidate: the buckets before b one per warp, b and the rest one per thread
      const double t = dp_split_cycles(W, local, s, s > 0 ? r1 : 0, sw, rn, total - sw);
      if (!any || t < best) { best = t; best_s = s; }
      any = true;
      if (!split || dp_bucket_lo(b) < kDpWarpMinRows || s + count[b] > cap) {
        all_taken = false;
        break;
      }
    }
    s += count[b];
    sw += (double)rows[b];
  }
  if (all_taken && s > 0 && (!any || dp_split_cycles(W, local, s, r1, sw, 0, 0) < best)) best_s = s;  // every hit one per warp
  *warp_n = best_s;
}

template <int GAP, bool LOCAL>
long long launch_dp_mode(DpKernelArgs a, const DpLaunch& m, cudaStream_t st) {
  constexpr int W = 2 * GAP + 1;
  const int threads = kDpThreads;
  struct Occupancy {
    int sms = 0, per_sm = 1, warp_per_sm = 1;
  };
  static const Occupancy occ = [] {  // once per kernel pair (thread-safe static initialisation)
    Occupancy o;
    int dev = 0;
    CLAST_CK(cudaGetDevice(&dev));
    CLAST_CK(cudaDeviceGetAttribute(&o.sms, cudaDevAttrMultiProcessorCount, dev));
    CLAST_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o.per_sm, k_banded_dp<GAP, LOCAL, kDpBlocksPerSm<GAP>>, kDpThreads, 0));
    CLAST_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o.warp_per_sm, k_banded_dp_warp<GAP, LOCAL>, kDpThreads, 0));
    o.per_sm = std::max(1, o.per_sm);
    o.warp_per_sm = std::max(1, o.warp_per_sm);
    return o;
  }();
  const int sms = occ.sms, per_sm = occ.per_sm, warp_per_sm = occ.warp_per_sm;
  // hits one per warp: at most one wave of the warp kernel's resident warps (the
  // cost model has no waves); half as many more where all are equal and the issue
  // rate bounds them (3,245 local hits of 150 bp at gap 16, 285 more than a wave:
  // 0.077 against 0.118 ms one per thread; 6,509: 0.145 against 0.118)
  const long long cap = (long long)sms * warp_per_sm * (threads / 32);
  a.warp_n = nullptr;
  a.warp_fixed = 0;
  if (m.warp == kDpWarpAll || m.uniform_rows >= kDpMaxThreadRows) {
    a.warp_fixed = a.n;
  } else if (m.buckets.count && m.warp_n && (m.warp == kDpWarpAuto || m.long_hits)) {
    k_dp_warp_split<<<1, 32, 0, st>>>(m.buckets.count, m.buckets.rows, W, LOCAL, cap, m.warp == kDpWarpAuto,
                                      m.warp_n);
    CLAST_LAUNCHED();
    a.warp_n = m.warp_n;
  } else if (m.warp == kDpWarpAuto && m.uniform_rows >= kDpWarpMinRows && 2 * a.n <= 3 * cap) {
    const double r = (double)m.uniform_rows, rows = r * (double)a.n;
    if (dp_split_cycles(W, LOCAL, a.n, r, rows, 0, 0) < dp_split_cycles(W, LOCAL, 0, 0, 0, r, rows)) a.warp_fixed = a.n;
  }
  const int64_t rest = a.n - (a.warp_n ? 0 : a.warp_fixed);  // hits left for the one-per-thread kernels (at most)
  bool joined = false;
  if (a.warp_n || a.warp_fixed > 0) {
    const long long most = a.warp_n ? std::min<long long>(cap, a.n) : a.warp_fixed;
    const long long blocks = std::min<long long>((most + 3) / 4, (long long)sms * warp_per_sm);
    cudaStream_t sw = st;
    if (m.aux && m.ev_fork && m.ev_join && rest > 0) {  // beside the one-per-thread kernel
      CLAST_CK(cudaEventRecord(m.ev_fork, st));
      CLAST_CK(cudaStreamWaitEvent(m.aux, m.ev_fork, 0));
      sw = m.aux;
    }
    k_banded_dp_warp<GAP, LOCAL><<<(unsigned)std::max<long long>(1, blocks), threads, 0, sw>>>(a);
    CLAST_LAUNCHED();
    if (sw != st) {
      CLAST_CK(cudaEventRecord(m.ev_join, sw));
      joined = true;
    }
  }
  const long long warp_hits = a.warp_n ? -1 : a.warp_fixed;
  if (rest <= 0) return warp_hits;
  // blocks of several rounds sort more hits together; short batches need the blocks
  const bool by_rows = m.uniform_rows >= 0;
  // the variant of more blocks only where they all have hits to run
  const bool full = kDpBlocksFull<GAP> > kDpBlocksPerSm<GAP> && by_rows && rest > (int64_t)sms * per_sm * threads;
  const int64_t waves = rest / ((int64_t)sms * (full ? kDpBlocksFull<GAP> : per_sm) * threads);
  const int rounds = !by_rows ? 1 : waves >= 8 ? kDpMaxRounds : waves >= 4 ? 2 : 1;
  const unsigned grid = (unsigned)((rest + threads * rounds - 1) / (threads * rounds));
  if (full)
    k_banded_dp<GAP, LOCAL, kDpBlocksFull<GAP>><<<grid, threads, 0, st>>>(a, rounds, by_rows);
  else
    k_banded_dp<GAP, LOCAL, kDpBlocksPerSm<GAP>><<<grid, threads, 0, st>>>(a, rounds, by_rows);
  CLAST_LAUNCHED();
  if (joined) CLAST_CK(cudaStreamWaitEvent(st, m.ev_join, 0));
  return warp_hits;
}

template <int GAP>
long long launch_dp_gap(const DpKernelArgs& a, bool local, const DpLaunch& m, cudaStream_t st) {
  return local ? launch_dp_mode<GAP, true>(a, m, st) : launch_dp_mode<GAP, false>(a, m, st);
}

// ------------------------------------------------------------------------
// final per-read order
// ------------------------------------------------------------------------
// A read's hits lie together, window after window.  Their order, (score desc,
// window, seed qIdx desc, strand, target sequence, seed tIdx), is the one the
// stable sorts of alignmentHits (by rows desc, then qIdx desc) and
// resultSorting (qID/2 asc, score desc) leave a window's hits of one read in,
// merged over the windows as fixResult's stable sort does.  The hits were
// gathered by (window, strand, sequence, diagonal, qIdx), so the position in
// the read's run decides what (score, window, qIdx) leave open.  Filtered hits
// sort after every kept one.
struct FinalCtx {
  const uint64_t* hk;
  const int32_t* hq;
  const uint32_t* hs;
  DpOut o;
  const int64_t* hoff;  // per slot
  int64_t n_reads;
  int nw;
  int32_t* fcnt;
  int32_t* fsel;
};
__device__ __forceinline__ void final_key(const FinalCtx& c, int64_t a, int i, uint64_t& k1, uint64_t& k2) {
  const int64_t h = a + i;
  if (!c.o.keep[h]) {
    k1 = k2 = ~0ull;
    return;
  }
  const uint32_t score = (uint32_t)((int64_t)INT_MAX - (int64_t)c.o.score[h]);
  k1 = ((uint64_t)score << 32) | (uint32_t)slot_window(c.hs[h], c.nw);
  k2 = ((uint64_t)(uint32_t)((int64_t)INT_MAX - (int64_t)c.hq[h]) << 32) | (uint32_t)i;
}
// What deleteHits_duplicateResult compares of a hit (tID, tIdx, qID, qIdx).
struct FinalId {
  int tid, tidx, qidx;
  uint32_t slot;
  __device__ __forceinline__ bool operator==(const FinalId& x) const {
    return tid == x.tid && tidx == x.tidx && qidx == x.qidx && slot == x.slot;
  }
};
__device__ __forceinline__ FinalId final_id(const FinalCtx& c, int64_t h) {
  return FinalId{(int)(c.hk[h] >> 32), c.o.t_idx[h], c.o.q_idx[h], c.hs[h]};
}

// Sorts the reads of the warp's groups of N lanes (n hits from a, one per
// lane), drops every hit equal to its predecessor of the same window
// (deleteHits_duplicateResult) and writes the kept ones.  Every lane of the
// warp takes part; n = 0 for a group without a read.
template <int N>
__device__ __forceinline__ void final_lanes(const FinalCtx& c, int64_t r, int64_t a, int n) {
  const int lane = threadIdx.x & 31, j = lane & (N - 1);
  const unsigned group = N == 32 ? kFull : ((1u << (N & 31)) - 1) << (lane & ~(N - 1));
  uint64_t k1 = ~0ull, k2 = ~0ull;
  if (j < n) final_key(c, a, j, k1, k2);
  if (__any_sync(kFull, n > 1)) lanes_sort<N>(k1, k2, lane);
  const bool kept = k1 != ~0ull;
  const int w = kept ? (int)(uint32_t)k1 : -1;
  const int64_t h = a + (uint32_t)k2;
  FinalId id{0, 0, 0, 0};
  if (kept) id = final_id(c, h);
  unsigned same = 0;  // the kept hits of this lane's window
  for (int x = 0; x < c.nw; ++x) {
    const unsigned m = __ballot_sync(kFull, w == x);
    if (w == x) same = m;
  }
  const unsigned before = same & group & lanemask_lt();
  const int src = before ? 31 - __clz(before) : lane;
  FinalId pr;
  pr.tid = __shfl_sync(kFull, id.tid, src);
  pr.tidx = __shfl_sync(kFull, id.tidx, src);
  pr.qidx = __shfl_sync(kFull, id.qidx, src);
  pr.slot = __shfl_sync(kFull, id.slot, src);
  const bool out = kept && !(before && id == pr);
  const unsigned m = __ballot_sync(kFull, out) & group;
  if (out) c.fsel[a + __popc(m & lanemask_lt())] = (int32_t)(uint32_t)k2;
  if (j == 0 && r >= 0) c.fcnt[r] = __popc(m);
}

// Reads of up to 8 hits take 8 lanes (most have one or two), up to 32 the
// whole warp; longer ones are listed for k_final_long.
__global__ void k_final_small(FinalCtx c, uint32_t* __restrict__ list, GroupCtl* __restrict__ ctl) {
  const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  const int lane = threadIdx.x & 31;
  int64_t a = 0;
  int n = 0;
  const bool in = r < c.n_reads;
  if (in) {
    a = c.hoff[2 * (int64_t)c.nw * r];
    n = (int)(c.hoff[2 * (int64_t)c.nw * (r + 1)] - a);
  }
  final_lanes<8>(c, in && n <= 8 ? r : -1, a, n <= 8 ? n : 0);
  for (unsigned m = __ballot_sync(kFull, n > 8 && n <= 32 && (lane & 7) == 0); m; m &= m - 1) {
    const int src = __ffs(m) - 1;
    final_lanes<32>(c, __shfl_sync(kFull, r, src), __shfl_sync(kFull, a, src), __shfl_sync(kFull, n, src));
  }
  if (n > 32 && (lane & 7) == 0) list[atomicAdd(&ctl->n_long, 1)] = (uint32_t)r;
}

// More than 32 hits: one CTA per read, in shared memory up to kCtaSortCap,
// else in global memory (g1, g2: one word per hit).
constexpr int kFinalLongThreads = 256;
__global__ void __launch_bounds__(kFinalLongThreads) k_final_long(FinalCtx c, uint64_t* __restrict__ g1,
                                                                  uint64_t* __restrict__ g2,
                                                                  const uint32_t* __restrict__ list,
                                                                  const GroupCtl* __restrict__ ctl) {
  __shared__ uint64_t s1[kCtaSortCap], s2[kCtaSortCap];
  __shared__ int warp_n[kFinalLongThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int total = ctl->n_long;
  for (int li = blockIdx.x; li < total; li += gridDim.x) {
    const int64_t r = list[li];
    const int64_t a = c.hoff[2 * (int64_t)c.nw * r];
    const int n = (int)(c.hoff[2 * (int64_t)c.nw * (r + 1)] - a);
    uint64_t* k1 = n <= kCtaSortCap ? s1 : g1 + a;
    uint64_t* k2 = n <= kCtaSortCap ? s2 : g2 + a;
    for (int i = threadIdx.x; i < n; i += kFinalLongThreads) final_key(c, a, i, k1[i], k2[i]);
    __syncthreads();
    cta_network(k1, k2, n);
    __syncthreads();
    int done = 0;
    for (int c0 = 0; c0 < n; c0 += kFinalLongThreads) {
      const int j = c0 + (int)threadIdx.x;
      bool out = j < n && k1[j] != ~0ull;
      if (out) {
        const uint32_t w = (uint32_t)k1[j];
        int p = j - 1;  // the predecessor of the same window
        while (p >= 0 && (uint32_t)k1[p] != w) --p;
        if (p >= 0) out = !(final_id(c, a + (uint32_t)k2[j]) == final_id(c, a + (uint32_t)k2[p]));
      }
      const unsigned m = __ballot_sync(kFull, out);
      if (lane == 0) warp_n[warp] = __popc(m);
      __syncthreads();
      int at = done + __popc(m & lanemask_lt()), all = 0;
      for (int x = 0; x < kFinalLongThreads / 32; ++x) {
        if (x < warp) at += warp_n[x];
        all += warp_n[x];
      }
      if (out) c.fsel[a + at] = (int32_t)(uint32_t)k2[j];
      done += all;
      __syncthreads();
    }
    if (threadIdx.x == 0) c.fcnt[r] = done;
    __syncthreads();
  }
}

// The kept hits of every read, in order, 8 lanes per read.
__global__ void k_final_write(FinalCtx c, const int64_t* __restrict__ foff, OutView out) {
  const int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  if (r >= c.n_reads) return;
  const int64_t a = c.hoff[2 * (int64_t)c.nw * r], b = foff[r];
  const int n = c.fcnt[r];
  for (int j = threadIdx.x & 7; j < n; j += 8) {
    const int64_t h = a + c.fsel[a + j];
    const int64_t x = b + j;
    const uint32_t slot = c.hs[h];
    const int w = slot_window(slot, c.nw);
    const int strand = (int)(slot & 1u);
    if (out.q_id) {
      out.q_id[x] = out.q_first + (int32_t)(2 * r) + strand;
    } else {
      out.read[x] = (int32_t)r;
      out.strand[x] = strand;
      out.t_load[x] = out.load[w];
    }
    out.t_seq[x] = out.t_first[w] + (int32_t)(c.hk[h] >> 32);
    out.t_idx[x] = c.o.t_idx[h];
    out.q_idx[x] = c.o.q_idx[h];
    out.t_len[x] = c.o.t_len[h];
    out.q_len[x] = c.o.q_len[h];
    out.match[x] = c.o.match[h];
    out.score[x] = c.o.score[h];
    out.evalue[x] = c.o.evalue[h];
  }
}

// ------------------------------------------------------------------------
// merge of the groups' results in holder order (CHostResultHolder::fixResult)
// ------------------------------------------------------------------------
__global__ void k_merge_count(const GroupHits* __restrict__ w, int nw, int64_t nreads, int32_t* __restrict__ cnt) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nreads) return;
  int64_t c = 0;
  for (int i = 0; i < nw; ++i) c += w[i].foff[r + 1] - w[i].foff[r];
  cnt[r] = (int32_t)c;
}

// Item j of group wi goes after every item of the same read from an earlier
// group with score >= its score, and every item of a later group with a
// strictly higher score: the stable sort by (read, score desc) of the
// concatenation in window order.
__global__ void k_merge_place(const GroupHits* __restrict__ w, int nw, int64_t total, const int64_t* __restrict__ moff,
                              OutView out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= total) return;
  int wi = 0;
  while (wi + 1 < nw && w[wi + 1].base <= i) ++wi;
  const GroupHits& a = w[wi];
  const int64_t j = i - a.base;
  const int64_t r = a.f[0][j];
  const int sc = a.f[9][j];
  int64_t pos = moff[r] + (j - a.foff[r]);
  for (int k = 0; k < nw; ++k) {
    if (k == wi) continue;
    const GroupHits& b = w[k];
    int64_t lo = b.foff[r], hi = b.foff[r + 1];
    const int64_t first = lo;
    // scores are non-increasing within a read: count the prefix that precedes sc
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      const int v = b.f[9][mid];
      if (k < wi ? v >= sc : v > sc) lo = mid + 1;
      else hi = mid;
    }
    pos += lo - first;
  }
  out.read[pos] = (int32_t)r;
  out.strand[pos] = a.f[1][j];
  out.t_load[pos] = a.f[2][j];
  out.t_seq[pos] = a.f[3][j];
  out.t_idx[pos] = a.f[4][j];
  out.q_idx[pos] = a.f[5][j];
  out.t_len[pos] = a.f[6][j];
  out.q_len[pos] = a.f[7][j];
  out.match[pos] = a.f[8][j];
  out.score[pos] = sc;
  out.evalue[pos] = a.evalue[j];
}

// INT32 throughput probe: 8 independent chains per thread of the DP's
// integer operation mix (add, max, logic): 4 ops per chain and iteration.
__global__ void __launch_bounds__(256) k_int32_probe(int iters, int k1, int k2, int* __restrict__ sink) {
  int a[8], b[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    a[c] = threadIdx.x + c * k1;
    b[c] = blockIdx.x - c * k2;
  }
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      a[c] = max(a[c] + k1, b[c]);
      b[c] = (b[c] ^ a[c]) + k2;
    }
  }
  int x = 0;
#pragma unroll
  for (int c = 0; c < 8; ++c) x += a[c] ^ b[c];
  if (x == 0x7fffffff) sink[0] = x;  // keeps the chains live
}

__global__ void k_gather_i64(const int64_t* __restrict__ src, const int64_t* __restrict__ idx, int n,
                             int64_t* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = src[idx[i]];
}

}  // namespace

// ------------------------------------------------------------------------
// launch wrappers
// ------------------------------------------------------------------------
void scan_i32(Workspace& ws, const int32_t* in, int64_t n, int64_t* out, cudaStream_t st) {
  scan_1pass(ws, ArrayLoad<int32_t>{in}, n, out, st);
}
int64_t scan_state_words(int64_t n) { return (n + kScanTile) / kScanTile + 1; }
void scan_i32_to(const int32_t* in, int64_t n, int64_t* out, unsigned long long* state, long long* total,
                 cudaStream_t st) {
  const int64_t tiles = scan_state_words(n) - 1;
  k_scan_1pass<<<(unsigned)tiles, kScanThreads, 0, st>>>(ArrayLoad<int32_t>{in}, n, n + 1, out, state, total);
  CLAST_LAUNCHED();
}

void pack_bases(const char* bases, int64_t n, uint64_t* packed, uint64_t* nmask, cudaStream_t st) {
  const int64_t nwords = (n + 63) / 64 + 1;  // one extra word so kmer_at may read w+1
  k_pack<<<blocks_for(nwords, 256), 256, 0, st>>>(bases, n, packed, nmask, nwords);
  CLAST_LAUNCHED();
}

void build_strands(const char* reads, const int64_t* offsets, int64_t n_reads, char* strands, int64_t* strand_start,
                   int32_t* strand_len, cudaStream_t st) {
  if (n_reads <= 0) return;
  k_strands<<<blocks_for(n_reads * 32, 256), 256, 0, st>>>(reads, offsets, n_reads, strands, strand_start, strand_len);
  CLAST_LAUNCHED();
}

void read_lengths(const int64_t* offsets, int64_t n_reads, int* min_len, int* max_len, cudaStream_t st) {
  if (n_reads <= 0) return;
  k_read_lengths<<<(unsigned)std::min<int64_t>(148, blocks_for(n_reads, 256)), 256, 0, st>>>(offsets, n_reads, min_len,
                                                                                           max_len);
  CLAST_LAUNCHED();
}

void build_window(const char* src, const int64_t* src_off, const int32_t* gateway, const int32_t* lengths,
                  int nseqs, int64_t n, char* out, cudaStream_t st) {
  if (n <= 0 || nseqs <= 0) return;
  k_build_window<<<blocks_for((n + 15) / 16, 256), 256, 0, st>>>(src, src_off, gateway, lengths, nseqs, n, out);
  CLAST_LAUNCHED();
}

void sample_keys(const uint64_t* packed, const uint64_t* nmask, int64_t n_samples, int stride, int l, int pbits,
                 uint64_t* items, int32_t* vals, cudaStream_t st) {
  if (n_samples <= 0) return;
  k_sample_keys<<<blocks_for(n_samples, 256), 256, 0, st>>>(packed, nmask, n_samples, stride, l, pbits, items,
                                                             vals);
  CLAST_LAUNCHED();
}

int radix_sort_u64(Workspace& ws, uint64_t* keys, int32_t* vals, uint64_t* keys_alt, int32_t* vals_alt, int64_t n,
                   int lo_bit, int hi_bit, cudaStream_t st) {
  if (n <= 1) return 0;
  const int nblocks = (int)((n + kRsTile - 1) / kRsTile);
  uint32_t* hist = ws.get<uint32_t>("rs_hist", (size_t)256 * nblocks);
  int64_t* offs = ws.get<int64_t>("rs_offs", (size_t)256 * nblocks + 1);
  const bool pay = vals != nullptr;
  const size_t smem = (size_t)kRsTile * (sizeof(uint64_t) + (pay ? sizeof(int32_t) : 0));
  // more than 48 KB of dynamic shared memory needs the opt-in (per device)
  if (pay) CLAST_CK(cudaFuncSetAttribute(k_rs_scatter<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  else CLAST_CK(cudaFuncSetAttribute(k_rs_scatter<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  uint64_t* a = keys;
  uint64_t* b = keys_alt;
  int32_t* va = vals;
  int32_t* vb = vals_alt;
  int which = 0;
  for (int shift = lo_bit; shift < hi_bit; shift += 8) {
    k_rs_hist<<<nblocks, kRsThreads, 0, st>>>(a, n, shift, hist, nblocks);
    CLAST_LAUNCHED();
    scan_1pass(ws, ArrayLoad<uint32_t>{hist}, (int64_t)256 * nblocks, offs, st);
    if (pay) k_rs_scatter<true><<<nblocks, kRsThreads, smem, st>>>(a, va, b, vb, n, shift, offs, nblocks);
    else k_rs_scatter<false><<<nblocks, kRsThreads, smem, st>>>(a, nullptr, b, nullptr, n, shift, offs, nblocks);
    CLAST_LAUNCHED();
    std::swap(a, b);
    std::swap(va, vb);
    which ^= 1;
  }
  return which;
}

// Runs that pass the cut can span more than a tile and the next (see IndexLead).
static bool index_long_runs(int cut) { return cut == -1 || cut > kIxLongRun; }

int64_t index_state_words(int64_t n_samples, int64_t n_records, int cut) {
  const int64_t tiles = (n_samples + kIxTile - 1) / kIxTile;
  return tiles + 1 + ((n_records >> kIxChunkLog) + 7) / 8 +
         (index_long_runs(cut) ? tiles * (int64_t)(sizeof(IndexLead) / sizeof(unsigned long long)) : 0);
}

void index_place(const uint64_t* items, const int32_t* vals, int64_t n_samples, int pbits, int stride, int l, int cut,
                 const int32_t* gateway, const int32_t* lengths, int nseqs, uint32_t nbuckets, int2* entries,
                 ulonglong2* table, int64_t n_records, uint32_t* filter, int fshift, int fstride,
                 unsigned long long* state, unsigned long long* kept, unsigned long long* failed, cudaStream_t st) {
  if (n_samples <= 0) {  // no tile: all records are free
    CLAST_CK(cudaMemsetAsync(table, 0xff, (size_t)n_records * sizeof(ulonglong2), st));
    return;
  }
  const int64_t tiles = (n_samples + kIxTile - 1) / kIxTile;
  const int64_t chunks = n_records >> kIxChunkLog;
  unsigned char* chunk_free = reinterpret_cast<unsigned char*>(state + tiles + 1);
  IndexLead* leads = reinterpret_cast<IndexLead*>(state + tiles + 1 + (chunks + 7) / 8);
  const IndexBuild b{items, vals, n_samples, pbits, 1ull << (2 * l), stride, l, cut, gateway, lengths, nseqs, nbuckets,
                     entries, table, n_records, filter, fshift, fstride, state, chunk_free, leads, kept, failed};
  const unsigned grid = (unsigned)tiles, some = (unsigned)std::min<int64_t>(tiles, 148 * 8);
  if (index_long_runs(cut)) {
    if (pbits > 0) k_index_leads<false><<<grid, kIxThreads, 0, st>>>(b);
    else k_index_leads<true><<<grid, kIxThreads, 0, st>>>(b);
    CLAST_LAUNCHED();
    if (pbits > 0) k_index_place<false, true><<<grid, kIxThreads, 0, st>>>(b);
    else k_index_place<true, true><<<grid, kIxThreads, 0, st>>>(b);
    CLAST_LAUNCHED();
    if (pbits > 0) k_index_lead_entries<false><<<some, kIxThreads, 0, st>>>(b, tiles);
    else k_index_lead_entries<true><<<some, kIxThreads, 0, st>>>(b, tiles);
  } else {
    if (pbits > 0) k_index_place<false, false><<<grid, kIxThreads, 0, st>>>(b);
    else k_index_place<true, false><<<grid, kIxThreads, 0, st>>>(b);
  }
  CLAST_LAUNCHED();
  if (chunks > 0) {
    k_index_free<<<(unsigned)std::min<int64_t>(chunks, 148 * 8), 256, 0, st>>>(table, chunk_free, chunks);
    CLAST_LAUNCHED();
  }
}

void filter_from_table(const ulonglong2* table, int64_t n_records, int l, uint32_t* filter, int fshift, int fstride,
                       bool file, cudaStream_t st) {
  if (n_records <= 0) return;
  const unsigned grid = (unsigned)((n_records + 255) / 256);
  if (file) k_filter_from_table<true><<<grid, 256, 0, st>>>(table, n_records, l, filter, fshift, fstride);
  else k_filter_from_table<false><<<grid, 256, 0, st>>>(table, n_records, l, filter, fshift, fstride);
  CLAST_LAUNCHED();
}

void seed_fused(const QueryView& q, const IndexView& ix, const TargetView& t, int gap, int local,
                unsigned long long* cursors, unsigned long long* n_kmers, int64_t* off, int32_t* cnt, int32_t* nvalid,
                uint64_t* skey, uint32_t* sq, int64_t part_cap, cudaStream_t st) {
  if (q.nstrands <= 0) return;
  // one warp per strand (one resident wave looping over the strands measured slower)
  const unsigned grid = blocks_for((int64_t)q.nstrands * 32, kSeedFusedThreads);
  if (ix.l <= 16)
    k_seed_fused<true><<<grid, kSeedFusedThreads, 0, st>>>(q, ix, t, gap, local, cursors, n_kmers, off, cnt, nvalid,
                                                          skey, sq, part_cap);
  else
    k_seed_fused<false><<<grid, kSeedFusedThreads, 0, st>>>(q, ix, t, gap, local, cursors, n_kmers, off, cnt, nvalid,
                                                           skey, sq, part_cap);
  CLAST_LAUNCHED();
}

template <int NW>
void launch_seed_reads(const QueryView& q, const SeedWins& W, int width, int gap, int local, int max_len,
                       cudaStream_t st) {
  const unsigned grid = blocks_for((int64_t)q.nstrands / 2 * 32, kSeedFusedThreads);
  const unsigned few = std::min<unsigned>(grid, 148 * 12);  // blocks that share the listed reads
  const unsigned teams = (unsigned)std::min<int64_t>(q.nstrands / 2, 148 * 8);
  if (W.w[0].ix.l <= 16) {
    k_seed_reads<true, NW><<<grid, kSeedFusedThreads, 0, st>>>(q, W, width, gap, local);
    CLAST_LAUNCHED();
    k_seed_reads_long<true, NW, 1><<<few, kSeedFusedThreads, 0, st>>>(q, W, gap, local);
    CLAST_LAUNCHED();
    if (max_len - W.w[0].ix.l < kSeedRound) return;
    k_seed_reads_long<true, NW, kLongTeam<NW>><<<teams, 32 * kLongTeam<NW>, 0, st>>>(q, W, gap, local);
  } else {
    k_seed_reads<false, NW><<<grid, kSeedFusedThreads, 0, st>>>(q, W, width, gap, local);
    CLAST_LAUNCHED();
    k_seed_reads_long<false, NW, 1><<<few, kSeedFusedThreads, 0, st>>>(q, W, gap, local);
    CLAST_LAUNCHED();
    if (max_len - W.w[0].ix.l < kSeedRound) return;
    k_seed_reads_long<false, NW, kLongTeam<NW>><<<teams, 32 * kLongTeam<NW>, 0, st>>>(q, W, gap, local);
  }
  CLAST_LAUNCHED();
}

void seed_reads(const QueryView& q, const SeedWins& W, int nw, int width, int gap, int local, int max_len,
                cudaStream_t st) {
  if (q.nstrands <= 0 || nw <= 0) return;
  switch (nw) {
    case 1: launch_seed_reads<1>(q, W, width, gap, local, max_len, st); break;
    case 2: launch_seed_reads<2>(q, W, width, gap, local, max_len, st); break;
    case 3: launch_seed_reads<3>(q, W, width, gap, local, max_len, st); break;
    case 4: launch_seed_reads<4>(q, W, width, gap, local, max_len, st); break;
    default: throw std::invalid_argument("seed_reads: 1 to 4 windows per group");
  }
}

void seed_filter(uint64_t* skey, uint32_t* sq, const int64_t* off, const int32_t* cnt, int32_t* nvalid,
                 const uint32_t* first_q, const int32_t* win_start, int n_windows, int nw, int width, int gap,
                 int64_t nv, uint32_t* lists, int32_t* hcnt, int64_t part_cap, GroupCtl* ctl, cudaStream_t st) {
  if (nv <= 0) return;
  if (n_windows > 0) {
    k_window_first<<<blocks_for((int64_t)n_windows * nw * 32, 256), 256, 0, st>>>(nvalid, win_start, n_windows, nw, cnt,
                                                                                 first_q, hcnt, part_cap, ctl);
    CLAST_LAUNCHED();
  }
  SeedFilterCtx c{off, cnt, nvalid, width, gap, hcnt, &ctl->full};
  if (!first_q) {
    k_seed_filter_small<<<blocks_for(nv, 256), 256, 0, st>>>(skey, sq, c, nv, lists, ctl);
    CLAST_LAUNCHED();
  }
  k_seed_filter_mid<<<grid_cap(std::min<int64_t>((nv + 3) / 4, 148 * 64)), kWarpSmemThreads, 0, st>>>(
      skey, sq, c, lists, &ctl->n_seeds[0]);
  CLAST_LAUNCHED();
  k_seed_filter_big<true><<<grid_cap(nv < 4096 ? nv : 4096), 256, 0, st>>>(skey, sq, c, lists + nv, &ctl->n_seeds[1]);
  CLAST_LAUNCHED();
  k_seed_filter_big<false><<<grid_cap(nv < 296 ? nv : 296), 1024, 0, st>>>(skey, sq, c, lists + 2 * nv,
                                                                           &ctl->n_seeds[2]);
  CLAST_LAUNCHED();
}

void gather_hits(const uint64_t* skey, const uint32_t* sq, const int64_t* off, const int32_t* hcnt,
                 const int64_t* hoff, int64_t nv, int nw, uint64_t* hk, int32_t* hq, uint32_t* hs,
                 const int32_t* qlen, int l, int band, const FirstSeeds& first, GroupCtl* ctl, cudaStream_t st) {
  if (nv <= 0) return;
  k_gather_hits<<<blocks_for(nv, 256), 256, 0, st>>>(skey, sq, off, hcnt, hoff, nv, nw, hk, hq, hs, qlen, l, band, first,
                                                     ctl);
  CLAST_LAUNCHED();
}

__global__ void k_dp_order_keys(const uint32_t* __restrict__ hs, int nw, const int32_t* __restrict__ q_len, int64_t n,
                                int l, int rows_max, uint64_t* __restrict__ keys) {
  const int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= n) return;
  const int rows = max(0, min(rows_max, q_len[slot_strand(hs[h], nw)] - l + 1));
  keys[h] = ((uint64_t)(rows_max - rows) << 32) | (uint32_t)h;
}

void dp_order_keys(const uint32_t* hs, int nw, const int32_t* q_len, int64_t n_hits, int l, int rows_max,
                   uint64_t* keys, cudaStream_t st) {
  if (n_hits <= 0) return;
  k_dp_order_keys<<<blocks_for(n_hits, 256), 256, 0, st>>>(hs, nw, q_len, n_hits, l, rows_max, keys);
  CLAST_LAUNCHED();
}

DpBuckets dp_bucket_count(Workspace& ws, const uint32_t* hs, int nw, const int32_t* q_len, int64_t n_hits, int l,
                          cudaStream_t st) {
  unsigned int* count = ws.get<unsigned int>("dpb_count", kDpBuckets);
  unsigned long long* rows = ws.get<unsigned long long>("dpb_rows", kDpBuckets);
  CLAST_CK(cudaMemsetAsync(count, 0, kDpBuckets * sizeof(unsigned int), st));
  CLAST_CK(cudaMemsetAsync(rows, 0, kDpBuckets * sizeof(unsigned long long), st));
  if (n_hits > 0) {
    k_dp_bucket_count<<<grid_cap(std::min<int64_t>(blocks_for(n_hits, 256), 1184)), 256, 0, st>>>(hs, nw, q_len,
                                                                                                    n_hits, l, count, rows);
    CLAST_LAUNCHED();
  }
  DpBuckets b;
  b.count = count;
  b.rows = rows;
  return b;
}

int dp_warp_mode_from_env(int fallback) {
  const char* v = std::getenv("CLAST_DP_WARP");
  if (!v) return fallback;
  if (!std::strcmp(v, "off")) return kDpWarpOff;
  if (!std::strcmp(v, "all")) return kDpWarpAll;
  return fallback;
}

long long banded_dp(const TargetView* t, int nw, const QueryView& q, const uint64_t* hk, const int32_t* hq,
                    const uint32_t* hs, const uint64_t* order, int64_t n_hits, const DpParams& p, const DpOut& o,
                    cudaStream_t st, const DpLaunch& m) {
  if (n_hits <= 0) return 0;
  DpKernelArgs a{};
  for (int w = 0; w < nw; ++w) a.t[w] = t[w];
  a.nw = nw;
  a.q = q;
  a.hk = hk;
  a.hq = hq;
  a.hs = hs;
  a.order = order;
  a.n = n_hits;
  a.p = p;
  a.o = o;
  a.bad = m.bad;
  const bool local = p.local != 0;
  switch (p.gap) {
    case 2: return launch_dp_gap<2>(a, local, m, st);
    case 3: return launch_dp_gap<3>(a, local, m, st);
    case 4: return launch_dp_gap<4>(a, local, m, st);
    case 5: return launch_dp_gap<5>(a, local, m, st);
    case 6: return launch_dp_gap<6>(a, local, m, st);
    case 7: return launch_dp_gap<7>(a, local, m, st);
    case 8: return launch_dp_gap<8>(a, local, m, st);
    case 9: return launch_dp_gap<9>(a, local, m, st);
    case 10: return launch_dp_gap<10>(a, local, m, st);
    case 11: return launch_dp_gap<11>(a, local, m, st);
    case 12: return launch_dp_gap<12>(a, local, m, st);
    case 13: return launch_dp_gap<13>(a, local, m, st);
    case 14: return launch_dp_gap<14>(a, local, m, st);
    case 15: return launch_dp_gap<15>(a, local, m, st);
    case 16: return launch_dp_gap<16>(a, local, m, st);
    default: throw std::invalid_argument("gap out of range 2..16");
  }
}

void merge_groups(const GroupHits* groups, int n, int64_t total, int64_t nreads, int32_t* cnt, int64_t* moff,
                  const OutView& out, Workspace& ws, cudaStream_t st) {
  if (nreads <= 0) return;
  k_merge_count<<<blocks_for(nreads, 256), 256, 0, st>>>(groups, n, nreads, cnt);
  CLAST_LAUNCHED();
  scan_i32(ws, cnt, nreads, moff, st);
  if (total > 0) {
    k_merge_place<<<blocks_for(total, 256), 256, 0, st>>>(groups, n, total, moff, out);
    CLAST_LAUNCHED();
  }
}

double int32_probe(cudaStream_t st, int* sink) {
  int dev = 0, sms = 0;
  CLAST_CK(cudaGetDevice(&dev));
  CLAST_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const int blocks = sms * 8, threads = 256, iters = 4096;
  cudaEvent_t a, b;
  CLAST_CK(cudaEventCreate(&a));
  CLAST_CK(cudaEventCreate(&b));
  k_int32_probe<<<blocks, threads, 0, st>>>(64, 3, 5, sink);  // warm-up
  CLAST_LAUNCHED();
  CLAST_CK(cudaEventRecord(a, st));
  k_int32_probe<<<blocks, threads, 0, st>>>(iters, 3, 5, sink);
  CLAST_LAUNCHED();
  CLAST_CK(cudaEventRecord(b, st));
  CLAST_CK(cudaEventSynchronize(b));
  float ms = 0;
  CLAST_CK(cudaEventElapsedTime(&ms, a, b));
  cudaEventDestroy(a);
  cudaEventDestroy(b);
  const double ops = (double)blocks * threads * iters * 8 * 4;
  return ops / (ms * 1e-3) / 1e12;
}

void gather_i64(const int64_t* src, const int64_t* idx, int n, int64_t* out, cudaStream_t st) {
  if (n <= 0) return;
  k_gather_i64<<<blocks_for(n, 256), 256, 0, st>>>(src, idx, n, out);
  CLAST_LAUNCHED();
}

void final_order(const uint64_t* hk, const int32_t* hq, const uint32_t* hs, const DpOut& o, const int64_t* hoff,
                 int64_t n_reads, int nw, uint64_t* g1, uint64_t* g2, uint32_t* list, int32_t* fcnt, int32_t* fsel,
                 GroupCtl* ctl, cudaStream_t st) {
  if (n_reads <= 0) return;
  const FinalCtx c{hk, hq, hs, o, hoff, n_reads, nw, fcnt, fsel};
  k_final_small<<<blocks_for(n_reads * 8, 256), 256, 0, st>>>(c, list, ctl);
  CLAST_LAUNCHED();
  k_final_long<<<grid_cap(n_reads < 2048 ? n_reads : 2048), kFinalLongThreads, 0, st>>>(c, g1, g2, list, ctl);
  CLAST_LAUNCHED();
}
void final_write(const uint64_t* hk, const uint32_t* hs, const DpOut& o, const int64_t* hoff, int64_t n_reads, int nw,
                 const int32_t* fcnt, const int32_t* fsel, const int64_t* foff, const OutView& out, cudaStream_t st) {
  if (n_reads <= 0) return;
  const FinalCtx c{hk, nullptr, hs, o, hoff, n_reads, nw, const_cast<int32_t*>(fcnt), const_cast<int32_t*>(fsel)};
  k_final_write<<<blocks_for(n_reads * 8, 256), 256, 0, st>>>(c, foff, out);
  CLAST_LAUNCHED();
}

}  // namespace clast
