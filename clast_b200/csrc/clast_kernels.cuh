// clast_kernels.cuh -- launch wrappers of the sm_100a kernels (clast_kernels.cu).
// Every wrapper enqueues on `st` and returns immediately; sizes are element counts.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "clast_device.cuh"

namespace clast {

struct Workspace;  // device scratch pool (clast_engine.cu)

// out[0..n] = exclusive prefix sums of in[0..n) (out[n] = total).
void scan_i32(Workspace& ws, const int32_t* in, int64_t n, int64_t* out, cudaStream_t st);
// The same with the caller's zeroed state of scan_state_words(n) words, the total
// also in *total (device, may be null).
int64_t scan_state_words(int64_t n);
void scan_i32_to(const int32_t* in, int64_t n, int64_t* out, unsigned long long* state, long long* total,
                 cudaStream_t st);
// 2-bit codes (32 bases per word) and non-ACGT mask (64 per word) of bases[0..n);
// positions >= n count as 'N'.  packed needs ceil(n/32)+2 words, nmask ceil(n/64)+2.
void pack_bases(const char* bases, int64_t n, uint64_t* packed, uint64_t* nmask, cudaStream_t st);

// Query strands of n_reads one-strand reads: strand 2r = read r, strand 2r+1 its
// reverse complement (utilReverseSeq.cpp:3-19), laid out back to back, with kPad
// 'N' bytes before and after them.
void build_strands(const char* reads, const int64_t* offsets, int64_t n_reads, char* strands, int64_t* strand_start,
                   int32_t* strand_len, cudaStream_t st);

// Shortest and longest of the reads (*min_len preset to INT_MAX, *max_len to 0);
// no read may be longer than INT_MAX.
void read_lengths(const int64_t* offsets, int64_t n_reads, int* min_len, int* max_len, cudaStream_t st);

// ---- index of one target window (CDeviceHashTable.cu:20-174) ----
// Window base array (sequences with their joints) from a one-strand source set:
// sequence k of the window is src[src_off[k] .. src_off[k]+lengths[k]).
void build_window(const char* src, const int64_t* src_off, const int32_t* gateway, const int32_t* lengths,
                  int nseqs, int64_t n, char* out, cudaStream_t st);
// Samples at window positions j*stride: order_code of the l-mer (4^l when it
// has a non-ACGT base).  pbits > 0: items[j] = code << pbits | j; pbits = 0:
// items[j] = code, vals[j] = j.
void sample_keys(const uint64_t* packed, const uint64_t* nmask, int64_t n_samples, int stride, int l, int pbits,
                 uint64_t* items, int32_t* vals, cudaStream_t st);
// Stable LSD radix sort of 64-bit words by bits [lo_bit, hi_bit), carrying
// vals along unless vals is null.  Returns 0 when the result is in (keys,
// vals), 1 when it is in (keys_alt, vals_alt).
int radix_sort_u64(Workspace& ws, uint64_t* keys, int32_t* vals, uint64_t* keys_alt, int32_t* vals_alt, int64_t n,
                   int lo_bit, int hi_bit, cudaStream_t st);
// The index from the sorted samples (as sample_keys lays them out): entries of
// the kept ones (n_samples long, runs of equal codes apart), the hash table
// without atomics (layout: IndexView; every record of it is written, free ones
// as ~0) and the filter (zeroed by the caller).  state:
// index_state_words(n_samples, n_records, cut) zeroed words; *kept is raised by the
// records placed, *failed by records outside the table and by waits that gave
// up (neither happens).
int64_t index_state_words(int64_t n_samples, int64_t n_records, int cut);
void index_place(const uint64_t* items, const int32_t* vals, int64_t n_samples, int pbits, int stride, int l, int cut,
                 const int32_t* gateway, const int32_t* lengths, int nseqs, uint32_t nbuckets, int2* entries,
                 ulonglong2* table, int64_t n_records, uint32_t* filter, int fshift, int fstride,
                 unsigned long long* state, unsigned long long* kept, unsigned long long* failed, cudaStream_t st);
// The filter (zeroed by the caller) of a table's keys: as it is searched, or
// with `file` as index files hold it (fstride 1).
void filter_from_table(const ulonglong2* table, int64_t n_records, int l, uint32_t* filter, int fshift, int fstride,
                       bool file, cudaStream_t st);

// ---- seeds (CDeviceHitList_createRawSeedList.cu, _deleteSeeds*.cu, _sortSeeds.cu) ----
// A group of up to kMaxSeedWins target windows is searched together.  Its slots
// are the (strand, window) pairs, a read's slots side by side: slot (s, w) of
// nw windows is (s / 2) * 2 nw + 2 w + (s & 1).
constexpr int kMaxSeedWins = 4;
constexpr int kSeedParts = 32;
__host__ __device__ __forceinline__ int64_t strand_slot(int64_t s, int w, int nw) {
  return (s >> 1) * (2 * nw) + 2 * w + (s & 1);
}
__host__ __device__ __forceinline__ int64_t slot_strand(uint32_t v, int nw) {
  return nw == 1 ? (int64_t)v : 2 * (int64_t)(v / (uint32_t)(2 * nw)) + (v & 1u);
}
__host__ __device__ __forceinline__ int slot_window(uint32_t v, int nw) {
  return nw == 1 ? 0 : (int)((v >> 1) % (uint32_t)nw);
}

// Counters of one group's search, zeroed before it.
struct GroupCtl {
  unsigned long long cursor[kSeedParts];                // seeds and hits stored per partition
  unsigned long long kmers[kMaxSeedWins][kSeedParts];   // valid l-mers of the partition's strands
  unsigned long long seeds[kMaxSeedWins][kSeedParts];   // their seeds (seed_reads)
  unsigned long long cells;                             // DP cells
  long long hits, results;
  long long dp_warp;  // hits the DP's split sends to the one-per-warp kernel
  int bad;            // see DpLaunch::bad
  int full;           // a seed partition overflowed: the filters write no hits, the search runs again
  int n_seeds[3];     // slots listed for the seed filters' longer tiers
  int n_stored[4];    // reads whose seeds are stored: of one round, longer, and how many of each are taken
  int n_long;         // reads listed for k_final_long
};

// One-pass seeding of one window (lookups once): off/cnt/nvalid per strand,
// seeds in skey/sq, which hold kSeedParts partitions of part_cap seeds.  Strand
// s reserves its range in partition s % kSeedParts through cursors[partition];
// a partition whose cursor ends above part_cap was not fully written (its
// strands have no valid seed then) and the call must be repeated with part_cap
// >= the largest cursor.  n_kmers holds kSeedParts counters (the caller sums
// them), so that no single address takes one atomic per strand.
void seed_fused(const QueryView& q, const IndexView& ix, const TargetView& t, int gap, int local,
                unsigned long long* cursors, unsigned long long* n_kmers, int64_t* off, int32_t* cnt, int32_t* nvalid,
                uint64_t* skey, uint32_t* sq, int64_t part_cap, cudaStream_t st);
// Seeding of whole reads (strand 2r + 1 the reverse complement of strand 2r) in
// the nw windows of a group, in one pass.  Slots of up to 32 seeds of reads of
// up to 160 l-mers are filtered at once: hcnt hits at off, cnt 0, nvalid valid
// seeds, and the first of them in first_key / first_q (see k_window_first).
// The others' seeds are stored (off, cnt, nvalid) and the slots listed for
// seed_filter (lists: three of nw * nstrands words, n_listed: their counts).
// Seeds and hits share kSeedParts partitions of nw * part_cap of skey/sq, read
// r's in partition r % kSeedParts, reserved through cursor as in seed_fused.
// Every window must have been built with the same l.  max_len: no strand is
// longer (INT_MAX when that is not known).
struct SeedWin {
  IndexView ix;
  TargetView t;
  unsigned long long* n_kmers;  // kSeedParts l-mer counters
  unsigned long long* n_seeds;  // kSeedParts seed counters
  int paired;                   // an odd window whose filter words follow those of the window before it
};
struct SeedWins {
  SeedWin w[kMaxSeedWins];
  unsigned long long* cursor;
  int64_t* off;
  int32_t* cnt;
  int32_t* nvalid;
  int32_t* hcnt;
  uint64_t* first_key;
  uint32_t* first_q;
  uint32_t* lists;
  int* n_listed;
  uint32_t* long_reads;  // the reads whose seeds are stored, one word per read
  int* n_long;           // GroupCtl::n_stored
  int words;             // every window has less than 2^20 sequences (seed_word)
  uint64_t* skey;
  uint32_t* sq;
  int64_t part_cap;
};
void seed_reads(const QueryView& q, const SeedWins& W, int nw, int width, int gap, int local, int max_len,
                cudaStream_t st);

// sortSeeds + deletingIsolateSeeds + deleteDuplicateSeeds per slot: sorts the
// cnt[v] seeds of slot v by (sequence, diagonal, qIdx) and writes the surviving
// hits at off[v] onwards, hcnt[v] of them.  lists: 3 nv words.  With first_q
// (seed_reads) only the listed slots are left to filter.  The first slot
// of every (target window, query window) with a valid seed has its nvalid
// complemented.  part_cap: seeds that a partition holds (all windows').
void seed_filter(uint64_t* skey, uint32_t* sq, const int64_t* off, const int32_t* cnt, int32_t* nvalid,
                 const uint32_t* first_q, const int32_t* win_start, int n_windows, int nw, int width, int gap,
                 int64_t nv, uint32_t* lists, int32_t* hcnt, int64_t part_cap, GroupCtl* ctl, cudaStream_t st);
// First seeds of the slots that seed_reads filtered (key null: none).
struct FirstSeeds {
  const uint64_t* key;
  const uint32_t* q;
  const int32_t* nvalid;
  const int32_t* cnt;
};
// The hits of every slot back to back (hk: seed key, hq: qIdx, hs: slot); also
// adds band * (qlen - l) DP cells per hit to ctl->cells.
void gather_hits(const uint64_t* skey, const uint32_t* sq, const int64_t* off, const int32_t* hcnt,
                 const int64_t* hoff, int64_t nv, int nw, uint64_t* hk, int32_t* hq, uint32_t* hs,
                 const int32_t* qlen, int l, int band, const FirstSeeds& first, GroupCtl* ctl, cudaStream_t st);

// ---- banded DP + E-value (krnlAlignment.cu, krnlCalculateEvalue.cu) ----
struct DpOut {
  int32_t* t_idx; int32_t* q_idx; int32_t* t_len; int32_t* q_len; int32_t* match; int32_t* score;
  double* evalue; uint8_t* keep;
};
struct DpParams {
  int l, stride, gap, local;
  double cutoff, total_db, K, lambda;
};
// How the DP is launched: one thread per hit over a grid of all hits, in blocks
// that sort hits of one length (uniform_rows) by the rows of their forward pass.
//
// The first hits of the order (the longest, when the order is longest first) may
// run one per warp (an anti-diagonal wavefront over the band) instead of one per
// thread: a 5 kbp hit alone takes 0.54 against 0.95 ms there at gap 8 (0.56 and
// 1.65 in local mode, 0.54 and 2.13 at gap 16), at a lower throughput per cell.
// `warp` says how many:
// kDpWarpAuto splits where the cost model puts the end of both launches
// earliest -- on the device from the length buckets' counts and row sums
// (buckets + warp_n), or, for hits that all have `uniform_rows` rows, all or
// none on the host; kDpWarpOff runs every hit one per thread, kDpWarpAll one
// per warp.  Results are the same either way.
constexpr int kDpWarpAuto = 0, kDpWarpOff = 1, kDpWarpAll = 2;
// Rows from which a hit runs one per warp, in 32-bit integers, whatever the
// launch asks for: the one-per-thread kernel holds whole numbers in floats,
// which are exact below 2^24.  In a pass of r rows its potentials stay within
// 5 r + 34,000 of zero (they rise by up to 5 per row, and a score is never below
// what the left margin of -30,000 and a gap along the row give), and its match
// counts between -30,100 and r (a step adds at least as much to them as to the
// score).  A bound of the length buckets; such hits are the first of the order,
// so the others of their batch are split as in any other.
constexpr int kDpMaxThreadRows = 1 << 20;
struct DpBuckets {
  const unsigned int* count = nullptr;      // hits per length bucket (longest first)
  const unsigned long long* rows = nullptr;  // their rows, summed
};
struct DpLaunch {
  int warp = kDpWarpAuto;
  DpBuckets buckets;
  long long* warp_n = nullptr;  // device word for the split (with buckets)
  int uniform_rows = -1;
  bool long_hits = false;  // some hit may have kDpMaxThreadRows rows or more (needs buckets and warp_n)
  // with aux, the one-per-warp kernel runs there, beside the others (forked
  // from and joined back into the launch stream by the two events)
  cudaStream_t aux = nullptr;
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
  // device word set to 1 when a hit names a target sequence or strand outside
  // the window (an internal error: the hit is skipped, never read past)
  int* bad = nullptr;
};
// order (may be null): the hits in the order the threads take them, as words
// whose low 32 bits are hit indices; outputs stay at the hit's own index.
// Returns how many hits ran one per warp, or -1 when the split was made on the
// device (the count is then in *m.warp_n).
long long banded_dp(const TargetView* t, int nw, const QueryView& q, const uint64_t* hk, const int32_t* hq,
                    const uint32_t* hs, const uint64_t* order, int64_t n_hits, const DpParams& p, const DpOut& o,
                    cudaStream_t st, const DpLaunch& m = DpLaunch());
// Hits per length bucket (16 per power of two of the row count, longest
// first) and their row sums, in the workspace.
DpBuckets dp_bucket_count(Workspace& ws, const uint32_t* hs, int nw, const int32_t* q_len, int64_t n_hits, int l,
                          cudaStream_t st);
// CLAST_DP_WARP=off|all, else `fallback` (the environment overrides a
// context's setting, for tests and measurements).
int dp_warp_mode_from_env(int fallback);
// keys[h] = (rows_max - rows of hit h) << 32 | h, rows = q_len[hs[h]] - l + 1:
// ascending keys take the hits longest first.
void dp_order_keys(const uint32_t* hs, int nw, const int32_t* q_len, int64_t n_hits, int l, int rows_max,
                   uint64_t* keys, cudaStream_t st);

// ---- per-read result order and duplicate removal (utilResultSorting.cuh, CDeviceHitList.cu:32-128) ----
// fcnt[r] kept hits of read r, fsel[hoff of the read + j] the j-th of them (its
// position in the read's run).  g1, g2: one word per hit; list: one per read.
void final_order(const uint64_t* hk, const int32_t* hq, const uint32_t* hs, const DpOut& o, const int64_t* hoff,
                 int64_t n_reads, int nw, uint64_t* g1, uint64_t* g2, uint32_t* list, int32_t* fcnt, int32_t* fsel,
                 GroupCtl* ctl, cudaStream_t st);
// Where result items go: q_id (q_first + strand) when given, else read, strand
// and t_load.
struct OutView {
  int32_t *read, *strand, *t_load, *t_seq, *t_idx, *q_idx, *t_len, *q_len, *match, *score;
  double* evalue;
  int32_t* q_id;
  int32_t q_first;
  int32_t t_first[kMaxSeedWins], load[kMaxSeedWins];  // per window of the group
};
void final_write(const uint64_t* hk, const uint32_t* hs, const DpOut& o, const int64_t* hoff, int64_t n_reads, int nw,
                 const int32_t* fcnt, const int32_t* fsel, const int64_t* foff, const OutView& out, cudaStream_t st);

// ---- merge of the groups in holder order (CHostResultHolder::fixResult) ----
struct GroupHits {  // one group's results (reads ascending), fields in OutView's order
  const int32_t* f[10];
  const double* evalue;
  const int64_t* foff;  // per read offsets, n_reads + 1
  int64_t base;         // position of its first item in the concatenation of all groups
};
// groups: device array of n; total = items of all groups; moff (nreads+1)
// receives per-read offsets of the merged result.
void merge_groups(const GroupHits* groups, int n, int64_t total, int64_t nreads, int32_t* cnt, int64_t* moff,
                  const OutView& out, Workspace& ws, cudaStream_t st);
void gather_i64(const int64_t* src, const int64_t* idx, int n, int64_t* out, cudaStream_t st);
// Measured INT32 throughput of this GPU in tera-ops/s (add, max, logic mix).
double int32_probe(cudaStream_t st, int* sink);

}  // namespace clast
