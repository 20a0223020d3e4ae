// cx_finalize.cu -- aggregate result finalisation on the device.
//
// The reference's generated post-processing turns the group table into
// columnar result rows (AggregateDenseCount / AggregateDenseWrite,
// src/core/visitor.cpp:2589-2697: a group is present when its visible tuple
// has a validity bit or a non-zero word; a scalar aggregate always yields one
// row; rows in group order), then orders and cuts them (SortLimit*,
// src/core/visitor.cpp:307-581: each key compared in the column's result type,
// a valid value before NULL, ties broken by row index; then LIMIT).  Here the
// row offsets come from a device prefix sum (the reference copies counts to
// the host), and ORDER BY sorts runs of 1024 rows in shared memory, then ranks
// every row against all other runs at once (64-way merge by rank).
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <mutex>

#include "../../include/crystal_b200.h"
#include "cx_internal.h"

namespace {

int ffail(int code, const char* msg) { return cx_internal::set_error(code, msg); }

int fcuda(cudaError_t e, const char* what) {
  char buf[512];
  snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
  return cx_internal::set_error(CX_E_CUDA, buf);
}

constexpr int kMaxCols = 32;
constexpr int kMaxKeys = 8;
constexpr int kBlock = 256;
constexpr unsigned long long kPerBlock = 2048;  // groups per block of the count / write passes
constexpr unsigned kInvalid = 0xffffffffu;
constexpr unsigned long long kSelfScan = 2048;  // most blocks that fin_write lets sum the counts themselves
constexpr int kMaxWords = 2 * kMaxKeys;  // sort words of a row: per key a null flag (nullable columns) and the value
constexpr unsigned kRun = 1024;          // rows of a run sorted in shared memory
constexpr unsigned kWays = 64;           // runs merged by one ranking pass
constexpr unsigned long long kDirectGroups = (unsigned long long)kRun * kWays;

struct FinDesc {
  unsigned long long groups;
  unsigned ts, cols;
  int sparse, scalar;
  unsigned char type[kMaxCols];      // CX_COL_INT64 / UINT64 / FLOAT64
  unsigned char nullable[kMaxCols];
  int nkeys;
  int key_col[kMaxKeys];
  int key_desc[kMaxKeys];
  int words;                         // sort words per row
};

__device__ __forceinline__ bool bit_at(const unsigned long long* v, unsigned long long i) {
  return (v[i >> 6] >> (i & 63)) & 1ULL;
}

__device__ __forceinline__ bool present(const unsigned long long* __restrict__ src,
                                        const unsigned long long* __restrict__ val, const FinDesc& d,
                                        unsigned long long g) {
  if (d.scalar) return true;
  const unsigned long long base = g * d.ts;
  if (d.sparse) {
    for (unsigned c = 0; c < d.ts; ++c)
      if (src[base + c] != 0ULL) return true;
    return false;
  }
  for (unsigned c = 0; c < d.cols; ++c)
    if ((val && bit_at(val, base + c)) || src[base + c] != 0ULL) return true;
  return false;
}

// Pass 1: present groups per block of kPerBlock groups.
__global__ void __launch_bounds__(kBlock) fin_count(const unsigned long long* __restrict__ src,
                                                    const unsigned long long* __restrict__ val, const FinDesc d,
                                                    unsigned long long* __restrict__ counts,
                                                    unsigned long long* __restrict__ nan_keys) {
  const unsigned long long g0 = (unsigned long long)blockIdx.x * kPerBlock;
  unsigned long long cnt = 0;
  for (unsigned long long g = g0 + threadIdx.x; g < g0 + kPerBlock && g < d.groups; g += kBlock) {
    if (!present(src, val, d, g)) continue;
    ++cnt;
    if (!nan_keys) continue;
    for (int k = 0; k < d.nkeys; ++k) {
      const double x = __longlong_as_double((long long)src[g * d.ts + d.key_col[k]]);
      if (d.type[d.key_col[k]] == CX_COL_FLOAT64 && x != x) *nan_keys = 1ULL;
    }
  }
  __shared__ unsigned long long part[kBlock / 32];
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long s = 0;
    for (int w = 0; w < kBlock / 32; ++w) s += part[w];
    counts[blockIdx.x] = s;
  }
}

// Pass 2: exclusive prefix of the block counts (one CTA) and the row total.
__global__ void __launch_bounds__(1024) fin_scan(unsigned long long* counts, unsigned long long nblocks,
                                                 unsigned long long* total) {
  __shared__ unsigned long long carry;
  __shared__ unsigned long long wsum[32];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (unsigned long long b = 0; b < nblocks; b += 1024) {
    const unsigned long long i = b + threadIdx.x;
    const unsigned long long v = i < nblocks ? counts[i] : 0ULL;
    unsigned long long x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
      unsigned long long w = wsum[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      wsum[lane] = w;
    }
    __syncthreads();
    const unsigned long long incl = x + (warp > 0 ? wsum[warp - 1] : 0ULL);
    if (i < nblocks) counts[i] = carry + incl - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry += incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

// Pass 3: present groups become rows, column by column, in group order; rows
// from `limit` on are counted but not written.  With `rowgrp`, only each row's
// group is written (the ORDER BY of a large result sorts those).  `offsets`
// holds the blocks' exclusive prefix, or (total non-null) the block counts,
// which every block then sums up to its own: for up to kSelfScan blocks that
// is at most 16 KB from L2 per block, less than the launch of a scan kernel.
__global__ void __launch_bounds__(kBlock) fin_write(const unsigned long long* __restrict__ src,
                                                    const unsigned long long* __restrict__ val, const FinDesc d,
                                                    const unsigned long long* __restrict__ offsets,
                                                    unsigned long long* __restrict__ cols, unsigned long long* vcols,
                                                    unsigned long long row_cap, unsigned long long limit,
                                                    unsigned* __restrict__ rowgrp, unsigned long long* total) {
  const unsigned long long g0 = (unsigned long long)blockIdx.x * kPerBlock;
  const unsigned long long vw = (row_cap + 63) / 64;
  __shared__ unsigned long long warp_tot[kBlock / 32];
  __shared__ unsigned long long base_s;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (total) {
    unsigned long long sum = 0;
    for (unsigned b = threadIdx.x; b < blockIdx.x; b += kBlock) sum += offsets[b];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if (lane == 0) warp_tot[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned long long t = 0;
      for (int w = 0; w < kBlock / 32; ++w) t += warp_tot[w];
      base_s = t;
      if (blockIdx.x == gridDim.x - 1) *total = t + offsets[blockIdx.x];
    }
  } else if (threadIdx.x == 0) {
    base_s = offsets[blockIdx.x];
  }
  __syncthreads();
  for (unsigned long long chunk = g0; chunk < g0 + kPerBlock && chunk < d.groups; chunk += kBlock) {
    const unsigned long long g = chunk + threadIdx.x;
    const bool p = g < d.groups && g < g0 + kPerBlock && present(src, val, d, g);
    const unsigned ballot = __ballot_sync(0xffffffffu, p);
    if (lane == 0) warp_tot[warp] = __popc(ballot);
    __syncthreads();
    unsigned long long row = base_s;
    for (int w = 0; w < warp; ++w) row += warp_tot[w];
    row += __popc(ballot & ((1u << lane) - 1u));
    if (p && rowgrp) {
      rowgrp[row] = (unsigned)g;
    } else if (p && row < limit) {
      const unsigned long long base = g * d.ts;
      for (unsigned c = 0; c < d.cols; ++c) {
        cols[c * row_cap + row] = src[base + c];
        const bool valid = d.sparse || !d.nullable[c] || (val && bit_at(val, base + c));
        if (valid) atomicOr(&vcols[c * vw + (row >> 6)], 1ULL << (row & 63));
      }
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (int w = 0; w < kBlock / 32; ++w) base_s += warp_tot[w];
    __syncthreads();
  }
}

// True when row `r` orders before row `l` (the reference's comparator).
__device__ __forceinline__ bool right_before_left(const unsigned long long* __restrict__ cols,
                                                  const unsigned long long* __restrict__ vcols, const FinDesc& d,
                                                  unsigned long long row_cap, unsigned l, unsigned r) {
  if (r == l) return false;
  if (r == kInvalid) return false;
  if (l == kInvalid) return true;
  const unsigned long long vw = (row_cap + 63) / 64;
  for (int k = 0; k < d.nkeys; ++k) {
    const int c = d.key_col[k];
    if (d.nullable[c]) {
      const bool lv = bit_at(vcols + (unsigned long long)c * vw, l), rv = bit_at(vcols + (unsigned long long)c * vw, r);
      if (lv != rv) return rv;
      if (!lv) continue;
    }
    const unsigned long long a = cols[(unsigned long long)c * row_cap + l], b = cols[(unsigned long long)c * row_cap + r];
    bool lt, gt;  // right < left, left < right
    if (d.type[c] == CX_COL_INT64) {
      lt = (long long)b < (long long)a;
      gt = (long long)a < (long long)b;
    } else if (d.type[c] == CX_COL_FLOAT64) {
      lt = __longlong_as_double((long long)b) < __longlong_as_double((long long)a);
      gt = __longlong_as_double((long long)a) < __longlong_as_double((long long)b);
    } else {
      lt = b < a;
      gt = a < b;
    }
    if (lt) return !d.key_desc[k];
    if (gt) return d.key_desc[k] != 0;
  }
  return r < l;
}

// A bitonic network over row indices with the comparator itself: only for
// DOUBLE keys that hold a NaN, which compares as equal to everything, so the
// order follows from the network and not from the keys.
__global__ void fin_sort_init(unsigned* idx, unsigned long long rows, unsigned long long n) {
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x)
    idx[i] = i < rows ? (unsigned)i : kInvalid;
}

// One compare-exchange step (k, j) of the global bitonic network.
__global__ void fin_sort_step(const unsigned long long* __restrict__ cols, const unsigned long long* __restrict__ vcols,
                              const FinDesc d, unsigned long long row_cap, unsigned* idx, unsigned long long n,
                              unsigned long long k, unsigned long long j) {
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned long long x = i ^ j;
    if (x <= i) continue;
    const unsigned l = idx[i], r = idx[x];
    const bool rb = right_before_left(cols, vcols, d, row_cap, l, r);
    const bool lb = l != r && !rb;
    if ((i & k) == 0 ? rb : lb) { idx[i] = r; idx[x] = l; }
  }
}

// Reorders the first `out` sorted rows into temporary columns.
__global__ void fin_gather(const unsigned long long* __restrict__ cols, const unsigned long long* __restrict__ vcols,
                           const FinDesc d, unsigned long long row_cap, const unsigned* __restrict__ idx,
                           unsigned long long out, unsigned long long* __restrict__ tcols,
                           unsigned long long* __restrict__ tv) {
  const unsigned long long vw = (row_cap + 63) / 64;
  for (unsigned long long o = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; o < out;
       o += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned src = idx[o];
    for (unsigned c = 0; c < d.cols; ++c) {
      tcols[c * row_cap + o] = cols[c * row_cap + src];
      if (bit_at(vcols + c * vw, src)) atomicOr(&tv[c * vw + (o >> 6)], 1ULL << (o & 63));
    }
  }
}

// The sort words of group g: comparing them as unsigned numbers one after
// another, then the group, gives the comparator's order (no NaN among the
// keys).  Per key: 0 / 1 for a valid / NULL value where the column is
// nullable, then the value with its order mapped to unsigned order (sign bit
// flipped for INT64, the IEEE total order with -0.0 = +0.0 for FLOAT64),
// complemented for DESC; a NULL's value word is 0.
__device__ __forceinline__ unsigned long long sort_word(const unsigned long long* __restrict__ src,
                                                        const unsigned long long* __restrict__ val, const FinDesc& d,
                                                        unsigned long long g, int k, bool flag) {
  const int c = d.key_col[k];
  const unsigned long long at = g * d.ts + c;
  const bool valid = d.sparse || !d.nullable[c] || (val && bit_at(val, at));
  if (flag) return valid ? 0ULL : 1ULL;
  if (!valid) return 0ULL;
  unsigned long long x = src[at];
  if (d.type[c] == CX_COL_INT64) {
    x ^= 1ULL << 63;
  } else if (d.type[c] == CX_COL_FLOAT64) {
    if (x == 1ULL << 63) x = 0ULL;
    x = (x >> 63) ? ~x : x | (1ULL << 63);
  }
  return d.key_desc[k] ? ~x : x;
}

// ORDER BY, first pass: CTA b sorts the present groups of [b * kRun, ...) (or,
// with `rowgrp`, the rows of that range) by their sort words in shared memory
// and leaves them as run b: groups and words at b * kRun, its length in
// lens[b].  A run of 1024 takes 55 network steps, of which the 45 with a
// distance of at most 32 need no CTA barrier (a warp's 32 pairs lie in its own
// 64 slots).  The first two words move with the order: looked up through it,
// a step waited for two dependent shared-memory loads (16.2 -> 14.9 us for 62
// runs).  Runs of 1024 rather than 2048: twice the CTAs (62 for a
// 62,500-group result) and 11 barrier steps fewer; the ranking pass pays 10
// instead of 11 search steps, in twice as many runs.
__global__ void __launch_bounds__(kRun / 2) fin_sort_runs(const unsigned long long* __restrict__ src,
                                                          const unsigned long long* __restrict__ val, const FinDesc d,
                                                          const unsigned* __restrict__ rowgrp, unsigned long long rows,
                                                          unsigned* __restrict__ groups,
                                                          unsigned long long* __restrict__ words,
                                                          unsigned long long cap, unsigned* __restrict__ lens) {
  extern __shared__ unsigned long long s_words[];  // [words][kRun], by slot of arrival
  __shared__ unsigned s_grp[kRun];                 // group by slot of arrival
  __shared__ unsigned s_ord[kRun];                 // the order being sorted: slots
  __shared__ unsigned long long s_first[kRun];     // first and second word, moved along with s_ord
  __shared__ unsigned long long s_second[kRun];
  __shared__ unsigned s_n;
  const unsigned lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  for (unsigned h = 0; h < 2; ++h) {
    const unsigned long long r = (unsigned long long)blockIdx.x * kRun + h * (kRun / 2) + threadIdx.x;
    const unsigned long long g = rowgrp ? (r < rows ? rowgrp[r] : 0ULL) : r;
    const bool p = rowgrp ? r < rows : r < d.groups && present(src, val, d, r);
    const unsigned m = __ballot_sync(0xffffffffu, p);
    unsigned at = 0;
    if (lane == 0 && m) at = atomicAdd(&s_n, __popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
    if (p) {
      s_grp[at] = (unsigned)g;
      int w = 0;
      for (int k = 0; k < d.nkeys; ++k) {
        if (d.nullable[d.key_col[k]]) s_words[(w++) * kRun + at] = sort_word(src, val, d, g, k, true);
        s_words[(w++) * kRun + at] = sort_word(src, val, d, g, k, false);
      }
    }
  }
  __syncthreads();
  const unsigned n = s_n;
  unsigned n2 = 64;
  while (n2 < n) n2 <<= 1;
  for (unsigned i = threadIdx.x; i < n2; i += kRun / 2) {
    s_ord[i] = i < n ? i : kInvalid;
    s_first[i] = i < n ? s_words[i] : ~0ULL;
    s_second[i] = i < n && d.words > 1 ? s_words[kRun + i] : ~0ULL;
  }
  __syncthreads();
  const unsigned t = threadIdx.x;
  for (unsigned k = 2; k <= n2; k <<= 1) {
    for (unsigned j = k >> 1; j > 0; j >>= 1) {
      if (t < n2 / 2) {
        const unsigned i = 2 * t - (t & (j - 1)), x = i + j;
        const unsigned l = s_ord[i], r = s_ord[x];
        const unsigned long long lw = s_first[i], rw = s_first[x], lw2 = s_second[i], rw2 = s_second[x];
        bool rb;  // the right element orders before the left one
        if (r == kInvalid || l == kInvalid) rb = l == kInvalid && r != kInvalid;
        else if (lw != rw) rb = rw < lw;
        else if (lw2 != rw2) rb = rw2 < lw2;
        else {
          rb = s_grp[r] < s_grp[l];
          for (int w = 2; w < d.words; ++w) {
            const unsigned long long a = s_words[w * kRun + l], b = s_words[w * kRun + r];
            if (a != b) { rb = b < a; break; }
          }
        }
        if (((i & k) == 0) == rb) {
          s_ord[i] = r; s_ord[x] = l;
          s_first[i] = rw; s_first[x] = lw;
          s_second[i] = rw2; s_second[x] = lw2;
        }
      }
      // The next step reads slots of other warps only from a distance of 64 on.
      const unsigned next = j > 1 ? j >> 1 : k;
      if (j > 32 || next > 32) __syncthreads();
      else __syncwarp();
    }
  }
  __syncthreads();
  const unsigned long long base = (unsigned long long)blockIdx.x * kRun;
  for (unsigned i = threadIdx.x; i < n; i += kRun / 2) {
    const unsigned o = s_ord[i];
    groups[base + i] = s_grp[o];
    for (int w = 0; w < d.words; ++w) words[w * cap + base + i] = s_words[w * kRun + o];
  }
  if (threadIdx.x == 0) lens[blockIdx.x] = n;
}

// Rows of the sorted run [0, n) at `base` that order before (words, group) e:
// every row of an earlier run has a smaller group, of a later run a larger one.
__device__ __forceinline__ unsigned rows_before(const unsigned long long* __restrict__ words, unsigned long long cap,
                                                int nw, unsigned long long base, unsigned n, unsigned long long e0,
                                                unsigned long long e_at, bool earlier_run) {
  unsigned lo = 0, hi = n;
  if (n) {
    // Runs follow group order, so by a leading group column most of them lie
    // wholly before or after e: their ends settle that without a search
    // (62,500 groups by (key, sum): the pass 14.1 -> 9.4 us).
    const unsigned long long a = words[base], z = words[base + n - 1];
    if (z < e0) return n;
    if (a > e0) return 0;
  }
  while (lo < hi) {
    const unsigned mid = (lo + hi) >> 1;
    const unsigned long long m = words[base + mid];
    bool before = m < e0;
    if (m == e0) {
      before = earlier_run;
      for (int w = 1; w < nw; ++w) {
        const unsigned long long a = words[w * cap + base + mid], b = words[w * cap + e_at];
        if (a != b) { before = a < b; break; }
      }
    }
    if (before) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// ORDER BY, ranking pass: merges groups of kWays runs (stride run_len).  A CTA
// takes 32 neighbouring rows of one run; each of its 8 warps searches an eighth
// of the other runs for all 32 (neighbours' searches share their path, so a
// warp's loads mostly fall on one line), and the sum of the places is the
// row's rank.  Latency-bound: 8 warps of independent searches per 32 rows keep
// 64 runs x 10 steps at 80 dependent loads per thread.  The last pass writes
// the result columns (rank < limit) straight from the group table; an earlier
// one writes the merged run.  Measured, cx_finalize as a whole on a 62,500-group
// result ordered by two columns: 61 us; 1,300 us as a network of 136 global
// compare-exchange launches with its scratch from the default pool.
__global__ void __launch_bounds__(256) fin_merge_runs(const unsigned long long* __restrict__ src,
                                                      const unsigned long long* __restrict__ val, const FinDesc d,
                                                      const unsigned* __restrict__ groups,
                                                      const unsigned long long* __restrict__ words,
                                                      unsigned long long cap, const unsigned* __restrict__ lens,
                                                      unsigned nruns, unsigned long long run_len, unsigned slices,
                                                      unsigned* __restrict__ out_groups,
                                                      unsigned long long* __restrict__ out_words,
                                                      unsigned* __restrict__ out_lens,
                                                      unsigned long long* __restrict__ cols, unsigned long long* vcols,
                                                      unsigned long long row_cap, unsigned long long limit,
                                                      unsigned long long* total) {
  __shared__ unsigned s_len[kWays];
  __shared__ unsigned s_rank[32];
  const unsigned run = blockIdx.x / slices, slice0 = blockIdx.x % slices;
  const unsigned first = run / kWays * kWays;
  const unsigned ways = min(kWays, nruns - first);
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x < kWays) s_len[threadIdx.x] = threadIdx.x < ways ? lens[first + threadIdx.x] : 0u;
  __syncthreads();
  if (slice0 == 0 && run == first && threadIdx.x == 0) {
    unsigned long long sum = 0;
    for (unsigned w = 0; w < ways; ++w) sum += s_len[w];
    if (out_lens) out_lens[run / kWays] = (unsigned)sum;
    else *total = sum;
  }
  const unsigned n = s_len[run - first];
  const unsigned long long vw = (row_cap + 63) / 64;
  for (unsigned long long at0 = (unsigned long long)slice0 * 32; at0 < n; at0 += (unsigned long long)slices * 32) {
    if (threadIdx.x < 32) s_rank[threadIdx.x] = 0u;
    __syncthreads();
    const unsigned long long at = at0 + lane;
    const unsigned long long e_at = (unsigned long long)run * run_len + at;
    if (at < n) {
      const unsigned long long e0 = words[e_at];
      unsigned rank = 0;
      for (unsigned w = warp; w < ways; w += 8)
        rank += first + w == run ? (unsigned)at
                                 : rows_before(words, cap, d.words, (unsigned long long)(first + w) * run_len, s_len[w],
                                               e0, e_at, first + w < run);
      if (rank) atomicAdd(&s_rank[lane], rank);
    }
    __syncthreads();
    if (at < n) {
      const unsigned long long rank = s_rank[lane];
      const unsigned g = groups[e_at];
      if (out_groups) {
        const unsigned long long o = (unsigned long long)first * run_len + rank;
        if (warp == 0) out_groups[o] = g;
        for (int w = (int)warp; w < d.words; w += 8) out_words[w * cap + o] = words[w * cap + e_at];
      } else if (rank < limit) {
        const unsigned long long base = (unsigned long long)g * d.ts;
        for (unsigned c = warp; c < d.cols; c += 8) {
          cols[c * row_cap + rank] = src[base + c];
          const bool valid = d.sparse || !d.nullable[c] || (val && bit_at(val, base + c));
          if (valid) atomicOr(&vcols[c * vw + (rank >> 6)], 1ULL << (rank & 63));
        }
      }
    }
    __syncthreads();
  }
}

// Scratch of cx_finalize comes from one memory pool per device.  The default
// pool gives its memory back to the driver at every synchronisation, so each
// call paid for mapping it again (allocate, free, synchronise: 0.44 ms against
// 5 us from this pool, 4 KB to 8 MB alike); this pool keeps at most kPoolKeep
// bytes past a synchronisation.  Allocations are ordered by their stream, so
// threads and streams may share it; if it cannot be made, the default pool serves.
constexpr unsigned long long kPoolKeep = 32ULL << 20;

cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s) {
  static std::mutex mu;
  static cudaMemPool_t pools[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  cudaMemPool_t pool = nullptr;
  if (dev >= 0 && dev < 64) {
    std::lock_guard<std::mutex> lk(mu);
    if (!pools[dev]) {
      cudaMemPoolProps props{};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      unsigned long long keep = kPoolKeep;
      if (cudaMemPoolCreate(&pools[dev], &props) != cudaSuccess) pools[dev] = nullptr;
      else cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
    }
    pool = pools[dev];
  }
  if (pool && cudaMallocFromPoolAsync(p, bytes, pool, s) == cudaSuccess) return cudaSuccess;
  cudaGetLastError();
  return cudaMallocAsync(p, bytes, s);
}

unsigned grid_for(unsigned long long n) {
  unsigned long long g = (n + 255) / 256;
  if (g > 148ULL * 32) g = 148ULL * 32;
  return g == 0 ? 1 : (unsigned)g;
}

}  // namespace

extern "C" int cx_finalize(const uint64_t* dev_result, const uint64_t* dev_validity, const cx_result_layout* layout,
                           const cx_sort_key* keys, int nkeys, uint64_t limit, uint64_t* dev_columns,
                           uint64_t* dev_col_validity, uint64_t row_cap, uint64_t* rows_out, void* stream_v) {
  if (!dev_result || !layout || !dev_columns || !dev_col_validity || !rows_out || nkeys < 0 || (nkeys > 0 && !keys))
    return ffail(CX_E_INVALID, "cx_finalize: bad argument");
  if (layout->columns == 0 || layout->columns > (uint32_t)kMaxCols || layout->tuple_size < layout->columns ||
      nkeys > kMaxKeys)
    return ffail(CX_E_INVALID, "cx_finalize: 1..32 visible columns within the tuple, at most 8 sort keys");
  if (!layout->sparse && !dev_validity && !layout->scalar)
    return ffail(CX_E_INVALID, "cx_finalize: a dense result needs its validity words");
  FinDesc d{};
  d.groups = layout->scalar ? (layout->groups ? 1ULL : 0ULL) : layout->groups;
  d.ts = layout->tuple_size;
  d.cols = layout->columns;
  d.sparse = layout->sparse;
  d.scalar = layout->scalar;
  for (uint32_t c = 0; c < d.cols; ++c) {
    d.type[c] = layout->column_type ? layout->column_type[c] : (unsigned char)CX_COL_UINT64;
    d.nullable[c] = layout->column_nullable ? layout->column_nullable[c] : 0;
    if (d.type[c] > CX_COL_FLOAT64) return ffail(CX_E_INVALID, "cx_finalize: unknown column type");
  }
  d.nkeys = nkeys;
  for (int k = 0; k < nkeys; ++k) {
    if (keys[k].column < 0 || (uint32_t)keys[k].column >= d.cols) return ffail(CX_E_INVALID, "cx_finalize: sort key outside the columns");
    d.key_col[k] = keys[k].column;
    d.key_desc[k] = keys[k].descending != 0;
  }
  if (row_cap < d.groups) return ffail(CX_E_CAPACITY, "cx_finalize: the row capacity is below the group count");
  if (row_cap > 0xfffffffeULL) return ffail(CX_E_CAPACITY, "cx_finalize: more than 2^32-2 rows");
  cudaStream_t s = (cudaStream_t)stream_v;
  const unsigned long long vw = (row_cap + 63) / 64;
  const unsigned long long* src = (const unsigned long long*)dev_result;
  const unsigned long long* val = (const unsigned long long*)dev_validity;
  unsigned long long* cols = (unsigned long long*)dev_columns;
  unsigned long long* vcols = (unsigned long long*)dev_col_validity;
  d.words = 0;
  bool double_keys = false;
  for (int k = 0; k < nkeys; ++k) {
    d.words += 1 + (d.nullable[d.key_col[k]] ? 1 : 0);
    double_keys = double_keys || d.type[d.key_col[k]] == CX_COL_FLOAT64;
  }
  const size_t sort_smem = (size_t)d.words * kRun * 8;
  cudaError_t e = cudaMemsetAsync(vcols, 0, d.cols * vw * 8, s);
  if (e != cudaSuccess) return fcuda(e, "cudaMemsetAsync");
  if (sort_smem > 16 * 1024 &&
      (e = cudaFuncSetAttribute(fin_sort_runs, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxWords * (int)kRun * 8)) != cudaSuccess)
    return fcuda(e, "cudaFuncSetAttribute");
  const unsigned long long nblocks = (d.groups + kPerBlock - 1) / kPerBlock;
  unsigned long long rows = 0;
  // Sorted runs of `n` rows: scratch of a ranking pass's input or output.
  struct Runs { unsigned* groups; unsigned long long* words; unsigned* lens; unsigned long long cap; };
  auto runs_bytes = [&](unsigned long long nruns) { return nruns * kRun * (8ULL * d.words + 4) + nruns * 4; };
  auto runs_at = [&](char* p, unsigned long long nruns) {
    Runs r;
    r.cap = nruns * kRun;
    r.words = (unsigned long long*)p;
    r.groups = (unsigned*)(p + r.cap * 8ULL * d.words);
    r.lens = r.groups + r.cap;
    return r;
  };
  if (nkeys > 0 && nblocks && !double_keys && d.groups <= kDirectGroups) {
    // Small group tables: every 1024 groups become one sorted run, one ranking
    // pass orders the rows -- two kernels, no row count on the way.
    const unsigned nruns = (unsigned)((d.groups + kRun - 1) / kRun);
    char* tmp = nullptr;
    if ((e = scratch_alloc((void**)&tmp, 8 + runs_bytes(nruns), s)) != cudaSuccess) return fcuda(e, "cudaMallocAsync");
    const Runs r = runs_at(tmp + 8, nruns);
    fin_sort_runs<<<nruns, kRun / 2, sort_smem, s>>>(src, val, d, nullptr, 0, r.groups, r.words, r.cap, r.lens);
    fin_merge_runs<<<nruns * (kRun / 32), 256, 0, s>>>(src, val, d, r.groups, r.words, r.cap, r.lens, nruns, kRun, kRun / 32,
                                                       nullptr, nullptr, nullptr, cols, vcols, row_cap, limit,
                                                       (unsigned long long*)tmp);
    e = cudaMemcpyAsync(&rows, tmp, 8, cudaMemcpyDeviceToHost, s);
    cudaFreeAsync(tmp, s);
    if (e != cudaSuccess) return fcuda(e, "cudaMemcpyAsync");
    if ((e = cudaGetLastError()) != cudaSuccess) return fcuda(e, "cx_finalize launch");
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fcuda(e, "cudaStreamSynchronize");
    *rows_out = rows < limit ? rows : limit;
    return CX_OK;
  }
  if (nblocks) {
    unsigned long long* tmp = nullptr;  // block counts, the total, whether a DOUBLE key holds a NaN
    if ((e = scratch_alloc((void**)&tmp, (nblocks + 2) * 8, s)) != cudaSuccess) return fcuda(e, "cudaMallocAsync");
    unsigned long long* total = tmp + nblocks;
    unsigned long long head[2] = {0, 0};
    auto drop = [&](cudaError_t err, const char* what) { cudaFreeAsync(tmp, s); return fcuda(err, what); };
    if ((e = cudaMemsetAsync(total, 0, 16, s)) != cudaSuccess) return drop(e, "cudaMemsetAsync");
    fin_count<<<(unsigned)nblocks, kBlock, 0, s>>>(src, val, d, tmp, double_keys ? total + 1 : nullptr);
    const bool self_scan = nkeys == 0 && nblocks <= kSelfScan;
    if (!self_scan) fin_scan<<<1, 1024, 0, s>>>(tmp, nblocks, total);
    if (nkeys == 0)
      fin_write<<<(unsigned)nblocks, kBlock, 0, s>>>(src, val, d, tmp, cols, vcols, row_cap, limit, nullptr,
                                                     self_scan ? total : nullptr);
    if ((e = cudaMemcpyAsync(head, total, 16, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return drop(e, "cudaMemcpyAsync");
    if ((e = cudaGetLastError()) != cudaSuccess) return drop(e, "cx_finalize launch");
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return drop(e, "cudaStreamSynchronize");
    rows = head[0];
    if (nkeys > 0 && rows > 0 && head[1]) {
      // A NaN among the keys: the comparator's own network over the rows in group order.
      unsigned long long n = 1;
      while (n < rows) n <<= 1;
      const unsigned long long out = rows < limit ? rows : limit;
      char* net = nullptr;
      if ((e = scratch_alloc((void**)&net, (d.cols * row_cap + d.cols * vw) * 8 + n * 4, s)) != cudaSuccess)
        return drop(e, "cudaMallocAsync");
      unsigned long long* tcols = (unsigned long long*)net;
      unsigned long long* tv = tcols + d.cols * row_cap;
      unsigned* idx = (unsigned*)(tv + d.cols * vw);
      cudaMemsetAsync(tv, 0, d.cols * vw * 8, s);
      fin_write<<<(unsigned)nblocks, kBlock, 0, s>>>(src, val, d, tmp, tcols, tv, row_cap, row_cap, nullptr, nullptr);
      fin_sort_init<<<grid_for(n), 256, 0, s>>>(idx, rows, n);
      for (unsigned long long k = 2; k <= n; k <<= 1)
        for (unsigned long long j = k >> 1; j > 0; j >>= 1)
          fin_sort_step<<<grid_for(n), 256, 0, s>>>(tcols, tv, d, row_cap, idx, n, k, j);
      if (out) fin_gather<<<grid_for(out), 256, 0, s>>>(tcols, tv, d, row_cap, idx, out, cols, vcols);
      cudaFreeAsync(net, s);
    } else if (nkeys > 0 && rows > 0) {
      // Rows in group order, sorted runs of 1024 of them, then ranking passes
      // that merge 64 runs at a time; the last one writes the columns.
      const unsigned long long nruns = (rows + kRun - 1) / kRun;
      const unsigned long long per = (runs_bytes(nruns) + 15) & ~15ULL;
      const bool passes = nruns > kWays;
      char* sorted = nullptr;
      if ((e = scratch_alloc((void**)&sorted, per * (passes ? 2 : 1) + nruns * kRun * 4, s)) != cudaSuccess)
        return drop(e, "cudaMallocAsync");
      Runs in = runs_at(sorted, nruns), outr = runs_at(sorted + (passes ? per : 0), nruns);
      unsigned* rowgrp = (unsigned*)(sorted + per * (passes ? 2 : 1));
      fin_write<<<(unsigned)nblocks, kBlock, 0, s>>>(src, val, d, tmp, nullptr, nullptr, row_cap, 0, rowgrp, nullptr);
      fin_sort_runs<<<(unsigned)nruns, kRun / 2, sort_smem, s>>>(src, val, d, rowgrp, rows, in.groups, in.words, in.cap, in.lens);
      unsigned long long left = nruns, len = kRun;
      while (true) {
        const bool last = left <= kWays;
        // One CTA per 32 rows of a run, at most 2^16 for one run.
        const unsigned long long slices = len / 32 < 65536 / left + 1 ? len / 32 : 65536 / left + 1;
        fin_merge_runs<<<(unsigned)(left * slices), 256, 0, s>>>(
            src, val, d, in.groups, in.words, in.cap, in.lens, (unsigned)left, len, (unsigned)slices,
            last ? nullptr : outr.groups, last ? nullptr : outr.words, last ? nullptr : outr.lens, cols, vcols, row_cap,
            limit, total);
        if (last) break;
        Runs t = in;
        in = outr;
        outr = t;
        left = (left + kWays - 1) / kWays;
        len *= kWays;
      }
      cudaFreeAsync(sorted, s);
    }
    cudaFreeAsync(tmp, s);
  }
  const unsigned long long out = rows < limit ? rows : limit;
  if ((e = cudaGetLastError()) != cudaSuccess) return fcuda(e, "cx_finalize launch");
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return fcuda(e, "cudaStreamSynchronize");
  *rows_out = out;
  return CX_OK;
}
