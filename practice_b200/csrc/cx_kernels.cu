// cx_kernels.cu -- statically compiled (nvcc, sm_100a) kernels of the runtime:
// sparse-result compaction and the seeded synthetic column generator.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <mutex>
#include <string>

#include "../../include/crystal_b200.h"
#include "cx_internal.h"
#include "cx_rng.h"

namespace {

// Every failure is recorded as the calling thread's cx_last_error().
int cuda_fail(cudaError_t e, const char* what) {
  char buf[512];
  snprintf(buf, sizeof buf, "%s: %s", what, cudaGetErrorString(e));
  return cx_internal::set_error(CX_E_CUDA, buf);
}

int invalid(const char* what) { return cx_internal::set_error(CX_E_INVALID, what); }

constexpr int kCompactBlock = 256;
constexpr int kCompactPerBlock = 2048;  // groups per block
// The write pass of a sparse result is a short dependent chain per block (bits,
// places, a few tuples): small blocks keep twice as many of them in flight
// (4,028 blocks: 20 -> 17 us).
constexpr int kWriteBlock = 128;

constexpr unsigned long long kCompactSelfScan = 2048;  // most blocks whose write pass sums the counts itself

// Presence flags of the block's groups [g0, g0 + n): the tuples are read as one
// stream of words (two per load where the table is 16-byte aligned; g0 * ts is
// even), and a non-zero word marks its group.  A thread per tuple read the same
// bytes in loads of stride 8 * ts, ten lines each for five-word tuples.
template <int B>
__device__ __forceinline__ void compact_flags(const unsigned long long* __restrict__ src, unsigned long long g0,
                                              unsigned n, unsigned ts, unsigned char* s_flag) {
  for (unsigned i = threadIdx.x; i < kCompactPerBlock / 4; i += B) ((unsigned*)s_flag)[i] = 0u;
  __syncthreads();
  const unsigned long long* base = src + g0 * ts;
  const unsigned long long words = (unsigned long long)n * ts;
  const bool narrow = ts <= (1u << 20);  // word numbers of a block fit 32 bits: no 64-bit division
  auto group_of = [&](unsigned long long w) -> unsigned { return narrow ? (unsigned)w / ts : (unsigned)(w / ts); };
  if ((((unsigned long long)src) & 15ULL) == 0ULL) {
    const unsigned long long pairs = words / 2;
    const ulonglong2* v = (const ulonglong2*)base;
    unsigned long long i = threadIdx.x;
    for (; i + 3 * B < pairs; i += 4 * B) {
      ulonglong2 x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) x[k] = __ldcs(v + i + k * B);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const unsigned long long w = 2 * (i + k * B);
        if (x[k].x) s_flag[group_of(w)] = 1;
        if (x[k].y) s_flag[group_of(w + 1)] = 1;
      }
    }
    for (; i < pairs; i += B) {
      const ulonglong2 x = __ldcs(v + i);
      if (x.x) s_flag[group_of(2 * i)] = 1;
      if (x.y) s_flag[group_of(2 * i + 1)] = 1;
    }
    if ((words & 1) && threadIdx.x == 0 && base[words - 1]) s_flag[n - 1] = 1;
  } else {
    for (unsigned long long i = threadIdx.x; i < words; i += B)
      if (base[i]) s_flag[group_of(i)] = 1;
  }
  __syncthreads();
}

// Pass 1: number of present groups (any non-zero slot) per block of groups and,
// where `mask` has room, one presence bit per group, so that pass 3 reads the
// present tuples and not the table again.
__global__ void __launch_bounds__(kCompactBlock)
compact_count(const unsigned long long* __restrict__ src, unsigned long long groups, unsigned ts,
              unsigned long long* __restrict__ block_counts, unsigned* __restrict__ mask) {
  __shared__ __align__(16) unsigned char s_flag[kCompactPerBlock];
  __shared__ unsigned part[kCompactBlock / 32];
  const unsigned long long g0 = (unsigned long long)blockIdx.x * kCompactPerBlock;
  const unsigned n = (unsigned)(groups - g0 < kCompactPerBlock ? groups - g0 : kCompactPerBlock);
  compact_flags<kCompactBlock>(src, g0, n, ts, s_flag);
  unsigned cnt = 0;
  for (unsigned i = threadIdx.x; i < kCompactPerBlock; i += kCompactBlock) {
    const unsigned m = __ballot_sync(0xffffffffu, s_flag[i]);
    if ((threadIdx.x & 31) == 0) {
      cnt += __popc(m);
      if (mask) mask[(g0 + i) >> 5] = m;
    }
  }
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = cnt;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned s = 0;
    for (int w = 0; w < kCompactBlock / 32; ++w) s += part[w];
    block_counts[blockIdx.x] = s;
  }
}

// Pass 2: exclusive prefix over block counts (one block, sequential chunks).
__global__ void __launch_bounds__(1024)
compact_scan(unsigned long long* counts, unsigned long long nblocks, unsigned long long* total) {
  __shared__ unsigned long long carry;
  __shared__ unsigned long long warp_sums[32];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (unsigned long long base = 0; base < nblocks; base += 1024) {
    const unsigned long long i = base + threadIdx.x;
    const unsigned long long v = i < nblocks ? counts[i] : 0ULL;
    unsigned long long x = v;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
      unsigned long long w = warp_sums[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      warp_sums[lane] = w;
    }
    __syncthreads();
    const unsigned long long incl = x + (warp > 0 ? warp_sums[warp - 1] : 0ULL);
    if (i < nblocks) counts[i] = carry + incl - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry += incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

// Pass 3: write present tuples in group order, as one stream of words per
// block.  `offsets`: the blocks' exclusive prefix, or (total non-null) their
// counts, which each block sums up to its own (at most 16 KB from L2, less than
// the launch of a scan).  `mask` null: presence is read from the table again.
__global__ void __launch_bounds__(kWriteBlock)
compact_write(const unsigned long long* __restrict__ src, unsigned long long groups, unsigned ts,
              const unsigned long long* __restrict__ offsets, const unsigned* __restrict__ mask,
              unsigned long long* __restrict__ dst, unsigned long long* total) {
  __shared__ __align__(16) unsigned char s_flag[kCompactPerBlock];
  __shared__ unsigned short s_list[kCompactPerBlock];  // the block's present groups in order
  __shared__ unsigned long long part[kWriteBlock / 32];
  __shared__ unsigned s_before[kCompactPerBlock / 32 + 1];
  const unsigned long long g0 = (unsigned long long)blockIdx.x * kCompactPerBlock;
  const unsigned n = (unsigned)(groups - g0 < kCompactPerBlock ? groups - g0 : kCompactPerBlock);
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned long long sum = 0;
  if (total) {
    for (unsigned b = threadIdx.x; b < blockIdx.x; b += kWriteBlock) sum += offsets[b];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
  }
  if (lane == 0) part[warp] = sum;
  if (!mask) compact_flags<kWriteBlock>(src, g0, n, ts, s_flag);
  constexpr unsigned kWords = kCompactPerBlock / 32;
  for (unsigned w = warp; w < kWords; w += kWriteBlock / 32) {
    const unsigned m = mask ? mask[(g0 >> 5) + w] : __ballot_sync(0xffffffffu, s_flag[w * 32 + lane]);
    if (lane == 0) s_before[w + 1] = __popc(m);
  }
  __syncthreads();
  unsigned long long before = total ? 0ULL : offsets[blockIdx.x];
  if (total)
    for (int w = 0; w < kWriteBlock / 32; ++w) before += part[w];
  if (warp == 0) {
    // Prefix of the 64 word counts: two per lane and a scan over the lanes.
    static_assert(kWords == 64, "two words per lane");
    const unsigned c0 = s_before[2 * lane + 1], c1 = s_before[2 * lane + 2];
    unsigned sum2 = c0 + c1;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, sum2, o);
      if (lane >= (unsigned)o) sum2 += y;
    }
    __syncwarp();
    s_before[2 * lane + 1] = sum2 - c1;
    s_before[2 * lane + 2] = sum2;
    if (lane == 0) s_before[0] = 0;
    if (total && blockIdx.x == gridDim.x - 1 && lane == 31) *total = before + sum2;
  }
  __syncthreads();
  for (unsigned w = warp; w < kWords; w += kWriteBlock / 32) {
    const unsigned m = mask ? mask[(g0 >> 5) + w] : __ballot_sync(0xffffffffu, s_flag[w * 32 + lane]);
    if ((m >> lane) & 1u) s_list[s_before[w] + __popc(m & ((1u << lane) - 1u))] = (unsigned short)(w * 32 + lane);
  }
  __syncthreads();
  const unsigned long long words = (unsigned long long)s_before[kWords] * ts;
  for (unsigned long long i = threadIdx.x; i < words; i += kWriteBlock) {
    const unsigned r = ts <= (1u << 20) ? (unsigned)i / ts : (unsigned)(i / ts);
    dst[before * ts + i] = src[(g0 + s_list[r]) * ts + (i - (unsigned long long)r * ts)];
  }
}

// The three passes with `counts` (a word per block) and, if not null, `mask`
// (kCompactPerBlock bits per block) as scratch.  Measured on 8.25M five-word
// groups with some 40,000 present (330 MB): 76 us with the mask, of which the one
// read of the table takes 51 us at the copy peak; 129 us as a thread per tuple
// reading the table twice (calls enqueued back to back; with a wait after each,
// where the scratch is mapped again, 0.50 against 0.58 ms).
void compact_launch(const uint64_t* src, uint64_t groups, uint32_t ts, uint64_t* dst, uint64_t* dev_count,
                    unsigned long long* counts, unsigned* mask, unsigned long long nblocks, cudaStream_t s) {
  const bool self_scan = nblocks <= kCompactSelfScan;
  unsigned long long* total = (unsigned long long*)dev_count;
  compact_count<<<(unsigned)nblocks, kCompactBlock, 0, s>>>((const unsigned long long*)src, groups, ts, counts, mask);
  if (!self_scan) compact_scan<<<1, 1024, 0, s>>>(counts, nblocks, total);
  compact_write<<<(unsigned)nblocks, kWriteBlock, 0, s>>>((const unsigned long long*)src, groups, ts, counts, mask,
                                                            (unsigned long long*)dst, self_scan ? total : nullptr);
}

__global__ void gen_uniform_kernel(unsigned long long stream, unsigned long long seed, long long lo, unsigned long long span,
                                   unsigned long long row0, unsigned long long rows, int* __restrict__ out) {
  const unsigned long long key = cx_rng_stream_key(seed, stream);
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows;
       i += (unsigned long long)gridDim.x * blockDim.x)
    out[i] = (int)(lo + (long long)cx_rng_below(cx_rng_hash(key, row0 + i), span));
}

__global__ void gen_datekey_kernel(unsigned long long stream, unsigned long long seed, unsigned days,
                                   unsigned long long row0, unsigned long long rows, int* __restrict__ out) {
  const unsigned long long key = cx_rng_stream_key(seed, stream);
  for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < rows;
       i += (unsigned long long)gridDim.x * blockDim.x) {
    const unsigned d = (unsigned)cx_rng_below(cx_rng_hash(key, row0 + i), days);
    out[i] = cx_datekey_of_day(d);
  }
}

__global__ void gen_validity_kernel(unsigned long long stream, unsigned long long seed, unsigned long long rows,
                                    unsigned permille, unsigned long long* __restrict__ out) {
  const unsigned long long key = cx_rng_stream_key(seed, stream);
  const unsigned long long words = (rows + 63) / 64;
  for (unsigned long long w = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; w < words;
       w += (unsigned long long)gridDim.x * blockDim.x) {
    unsigned long long bits = 0;
    for (int b = 0; b < 64; ++b) {
      const unsigned long long r = w * 64 + b;
      if (r >= rows) break;
      const bool is_null = cx_rng_below(cx_rng_hash(key, r), 1000) < permille;
      if (!is_null) bits |= 1ULL << b;
    }
    out[w] = bits;
  }
}

unsigned grid_for(unsigned long long n, unsigned block) {
  unsigned long long g = (n + block - 1) / block;
  if (g > 148ULL * 32) g = 148ULL * 32;
  return g == 0 ? 1 : (unsigned)g;
}

}  // namespace

extern "C" int cx_compact_sparse(const uint64_t* src, uint64_t groups, uint32_t ts, uint64_t* dst, uint64_t* dev_count,
                                 void* stream_v) {
  if (!src || !dst || !dev_count || ts == 0) return invalid("cx_compact_sparse: null buffer or zero tuple size");
  cudaStream_t s = (cudaStream_t)stream_v;
  const unsigned long long nblocks = (groups + kCompactPerBlock - 1) / kCompactPerBlock;
  if (nblocks == 0) {
    cudaError_t e = cudaMemsetAsync(dev_count, 0, 8, s);
    return e == cudaSuccess ? CX_OK : cuda_fail(e, "cudaMemsetAsync");
  }
  unsigned long long* counts = nullptr;
  cudaError_t e = cudaMallocAsync((void**)&counts, nblocks * (8 + kCompactPerBlock / 8), s);
  if (e != cudaSuccess) return cuda_fail(e, "cudaMallocAsync");
  compact_launch(src, groups, ts, dst, dev_count, counts, (unsigned*)(counts + nblocks), nblocks, s);
  e = cudaGetLastError();
  cudaFreeAsync(counts, s);
  return e == cudaSuccess ? CX_OK : cuda_fail(e, "compaction launch");
}

// ------------------------------------------------ no-allocation compaction ---
// Some callers cannot let this library allocate device memory: a serving loop
// that has reserved the whole HBM budget for admitted queries (an allocation
// here could fail or silently break its accounting), and engines whose memory
// guard must see every device byte before a query runs.  For them the block
// counts of the compaction live in this fixed file-scope array instead of a
// cudaMallocAsync buffer.  It holds kNoAllocMaxBlocks counts (128 KiB), so one
// call compacts at most kNoAllocMaxBlocks * kCompactPerBlock group tuples; every
// GPU that loads the library keeps the array until the process exits.
constexpr unsigned long long kNoAllocMaxBlocks = 16384;
static __device__ __align__(256) unsigned long long g_noalloc_block_counts[kNoAllocMaxBlocks];

namespace {
std::mutex g_noalloc_mu;
unsigned long long* g_noalloc_ptr[256] = {};  // last resolved device address of the array, per device ordinal
}  // namespace

extern "C" int cx_compact_sparse_noalloc(const uint64_t* src, uint64_t groups, uint32_t ts, uint64_t* dst,
                                         uint64_t* dev_count, void* stream_v) {
  if (!src || !dst || !dev_count || ts == 0)
    return invalid("cx_compact_sparse_noalloc: null buffer or zero tuple size");
  const unsigned long long nblocks = (groups + kCompactPerBlock - 1) / kCompactPerBlock;
  if (nblocks > kNoAllocMaxBlocks) {
    char buf[256];
    snprintf(buf, sizeof buf, "cx_compact_sparse_noalloc: %llu groups exceed the fixed maximum of %llu groups per call",
             (unsigned long long)groups, kNoAllocMaxBlocks * kCompactPerBlock);
    return cx_internal::set_error(CX_E_CAPACITY, buf);
  }
  cudaStream_t s = (cudaStream_t)stream_v;
  if (nblocks == 0) {
    cudaError_t e = cudaMemsetAsync(dev_count, 0, 8, s);
    return e == cudaSuccess ? CX_OK : cuda_fail(e, "cudaMemsetAsync");
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
  if (dev < 0 || dev >= 256) return invalid("cx_compact_sparse_noalloc: device ordinal out of range");
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  e = cudaStreamIsCapturing(s, &cap);
  if (e != cudaSuccess) return cuda_fail(e, "cudaStreamIsCapturing");
  unsigned long long* counts = nullptr;
  {
    // The host-side symbol is not a device address: resolve the array's
    // address in the current device's context.  Outside stream capture it is
    // resolved on every call, so a context re-created after cudaDeviceReset
    // (or another context made current) gets its own address; inside capture
    // the address resolved by an earlier call on this device is used, so the
    // first call on a device must come before any capture.
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (cap == cudaStreamCaptureStatusNone) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_noalloc_block_counts);
      if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress");
      g_noalloc_ptr[dev] = (unsigned long long*)p;
    } else if (!g_noalloc_ptr[dev]) {
      return cx_internal::set_error(CX_E_INVALID,
                                    "cx_compact_sparse_noalloc: the first call on a device must come before stream capture");
    }
    counts = g_noalloc_ptr[dev];
  }
  // compact_count writes every one of the nblocks counts, so the array needs
  // no clearing between calls.  It has no room for presence bits (4 MiB at the
  // maximum), so the write pass reads the table a second time.
  compact_launch(src, groups, ts, dst, dev_count, counts, nullptr, nblocks, s);
  e = cudaGetLastError();
  return e == cudaSuccess ? CX_OK : cuda_fail(e, "compaction launch");
}

extern "C" int cx_gen_uniform(uint64_t stream, uint64_t seed, int64_t lo, int64_t hi, uint64_t row0, uint64_t rows,
                              int32_t* out, void* cuda_stream) {
  if (!out || hi < lo || lo < INT32_MIN || hi > INT32_MAX) return invalid("cx_gen_uniform: null output or bad range");
  if (rows == 0) return CX_OK;
  gen_uniform_kernel<<<grid_for(rows, 256), 256, 0, (cudaStream_t)cuda_stream>>>(
      stream, seed, lo, (unsigned long long)(hi - lo + 1), row0, rows, out);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CX_OK : cuda_fail(e, "gen_uniform");
}

extern "C" int cx_gen_datekey(uint64_t stream, uint64_t seed, uint32_t days, uint64_t row0, uint64_t rows, int32_t* out,
                              void* cuda_stream) {
  if (!out || days == 0 || days > 36500) return invalid("cx_gen_datekey: null output or bad day count");
  if (rows == 0) return CX_OK;
  gen_datekey_kernel<<<grid_for(rows, 256), 256, 0, (cudaStream_t)cuda_stream>>>(stream, seed, days, row0, rows, out);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CX_OK : cuda_fail(e, "gen_datekey");
}

extern "C" int cx_gen_validity(uint64_t stream, uint64_t seed, uint64_t rows, uint32_t null_permille, uint64_t* out,
                               void* cuda_stream) {
  if (!out || null_permille > 1000) return invalid("cx_gen_validity: null output or permille above 1000");
  if (rows == 0) return CX_OK;
  gen_validity_kernel<<<grid_for((rows + 63) / 64, 256), 256, 0, (cudaStream_t)cuda_stream>>>(
      stream, seed, rows, null_permille, (unsigned long long*)out);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CX_OK : cuda_fail(e, "gen_validity");
}

// ------------------------------------------------- functional dependencies --
// Whether column B of a dimension determines column A (every row with the
// same B value has the same A value): each row claims tab[B - lo_b] for its
// A offset; a second, different offset sets the flag.  `tab` (radix_b ints)
// must hold -1 before the launch; afterwards it maps each B offset that
// occurs to its A offset.
namespace {

__global__ void __launch_bounds__(256)
fd_check(const int* __restrict__ a, const int* __restrict__ b, long long n, int lo_a, int lo_b, unsigned radix_b,
         int* __restrict__ tab, unsigned* __restrict__ flag) {
  for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (long long)gridDim.x * blockDim.x) {
    const unsigned bo = (unsigned)(b[r] - lo_b);
    const int ao = a[r] - lo_a;
    if (bo >= radix_b) { atomicOr(flag, 1u); continue; }
    const int old = atomicCAS(&tab[bo], -1, ao);
    if (old != -1 && old != ao) atomicOr(flag, 1u);
  }
}

}  // namespace

namespace cx_internal {

int fd_check_launch(const int* a, const int* b, long long n, int lo_a, int lo_b, int radix_b, int* tab, unsigned* flag,
                    cudaStream_t s) {
  if (!a || !b || !tab || !flag || n < 0 || radix_b <= 0) return invalid("fd_check: bad argument");
  cudaError_t e = cudaMemsetAsync(tab, 0xFF, (size_t)radix_b * sizeof(int), s);
  if (e != cudaSuccess) return cuda_fail(e, "fd_check: memset");
  if (n == 0) return CX_OK;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const long long blocks = std::min<long long>((n + 255) / 256, (long long)sms * 8);
  fd_check<<<(unsigned)blocks, 256, 0, s>>>(a, b, n, lo_a, lo_b, (unsigned)radix_b, tab, flag);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "fd_check");
  return CX_OK;
}

}  // namespace cx_internal
