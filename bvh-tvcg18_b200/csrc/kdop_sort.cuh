// kdop_sort.cuh -- stable device radix sort with generated keys, and one-pass
// scans, as templates the kernels of other files instantiate.
//
// A sort is least-significant-digit first over 8-bit digits of 64-bit keys
// with 32-bit values.  The caller states how many low bits of the keys vary
// (known on the host from the sizes at hand), so no key bits are read back and
// only ceil(bits / 8) passes run.
//   * One kernel writes the keys (a functor: no separate key pass) and counts
//     every digit of every pass.
//   * One kernel per pass does the rest: a block takes a tile off a ticket
//     counter, ranks its keys with __match_any_sync in input order, publishes
//     its digit counts and sums those of the tiles before it by looking back
//     at what they published (their counts, or their sums where already
//     known), and writes the keys in digit order through shared memory, so
//     that a warp's stores fall on consecutive addresses.  Tiles come off the
//     ticket in order, so a block waits only for blocks already running; the
//     wait is bounded all the same (WaitLimit).  A block whose wait gave up
//     goes on with the counts it has: places stay within the output, but not
//     every place is written.  So whatever reads the output as indices bounds
//     them (a minimum costs nothing beside the load it guards; a look at the
//     error word first took 7 of the 340 us of a reduction of 700,001 rows), and
//     the host reports the error.
//   * Up to kSmallSort keys are generated and sorted by one block in shared
//     memory, in one launch.
// Bound: latency below about 1 M keys (a launch per pass), memory above.  The
// form it replaced took four launches a pass (histogram, scan of the tiles'
// counts, block-sum add, scatter) plus a reduction and a read-back of the
// varying bits per sort: 700,001 contact rows took 1.12 ms in 32 passes.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "kdop_device.cuh"
#include "kdop_sort.h"

namespace kdop {

constexpr int kSortMaxPasses = 8;
constexpr int kSmallSort = 8192;           // keys one block sorts in shared memory

__device__ __forceinline__ unsigned sort_digit(uint64_t key, int shift, unsigned mask) {
  return (unsigned)(key >> shift) & mask;
}

// ---- bounded waits --------------------------------------------------------------
// A wait ends after a time, or as soon as another one of the same error word gave
// up: a launch whose waits fail takes that time once, not once per word.
struct WaitLimit {
  unsigned* err = nullptr;  // device word that gets DEV_ERR_TIMEOUT
  uint32_t ticks = 0;       // of 1,024 ns
  WaitLimit() = default;
  WaitLimit(unsigned* e, long long ns) : err(e), ticks((uint32_t)std::min<long long>(ns >> 10, 1ll << 31)) {}
};
__device__ __forceinline__ bool gave_up(const unsigned* err) {
  return (*(const volatile unsigned*)err & (unsigned)DEV_ERR_TIMEOUT) != 0u;
}

// ---- published tile words -----------------------------------------------------
// value | (1: the tile's own count, 2: the sum up to and with it) << 32 |
// epoch << 34; a word of another epoch is not there yet.
__device__ __forceinline__ void publish(unsigned long long* w, uint32_t v, unsigned flag, unsigned epoch) {
  *(volatile unsigned long long*)w =
      (unsigned long long)v | ((unsigned long long)flag << 32) | ((unsigned long long)epoch << 34);
}
// Whether a wait is to end: its clock (0: not begun yet) for the next look, 0 when
// it is over.  Out of line, so that the polls stay a load and a compare (inlined,
// a pass of the sort took 0.7 us more).
static __device__ __noinline__ uint32_t wait_clock(WaitLimit lim, uint32_t t0) {
  if (gave_up(lim.err)) return 0u;
  const uint32_t now = (uint32_t)(global_ns() >> 10) | 1u;
  if (!t0) return now;
  if (now - t0 <= lim.ticks) return t0;
  atomicOr(lim.err, (unsigned)DEV_ERR_TIMEOUT);
  return 0u;
}
// Waits for the word (bounded); its flag, and its value in v.
__device__ __forceinline__ unsigned await_word(const unsigned long long* w, unsigned epoch, uint32_t& v,
                                               WaitLimit lim) {
  uint32_t t0 = 0;
  do {
    for (int it = 0; it < 256; ++it) {
      const unsigned long long x = *(const volatile unsigned long long*)w;
      if ((unsigned)(x >> 34) == epoch) {
        v = (uint32_t)x;
        return (unsigned)(x >> 32) & 3u;
      }
    }
    t0 = wait_clock(lim, t0);
  } while (t0);
  v = 0;
  return 2u;
}
// An index out of a sorted or scanned buffer of numbers below n.
__device__ __forceinline__ uint32_t bounded(uint32_t i, int64_t n) { return min(i, (uint32_t)n - 1u); }

// Exclusive prefix of a block's total over the blocks before it (tiles in
// ticket order); called by the whole block, the result in every thread.
// words: one per tile, zeroed before the launch.
__device__ __forceinline__ uint32_t tile_prefix(unsigned long long* words, unsigned tile, uint32_t total,
                                                WaitLimit lim) {
  __shared__ uint32_t s_excl;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    if (lane == 0) publish(words + tile, total, tile == 0 ? 2u : 1u, 1u);
    uint32_t excl = 0;
    for (int64_t at = (int64_t)tile - 1; at >= 0; at -= 32) {
      // 32 tiles at once, the nearest on lane 0
      uint32_t v = 0;
      unsigned flag = 2u;
      if (at - lane >= 0) flag = await_word(words + (at - lane), 1u, v, lim);
      const unsigned sums = __ballot_sync(0xffffffffu, flag == 2u);
      const int last = sums ? __ffs(sums) - 1 : 31;  // nearest tile whose sum is known
      uint32_t x = lane <= last ? v : 0u;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      excl += x;
      if (sums) break;
    }
    if (lane == 0) {
      if (tile) publish(words + tile, excl + total, 2u, 1u);
      s_excl = excl;
    }
  }
  __syncthreads();
  return s_excl;
}

// Exclusive scan of one value per thread over a block of THREADS threads; the
// block's total in `total`.
template <int THREADS, typename T>
__device__ __forceinline__ T block_scan(T v, T& total) {
  __shared__ T ws[THREADS / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  T incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) ws[w] = incl;
  __syncthreads();
  if (w == 0) {
    T s = lane < THREADS / 32 ? ws[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < THREADS / 32) ws[lane] = s;
  }
  __syncthreads();
  const T base = w ? ws[w - 1] : T(0);
  total = ws[THREADS / 32 - 1];
  __syncthreads();  // ws is free again
  return base + incl - v;
}

// ---- sort -----------------------------------------------------------------------
// Scratch: digit counts of all passes, tickets, published words.
struct SortScratch {
  uint32_t* hist;               // kSortMaxPasses * 256
  uint32_t* ticket;             // kSortMaxPasses
  unsigned long long* words;    // tiles * 256
  static constexpr size_t kHead = (size_t)kSortMaxPasses * 256 * 4 + 256;
  explicit SortScratch(void* p) {
    char* c = static_cast<char*>(p);
    hist = reinterpret_cast<uint32_t*>(c);
    ticket = hist + kSortMaxPasses * 256;
    words = reinterpret_cast<unsigned long long*>(c + kHead);
  }
};

// Keys (and values) of every item and, for the passes over `bits` bits, the
// digit counts.  A digit that a whole warp shares (the high bits, mostly) is
// counted by one lane.
template <class Gen>
__global__ void __launch_bounds__(256) sort_keys_kernel(Gen gen, int64_t n, int bits, uint64_t* keys, uint32_t* vals,
                                                        uint32_t* hist) {
  __shared__ uint32_t h[kSortMaxPasses][256];
  const int passes = (bits + 7) / 8;
  for (int i = threadIdx.x; i < kSortMaxPasses * 256; i += 256) (&h[0][0])[i] = 0;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * 256;
  for (int64_t i0 = (int64_t)blockIdx.x * 256; i0 < n; i0 += stride) {
    const int64_t i = i0 + threadIdx.x;
    const bool ok = i < n;
    uint64_t k = 0;
    if (ok) {
      k = gen.key(i);
      keys[i] = k;
      vals[i] = gen.val(i);
    }
    const bool full = __all_sync(0xffffffffu, ok);
    for (int p = 0; p < passes; ++p) {
      const unsigned d = sort_digit(k, 8 * p, 255u);
      if (full && __all_sync(0xffffffffu, d == __shfl_sync(0xffffffffu, d, 0))) {
        if ((threadIdx.x & 31) == 0) atomicAdd(&h[p][d], 32u);
      } else if (ok) {
        atomicAdd(&h[p][d], 1u);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += 256) {
    const uint32_t c = (&h[0][0])[i];
    if (c) atomicAdd(&hist[i], c);
  }
}

// Up to 1024 * ITEMS keys generated and sorted by one block.
template <int ITEMS>
constexpr size_t small_sort_smem() {
  return (size_t)1024 * ITEMS * 8 + 32 * 257 * 4;
}
template <class Gen, int ITEMS>
__global__ void __launch_bounds__(1024) small_sort_kernel(Gen gen, int n, int bits, uint64_t vary, uint64_t* keys,
                                                         uint32_t* vals) {
  extern __shared__ uint64_t ex[];                                      // 1024 * ITEMS
  uint32_t* wc = reinterpret_cast<uint32_t*>(ex + 1024 * ITEMS);        // [32 warps][256 digits], a row 257 words
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  uint64_t k[ITEMS];
  uint32_t v[ITEMS];
  uint16_t rank[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const int at = w * 32 * ITEMS + r * 32 + lane;
    k[r] = at < n ? gen.key(at) : ~0ull;
    v[r] = at < n ? gen.val(at) : 0u;
  }
  for (int shift = 0; shift < bits; shift += 8) {
    if (((vary >> shift) & 255u) == 0u) continue;
    // the last pass may cover fewer than 8 varying bits: past them all keys
    // agree, and the items past n (all ones) still rank last
#pragma unroll
    for (int j = 0; j < 9; ++j)
      if (threadIdx.x + 1024 * j < 32 * 257) wc[threadIdx.x + 1024 * j] = 0;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      const unsigned d = sort_digit(k[r], shift, 255u);
      const unsigned peers = __match_any_sync(0xffffffffu, d);
      const uint32_t c = wc[w * 257 + d];
      rank[r] = (uint16_t)(c + __popc(peers & lt));
      __syncwarp();
      if ((peers & lt) == 0u) wc[w * 257 + d] = c + __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    // exclusive scan over (digit, warp): a digit's 8 consecutive warps a thread
    uint32_t* mine = wc + (threadIdx.x & 3) * 8 * 257 + (threadIdx.x >> 2);
    uint32_t c[8], sum = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      c[j] = mine[j * 257];
      sum += c[j];
    }
    uint32_t total;
    uint32_t run = block_scan<1024, uint32_t>(sum, total);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      mine[j * 257] = run;
      run += c[j];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
      rank[r] = (uint16_t)(rank[r] + wc[w * 257 + sort_digit(k[r], shift, 255u)]);
      ex[rank[r]] = k[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) k[r] = ex[w * 32 * ITEMS + r * 32 + lane];
    __syncthreads();
    uint32_t* exv = reinterpret_cast<uint32_t*>(ex);
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) exv[rank[r]] = v[r];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) v[r] = exv[w * 32 * ITEMS + r * 32 + lane];
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const int at = w * 32 * ITEMS + r * 32 + lane;
    if (at < n) {
      keys[at] = k[r];
      vals[at] = v[r];
    }
  }
}

// Keys of radix_sort: two buffers of n keys and values each; `keys` / `vals`
// point at the sorted ones afterwards.
struct SortBuffers {
  uint64_t *keys, *keys_tmp;
  uint32_t *vals, *vals_tmp;
};

// Test hook (kdop_ctx_set_wait_limit): the kinds of wait that a block nobody
// runs is to leave without an end.
enum : int { STUCK_SORT = 1, STUCK_SCAN = 2 };
// Blocks to launch for `blocks` tiles off `ticket`: all of them, or with the hook
// one less, whose tile (the first) nobody takes.
inline unsigned tile_blocks(const kdop_ctx* ctx, int kind, uint32_t* ticket, unsigned blocks) {
  if (!(ctx->test_stuck & kind) || blocks < 2u) return blocks;
  return cudaMemsetAsync(ticket, 1, 1, ctx->stream) == cudaSuccess ? blocks - 1u : blocks;
}

// One digit pass from b's keys and values to its temporaries (kdop_sort.cu).
cudaError_t launch_sort_pass(const kdop_ctx* ctx, const SortBuffers& b, int64_t n, int shift, const uint32_t* hist,
                             uint32_t* ticket, unsigned long long* words, unsigned epoch, WaitLimit lim);

// Stable ascending sort of the items 0 .. n-1 by gen.key(i), of which the low
// `bits` bits vary (the others are equal in all keys; of those, digits without a
// bit of `vary`, where the caller knows it, take no pass), n < 2^32; the values
// are gen.val(i).  gen may read b.vals at i (it is written at i only).
// scratch: radix_scratch_words(n) words, 8-byte aligned.  *lim.err gets
// DEV_ERR_TIMEOUT when a bounded wait gave up (some of the sorted keys and values
// are then whatever lay there); the caller clears and reads it.  On the
// context's stream.
template <class Gen>
cudaError_t radix_sort(kdop_ctx* ctx, const Gen& gen, int64_t n, int bits, SortBuffers& b, void* scratch,
                       WaitLimit lim, uint64_t vary = ~0ull) {
  if (n <= 0) return cudaSuccess;
  cudaStream_t st = ctx->stream;
  long long& launches = ctx->launches;
  cudaError_t e;
  if (n <= kSmallSort) {
    if (n <= 1024) {
      small_sort_kernel<Gen, 1><<<1, 1024, small_sort_smem<1>(), st>>>(gen, (int)n, bits, vary, b.keys, b.vals);
    } else if (n <= 4096) {
      e = cudaFuncSetAttribute(small_sort_kernel<Gen, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)small_sort_smem<4>());
      if (e != cudaSuccess) return e;
      small_sort_kernel<Gen, 4><<<1, 1024, small_sort_smem<4>(), st>>>(gen, (int)n, bits, vary, b.keys, b.vals);
    } else {
      e = cudaFuncSetAttribute(small_sort_kernel<Gen, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)small_sort_smem<8>());
      if (e != cudaSuccess) return e;
      small_sort_kernel<Gen, 8><<<1, 1024, small_sort_smem<8>(), st>>>(gen, (int)n, bits, vary, b.keys, b.vals);
    }
    launches += 1;
    return cudaGetLastError();
  }
  SortScratch s(scratch);
  const int64_t tiles = (n + kSortTile - 1) / kSortTile;
  if ((e = cudaMemsetAsync(scratch, 0, SortScratch::kHead + (size_t)tiles * 256 * 8, st)) != cudaSuccess) return e;
  sort_keys_kernel<<<(unsigned)std::min<int64_t>((n + 1023) / 1024, 1184), 256, 0, st>>>(gen, n, bits, b.keys, b.vals,
                                                                                        s.hist);
  launches += 1;
  unsigned epoch = 1;
  for (int p = 0; 8 * p < bits; ++p) {
    if (((vary >> (8 * p)) & 255u) == 0u) continue;
    e = launch_sort_pass(ctx, b, n, 8 * p, s.hist + 256 * p, s.ticket + p, s.words, epoch, lim);
    if (e != cudaSuccess) return e;
    launches += 1;
    ++epoch;
    std::swap(b.keys, b.keys_tmp);
    std::swap(b.vals, b.vals_tmp);
  }
  return cudaGetLastError();
}

// Bits that hold the values 0 .. max.
inline int bits_of(uint64_t max) {
  int b = 0;
  while (max) {
    ++b;
    max >>= 1;
  }
  return b;
}

}  // namespace kdop
