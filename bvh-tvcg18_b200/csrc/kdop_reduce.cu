// kdop_reduce.cu -- contact point reduction on the device.
//
// Reference: the fourth phase of prox::collision_detection
// (SIMULATION/PROX/PROX/include/prox_collision_detection.h:341-350):
// std::sort of the contact points by ContactPoint::operator<
// (prox_contact_point.h:135-194: body i, body j, p.y, p.x, p.z, n.y, n.x, n.z,
// depth, each compared by float `<`), then std::unique with
// ContactPoint::operator== (:91-133: same bodies and every component with
// |new - kept| not above working_precision<float>() = 10 FLT_EPSILON,
// FOUNDATION/TINY/TINY/include/tiny_precision.h:21-24), which keeps a row
// only when it differs from the last row kept.
//
// Here: one stable radix sort by (body i, body j, p.y), whose width follows
// from the bodies' numbers (50 bits for 512 bodies), then the rows that tie in
// it -- runs of equal keys -- are ranked among themselves by the other six
// fields, a thread per row counting the run's rows before its own.  The rows of
// runs longer than kRankMax, and those that tie in (p.x, p.z) with more than
// kTiesMax, are ordered by three more stable radix sorts of those rows alone,
// over the digits that vary in them, and a fourth by run.  (Sorting all rows by all nine fields, five
// 64-bit sorts of up to eight passes each, moved every row's key 32 times: of
// the 3.6 M rows of 256 touching pairs 40 % are in runs of one or two rows and
// 17 % in runs of more than 32, the longest 371.)  Floats are mapped to
// integers that order like float `<`, -0 folded onto +0.  Many rows alike, as flat
// faces that rest on each other give (700,001 rows, five sorts of all of them ->
// now): runs of 500 duplicates 969 -> 881 us, of 500 points eight times each 990
// -> 917, runs of 1,000 duplicates 1,196 -> 833, one of 20,000 in 20,000 4,768 ->
// 4,258.
//
// The unique is sequential by definition (a row is compared with the last row
// kept, not with its predecessor, and the tolerance is not transitive), but it
// splits into independent segments: a row whose p.y exceeds its predecessor's
// by more than the tolerance, or whose bodies differ, can equal no earlier row
// (rounded subtraction is monotonic, so every earlier p.y is further away).
// Within a run of equal p.y that itself starts a segment the same holds for a
// gap in p.x, by which such a run is sorted.  The thread of a segment's first
// row walks it; a one-pass scan of the keep flags compacts the rows.
#include <algorithm>

#include "kdop_device.cuh"
#include "kdop_internal.h"
#include "kdop_sort.cuh"

namespace kdop {

namespace {

constexpr float kEps = 1.19209290e-07f * 10.0f;  // working_precision<float>()
constexpr uint32_t kRankMax = 512;               // longest run ranked row by row
constexpr uint32_t kTiesMax = 32;                // most rows of one (p.x, p.z) in it that are

// Integer image of a float that orders like float `<` (NaN aside); -0 and +0
// map to the same value.
__device__ __forceinline__ uint32_t ord_key(float f) {
  uint32_t u = __float_as_uint(f);
  if ((u << 1) == 0u) u = 0u;
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ uint64_t two_keys(float hi, float lo) { return ((uint64_t)ord_key(hi) << 32) | ord_key(lo); }

// One row in registers: p, n.x | n.y, n.z, depth, cand.
struct Row {
  float4 a, b;
};
__device__ __forceinline__ Row load_row(const kdop_contact* rows, int64_t r) {
  const float4* p = reinterpret_cast<const float4*>(rows) + 2 * r;
  return Row{p[0], p[1]};
}

// (body i, body j, p.y): the first sort, `bj` bits for body j (body_bits = 0:
// p.y alone).
struct PointGen {
  const kdop_contact* rows;
  const uint2* bodies;
  int bj;
  bool with_bodies;
  __device__ uint64_t key(int64_t i) const {
    const uint64_t y = ord_key(rows[i].p[1]);
    if (!with_bodies) return y;
    const uint2 b = bodies[i];
    return ((((uint64_t)b.x << bj) | b.y) << 32) | y;
  }
  __device__ uint32_t val(int64_t i) const { return (uint32_t)i; }
};
// (body i, body j) after p.y, where both do not fit one key.
struct BodyGen {
  const uint2* bodies;
  const uint32_t* perm;
  int64_t n;
  __device__ uint64_t key(int64_t i) const {
    const uint2 b = bodies[bounded(perm[i], n)];
    return ((uint64_t)b.x << 32) | b.y;
  }
  __device__ uint32_t val(int64_t i) const { return perm[i]; }
};
// Field pairs of a row, the most significant last.
__device__ __forceinline__ uint64_t field_pair(const kdop_contact& c, int pass) {
  return pass == 0 ? two_keys(c.n[2], c.depth) : pass == 1 ? two_keys(c.n[1], c.n[0]) : two_keys(c.p[0], c.p[2]);
}
// Field pairs of the rows still to be ordered, least significant first, then the
// run.  Values are places.
struct LongGen {
  const kdop_contact* rows;
  const uint32_t* placed;  // row at a place so far
  const uint32_t* at;      // places to sort
  const uint32_t* run;     // run of a place
  int pass;
  int64_t n;
  __device__ uint64_t key(int64_t i) const {
    const uint32_t k = bounded(at[i], n);
    return pass == 3 ? run[k] : field_pair(rows[bounded(placed[k], n)], pass);
  }
  __device__ uint32_t val(int64_t i) const { return at[i]; }
};

__global__ void red_max_kernel(const uint2* __restrict__ bodies, int64_t n, unsigned* most) {
  unsigned x = 0, y = 0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const uint2 b = bodies[i];
    x = max(x, b.x);
    y = max(y, b.y);
  }
  x = __reduce_max_sync(0xffffffffu, x);
  y = __reduce_max_sync(0xffffffffu, y);
  if ((threadIdx.x & 31) == 0) {
    atomicMax(most, x);
    atomicMax(most + 1, y);
  }
}

struct ReduceArgs {
  const kdop_contact* rows;
  const uint2* bodies;
  int64_t n;
  const uint32_t* perm;   // rows in the first sort's order
  uint64_t* next;         // (p.x, p.z) of the rows in that order
  uint32_t* run;          // run of a sorted position
  uint32_t* starts;       // first position of a run; starts[runs] = n
  uint32_t* order;        // rows in full order
  Row* sorted;            // the same rows, copied
  uint32_t* keep;
  uint32_t* longs;        // places whose rows the rank kernel leaves to the sorts
  kdop_contact* out;
  uint2* out_bodies;
  int ordered;            // every row is at its place
  unsigned* head;         // ReduceHead words
  WaitLimit lim;
  unsigned long long* words_run;
  unsigned long long* words_keep;
};
// Counters of a reduction, one device block read back as a whole.
// H_BITS: of each field pair, bits set and bits clear in a row still to be
// ordered (64-bit words).
enum { H_ERR, H_TICKET_RUN, H_TICKET_KEEP, H_LONG, H_KEPT, H_MOST_I, H_MOST_J, H_BITS = 8, H_WORDS = H_BITS + 12 };

constexpr int RD_ITEMS = 4, RD_TILE = 256 * RD_ITEMS;

// Runs of equal (bodies, p.y): a scan of their first rows.
__global__ void __launch_bounds__(256) red_runs_kernel(ReduceArgs a) {
  __shared__ unsigned s_tile;
  if (threadIdx.x == 0) s_tile = atomicAdd(a.head + H_TICKET_RUN, 1u);
  __syncthreads();
  const unsigned tile = s_tile;
  const int64_t base = (int64_t)tile * RD_TILE + (int64_t)threadIdx.x * RD_ITEMS;
  uint32_t y_prev = 0;
  uint2 b_prev = make_uint2(0u, 0u);
  if (base > 0 && base <= a.n) {
    const uint32_t r = bounded(a.perm[base - 1], a.n);
    y_prev = ord_key(a.rows[r].p[1]);
    b_prev = a.bodies[r];
  }
  uint32_t first = 0, sum = 0;  // bit j: item j starts a run
#pragma unroll
  for (int j = 0; j < RD_ITEMS; ++j) {
    const int64_t k = base + j;
    if (k >= a.n) continue;
    const uint32_t r = bounded(a.perm[k], a.n);
    const float4 p = reinterpret_cast<const float4*>(a.rows)[2 * (int64_t)r];
    const uint32_t y = ord_key(p.y);
    const uint2 b = a.bodies[r];
    a.next[k] = two_keys(p.x, p.z);
    if (k == 0 || y != y_prev || b.x != b_prev.x || b.y != b_prev.y) {
      first |= 1u << j;
      ++sum;
    }
    y_prev = y;
    b_prev = b;
  }
  uint32_t total;
  uint32_t at = block_scan<256, uint32_t>(sum, total);
  at += tile_prefix(a.words_run, tile, total, a.lim);
#pragma unroll
  for (int j = 0; j < RD_ITEMS; ++j) {
    const int64_t k = base + j;
    if (k >= a.n) continue;
    if ((first >> j) & 1u) a.starts[at++] = (uint32_t)k;
    a.run[k] = at - 1;
    if (k == a.n - 1) a.starts[at] = (uint32_t)a.n;
  }
}

// Fields after p of two rows, in the sort's order: -1, 0, 1.
__device__ __forceinline__ int later_fields(const Row& x, const Row& y) {
  const uint64_t n = two_keys(x.b.x, x.a.w), m = two_keys(y.b.x, y.a.w);
  if (n != m) return n < m ? -1 : 1;
  const uint64_t d = two_keys(x.b.y, x.b.z), f = two_keys(y.b.y, y.b.z);
  return d < f ? -1 : d > f ? 1 : 0;
}

// Each row to its place in the full order: the rows of its run before it.  The
// counting reads (p.x, p.z) keys laid out in the first sort's order --
// neighbouring rows are mostly of one run, so a warp's loads fall on the same
// addresses -- and whole rows only where those tie (reading whole rows through
// the permutation took 399 us on 3.6 M rows).
__global__ void __launch_bounds__(256) red_rank_kernel(ReduceArgs a) {
  const int64_t k = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (k >= a.n) return;
  const uint32_t r = bounded(a.perm[k], a.n), g = bounded(a.run[k], a.n);
  const uint32_t s = bounded(a.starts[g], a.n), e = min(a.starts[g + 1], (uint32_t)a.n);
  const Row x = load_row(a.rows, r);
  if (e - s > kRankMax) {
    // ordered by the radix sorts below, until then in the first sort's order
    a.longs[k] = 1u;
    a.head[H_LONG] = 1u;
    a.order[k] = r;
    a.sorted[k] = x;
    return;
  }
  const uint64_t mine = a.next[k];
  uint32_t rank = 0, ties = 0;
#pragma unroll 8
  for (uint32_t j = s; j < e; ++j) {
    const uint64_t key = a.next[j];
    rank += key < mine ? 1u : 0u;
    ties += key == mine ? 1u : 0u;
  }
  const bool many = ties > kTiesMax;
  if (many) {
    // so are rows that tie in (p.x, p.z) with many others
#pragma unroll 8
    for (uint32_t j = s; j < (uint32_t)k; ++j) rank += a.next[j] == mine ? 1u : 0u;
    a.head[H_LONG] = 1u;
  } else if (ties > 1) {
    for (uint32_t j = s; j < e; ++j) {
      if (a.next[j] != mine || j == (uint32_t)k) continue;
      const int c = later_fields(load_row(a.rows, bounded(a.perm[j], a.n)), x);
      rank += (c < 0 || (c == 0 && j < (uint32_t)k)) ? 1u : 0u;  // equal rows keep their order
    }
  }
  const uint32_t at = bounded(s + rank, a.n);
  a.order[at] = r;
  a.sorted[at] = x;
  a.longs[at] = many ? 1u : 0u;
}

// Places left to the sorts in increasing order: at[pos[k]] = k; and which bits of
// their rows' fields vary (rows in one plane have one normal, duplicates nothing
// that differs: most passes of a sort would move nothing).
__global__ void __launch_bounds__(256) red_long_list_kernel(ReduceArgs a, const uint32_t* __restrict__ pos,
                                                            uint32_t* at) {
  unsigned long long set[3] = {0, 0, 0}, clear[3] = {0, 0, 0};
  for (int64_t k = (int64_t)blockIdx.x * 256 + threadIdx.x; k < a.n; k += (int64_t)gridDim.x * 256) {
    if (!a.longs[k]) continue;
    at[pos[k]] = (uint32_t)k;
    const kdop_contact& c = a.rows[bounded(a.order[k], a.n)];
#pragma unroll
    for (int p = 0; p < 3; ++p) {
      const uint64_t x = field_pair(c, p);
      set[p] |= x;
      clear[p] |= ~x;
    }
  }
  unsigned long long* bits = reinterpret_cast<unsigned long long*>(a.head + H_BITS);
#pragma unroll
  for (int p = 0; p < 3; ++p) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      set[p] |= __shfl_xor_sync(0xffffffffu, set[p], o);
      clear[p] |= __shfl_xor_sync(0xffffffffu, clear[p], o);
    }
    if ((threadIdx.x & 31) == 0 && (set[p] | clear[p])) {
      atomicOr(bits + 2 * p, set[p]);
      atomicOr(bits + 2 * p + 1, clear[p]);
    }
  }
}
// The i-th row in sorted order goes to the i-th place.
__global__ void red_long_place_kernel(ReduceArgs a, const uint32_t* __restrict__ placed,
                                      const uint32_t* __restrict__ at, const uint32_t* __restrict__ sorted_at,
                                      int64_t m) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const uint32_t r = bounded(placed[bounded(sorted_at[i], a.n)], a.n);
  a.order[at[i]] = r;
  a.sorted[at[i]] = load_row(a.rows, r);
}

// ContactPoint::operator== between the last kept row and a new one (bodies
// equal within a segment): no component differs by more than eps.  A NaN
// difference is not "more than eps", as in the reference.
__device__ __forceinline__ bool same_point(const Row& k, const Row& c) {
  return !(fabsf(fsub(c.a.y, k.a.y)) > kEps) && !(fabsf(fsub(c.a.x, k.a.x)) > kEps) &&
         !(fabsf(fsub(c.a.z, k.a.z)) > kEps) && !(fabsf(fsub(c.b.x, k.b.x)) > kEps) &&
         !(fabsf(fsub(c.a.w, k.a.w)) > kEps) && !(fabsf(fsub(c.b.y, k.b.y)) > kEps) &&
         !(fabsf(fsub(c.b.z, k.b.z)) > kEps);
}

// Whether the first row of a run can equal no earlier row.
__device__ __forceinline__ bool run_breaks(const ReduceArgs& a, uint32_t s) {
  if (s == 0) return true;
  const uint2 b = a.bodies[bounded(a.order[s], a.n)], q = a.bodies[bounded(a.order[s - 1], a.n)];
  return b.x != q.x || b.y != q.y || fabsf(fsub(a.sorted[s].a.y, a.sorted[s - 1].a.y)) > kEps;
}
// Whether the row at position k starts a segment.
__device__ __forceinline__ bool starts_segment(const ReduceArgs& a, uint32_t k) {
  const uint32_t s = bounded(a.starts[bounded(a.run[k], a.n)], a.n);
  if (s == k || k == 0) return run_breaks(a, k);
  // a gap in p.x inside a run that starts a segment (a NaN at its head would
  // equal any row)
  const float x = a.sorted[k].a.x, p = a.sorted[k - 1].a.x, x0 = a.sorted[s].a.x;
  return fabsf(fsub(x, p)) > kEps && x0 == x0 && run_breaks(a, s);
}

constexpr uint32_t KEEP = 1u, SEGMENT = 2u;  // bits of keep[]

// The kernels from here on run once without the host's knowing whether rows are
// still to be ordered; where some are, the walk and the write leave it to their
// second run.
__device__ __forceinline__ bool too_early(const ReduceArgs& a) { return !a.ordered && a.head[H_LONG]; }

__global__ void __launch_bounds__(256) red_segments_kernel(ReduceArgs a) {
  const int64_t k = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (k < a.n) a.keep[k] = starts_segment(a, (uint32_t)k) ? SEGMENT | KEEP : 0u;
}

// Thread per segment (its first row's): std::unique's walk -- a row is kept
// unless it equals the last row kept.
__global__ void __launch_bounds__(128) red_walk_kernel(ReduceArgs a) {
  const int64_t k = (int64_t)blockIdx.x * 128 + threadIdx.x;
  if (k >= a.n) return;
  const bool early = too_early(a);  // (beside the flag's load, not before it)
  if (!(a.keep[k] & SEGMENT) || early) return;
  if (k + 1 >= a.n || (a.keep[k + 1] & SEGMENT)) return;  // a segment of one row (most): kept
  Row last = a.sorted[k];
  int64_t j = k + 1;
  for (int c = 0; c < 8; ++c, ++j) {
    if (j >= a.n) return;
    const uint32_t f = a.keep[j];
    const Row x = a.sorted[j];
    if (f & SEGMENT) return;
    if (!same_point(last, x)) {
      a.keep[j] = KEEP;
      last = x;
    }
  }
  // a long segment: two rows' loads in flight (more take registers that the
  // short ones' warps go without)
  for (; j < a.n; j += 2) {
    uint32_t f[2];
    Row x[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int64_t at = min(j + q, a.n - 1);
      f[q] = j + q < a.n ? a.keep[at] : SEGMENT;
      x[q] = a.sorted[at];
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      if (f[q] & SEGMENT) return;
      if (!same_point(last, x[q])) {
        a.keep[j + q] = KEEP;
        last = x[q];
      }
    }
  }
}

__global__ void __launch_bounds__(256) red_write_kernel(ReduceArgs a) {
  __shared__ unsigned s_tile;
  if (threadIdx.x == 0) {
    const bool early = too_early(a);
    const unsigned tile = atomicAdd(a.head + H_TICKET_KEEP, 1u);
    s_tile = early ? 0xFFFFFFFFu : tile;
  }
  __syncthreads();
  if (s_tile == 0xFFFFFFFFu) return;
  const unsigned tile = s_tile;
  // consecutive threads hold consecutive rows: one scan step per item
  uint32_t keep[RD_ITEMS], pos[RD_ITEMS], sum = 0;
#pragma unroll
  for (int j = 0; j < RD_ITEMS; ++j) {
    const int64_t k = (int64_t)tile * RD_TILE + j * 256 + threadIdx.x;
    keep[j] = k < a.n ? a.keep[k] & KEEP : 0u;
    uint32_t total;
    pos[j] = sum + block_scan<256, uint32_t>(keep[j], total);
    sum += total;
  }
  const uint32_t excl = tile_prefix(a.words_keep, tile, sum, a.lim);
#pragma unroll
  for (int j = 0; j < RD_ITEMS; ++j) {
    const int64_t k = (int64_t)tile * RD_TILE + j * 256 + threadIdx.x;
    if (k == a.n - 1) a.head[H_KEPT] = excl + sum;
    if (!keep[j]) continue;
    const Row x = a.sorted[k];
    float4* o = reinterpret_cast<float4*>(a.out + excl + pos[j]);
    o[0] = x.a;
    o[1] = x.b;
    if (a.out_bodies) a.out_bodies[excl + pos[j]] = a.bodies[bounded(a.order[k], a.n)];
  }
}

// Bodies (mesh of A, mesh of B) of each contact row of a scene: the row's
// candidate, its pair, the pair's meshes.
__global__ void red_scene_bodies_kernel(const kdop_contact* __restrict__ rows, int64_t n,
                                        const uint32_t* __restrict__ cand_pair, const uint2* __restrict__ pairs,
                                        uint2* bodies) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) bodies[i] = pairs[cand_pair[rows[i].cand]];
}

unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

// Work buffer of a reduction of n rows (256-byte aligned pieces).
struct ReduceWork {
  size_t head, words_run, words_keep, keys, keys_tmp, next, perm, perm_tmp, radix, run, starts, order, sorted, keep, longs,
      long_at, long_vals, scan, total;
  explicit ReduceWork(int64_t n) {
    size_t at = 0;
    auto take = [&](size_t b) {
      size_t o = at;
      at += (b + 255) & ~(size_t)255;
      return o;
    };
    const size_t m = (size_t)std::max<int64_t>(n, 1), tiles = (m + RD_TILE - 1) / RD_TILE;
    head = take(H_WORDS * 4);
    words_run = take(tiles * 8);
    words_keep = take(tiles * 8);
    keys = take(m * 8);
    keys_tmp = take(m * 8);
    next = take(m * 8);
    perm = take(m * 4);
    perm_tmp = take(m * 4);
    radix = take(radix_scratch_words((int64_t)m) * 4);
    run = take(m * 4);
    starts = take((m + 1) * 4);
    order = take(m * 4);
    sorted = take(m * sizeof(Row));
    keep = take(m * 4);
    longs = take(m * 4);
    long_at = take(m * 4);
    long_vals = take(m * 4);
    scan = take(scan_scratch_words((int64_t)m) * 4);
    total = at;
  }
};

size_t reduce_work_bytes(int64_t n) { return ReduceWork(n).total; }

cudaError_t scene_contact_bodies(kdop_scene* s, int64_t n, uint2* bodies) {
  if (n <= 0) return cudaSuccess;
  red_scene_bodies_kernel<<<blocks_for(n, 256), 256, 0, s->ctx->stream>>>(s->contacts, n, s->cand + 2 * s->cand_cap,
                                                                           s->pairs, bodies);
  s->ctx->launches++;
  return cudaGetLastError();
}

// The rows left by the rank kernel: (n.z, depth), (n.y, n.x), (p.x, p.z), run, each
// a stable sort.  The first sort's keys, the half of its values that does not
// hold the order, next[] and keep[] are free here.
static cudaError_t order_long_runs(kdop_ctx* ctx, const ReduceArgs& a, const ReduceWork& L, char* w,
                                   const SortBuffers& first) {
  cudaStream_t st = ctx->stream;
  SortBuffers b{first.keys, first.keys_tmp, first.vals_tmp, reinterpret_cast<uint32_t*>(w + L.long_vals)};
  uint32_t* pos = a.keep;
  uint32_t* at = reinterpret_cast<uint32_t*>(w + L.long_at);
  uint32_t* placed = reinterpret_cast<uint32_t*>(a.next);
  cudaError_t e;
  if ((e = exclusive_scan_u32(a.longs, pos, a.n, reinterpret_cast<uint32_t*>(w + L.scan), st)) != cudaSuccess) return e;
  red_long_list_kernel<<<std::min(blocks_for(a.n, 256), 592u), 256, 0, st>>>(a, pos, at);
  ctx->launches++;
  if ((e = cudaMemcpyAsync(placed, a.order, (size_t)a.n * 4, cudaMemcpyDeviceToDevice, st)) != cudaSuccess) return e;
  uint32_t tail[2];
  unsigned long long bits[6];
  if ((e = cudaMemcpyAsync(&tail[0], pos + a.n - 1, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(&tail[1], a.longs + a.n - 1, 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
  if ((e = cudaMemcpyAsync(bits, a.head + H_BITS, sizeof(bits), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
  const int64_t m = (int64_t)tail[0] + tail[1];
  if (m == 0) return cudaSuccess;
  const uint32_t* from = at;
  for (int pass = 0; pass < 4; ++pass) {
    const uint64_t vary = pass < 3 ? bits[2 * pass] & bits[2 * pass + 1] : ~0ull;
    if (!vary) continue;
    e = radix_sort(ctx, LongGen{a.rows, placed, from, a.run, pass, a.n}, m, pass < 3 ? 64 : bits_of((uint64_t)a.n), b,
                   w + L.radix, a.lim, vary);
    if (e != cudaSuccess) return e;
    from = b.vals;
  }
  red_long_place_kernel<<<blocks_for(m, 256), 256, 0, st>>>(a, placed, at, from, m);
  ctx->launches++;
  return cudaGetLastError();
}

// Reduces n rows (device) with their bodies (device, below n_bodies where that
// is known, else n_bodies = 0); the kept rows go to out (and their bodies to
// out_bodies, may be NULL) in the reduced order; *n_out = rows kept.
// Synchronises.
cudaError_t reduce_contact_rows(kdop_ctx* ctx, const kdop_contact* rows, const uint2* bodies, int64_t n,
                                int64_t n_bodies, void* work, kdop_contact* out, uint2* out_bodies, int64_t* n_out) {
  cudaStream_t st = ctx->stream;
  *n_out = 0;
  if (n <= 0) return cudaSuccess;
  if (n >= ((int64_t)1 << 32) - 1) return cudaErrorInvalidValue;
  ReduceWork L(n);
  char* w = static_cast<char*>(work);
  ReduceArgs a;
  a.rows = rows;
  a.bodies = bodies;
  a.n = n;
  a.next = reinterpret_cast<uint64_t*>(w + L.next);
  a.run = reinterpret_cast<uint32_t*>(w + L.run);
  a.starts = reinterpret_cast<uint32_t*>(w + L.starts);
  a.order = reinterpret_cast<uint32_t*>(w + L.order);
  a.sorted = reinterpret_cast<Row*>(w + L.sorted);
  a.keep = reinterpret_cast<uint32_t*>(w + L.keep);
  a.longs = reinterpret_cast<uint32_t*>(w + L.longs);
  a.out = out;
  a.out_bodies = out_bodies;
  a.head = reinterpret_cast<unsigned*>(w + L.head);
  a.lim = WaitLimit(a.head + H_ERR, ctx->wait_ns);
  a.words_run = reinterpret_cast<unsigned long long*>(w + L.words_run);
  a.words_keep = reinterpret_cast<unsigned long long*>(w + L.words_keep);
  SortBuffers b{reinterpret_cast<uint64_t*>(w + L.keys), reinterpret_cast<uint64_t*>(w + L.keys_tmp),
                reinterpret_cast<uint32_t*>(w + L.perm), reinterpret_cast<uint32_t*>(w + L.perm_tmp)};
  unsigned h[H_WORDS];
  cudaError_t e;
  if ((e = cudaMemsetAsync(w + L.head, 0, L.keys - L.head, st)) != cudaSuccess) return e;
  int bi = bits_of(n_bodies > 0 ? (uint64_t)n_bodies - 1 : 0), bj = bi;
  if (n_bodies <= 0) {
    red_max_kernel<<<(unsigned)std::min<int64_t>((n + 255) / 256, 592), 256, 0, st>>>(bodies, n, a.head + H_MOST_I);
    ctx->launches++;
    if ((e = cudaMemcpyAsync(h, a.head, sizeof(h), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    bi = bits_of(h[H_MOST_I]);
    bj = bits_of(h[H_MOST_J]);
  }
  const bool one = bi + bj <= 32;
  e = radix_sort(ctx, PointGen{rows, bodies, bj, one}, n, 32 + (one ? bi + bj : 0), b, w + L.radix, a.lim);
  if (e == cudaSuccess && !one) e = radix_sort(ctx, BodyGen{bodies, b.vals, n}, n, 32 + bi, b, w + L.radix, a.lim);
  if (e != cudaSuccess) return e;
  a.perm = b.vals;
  const unsigned tiles = blocks_for(n, RD_TILE);
  red_runs_kernel<<<tile_blocks(ctx, STUCK_SCAN, a.head + H_TICKET_RUN, tiles), 256, 0, st>>>(a);
  red_rank_kernel<<<blocks_for(n, 256), 256, 0, st>>>(a);
  ctx->launches += 2;
  // without waiting for the host to learn whether rows are still to be ordered:
  // where there are some, the rest returns at once and runs when they are
  a.ordered = 0;
  for (int round = 0;; ++round) {
    red_segments_kernel<<<blocks_for(n, 256), 256, 0, st>>>(a);
    red_walk_kernel<<<blocks_for(n, 128), 128, 0, st>>>(a);
    red_write_kernel<<<tile_blocks(ctx, STUCK_SCAN, a.head + H_TICKET_KEEP, tiles), 256, 0, st>>>(a);
    ctx->launches += 3;
    if ((e = cudaMemcpyAsync(h, a.head, sizeof(h), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    if (round || h[H_ERR] || !h[H_LONG]) break;
    if ((e = order_long_runs(ctx, a, L, w, b)) != cudaSuccess) return e;
    a.ordered = 1;
    if ((e = cudaMemsetAsync(a.head + H_TICKET_KEEP, 0, 4, st)) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(a.words_keep, 0, L.keys - L.words_keep, st)) != cudaSuccess) return e;
  }
  if (h[H_ERR]) return cudaErrorLaunchTimeout;
  *n_out = h[H_KEPT];
  return cudaGetLastError();
}

}  // namespace kdop
