// kdop_sort.cu -- exclusive scan, and the reproducible order of a traversal's
// results (the role of the OpenCL back-end's qsort,
// cl/kdop_cl_tandem_traversal.h:1773-1788) by the radix sort of
// kdop_sort.cuh.
#include <algorithm>

#include "kdop_device.cuh"
#include "kdop_sort.cuh"

namespace kdop {

namespace {

constexpr int SC_THREADS = 1024, SC_ITEMS = 4;
constexpr int SC_BLOCK = SC_THREADS * SC_ITEMS;        // 4096 counts per scan block

// One digit pass over tiles of kSortTile keys.  Items past n (last tile) rank
// as digit 255 behind every key and are not written.  Eight keys a thread:
// sixteen took 128 registers, two blocks of 256 threads per SM, and 59 us a
// pass of 3.6 M keys against 50 (tiles of 2,048 to 8,192 keys are within 10 %
// of one another, as are ballots by bit and __match_any_sync, and one or eight
// words in flight in the look-back).
constexpr int SP_THREADS = 512, SP_WARPS = SP_THREADS / 32, SP_ITEMS = (int)kSortTile / SP_THREADS;
constexpr size_t kPassSmem = (size_t)kSortTile * 12 + SP_WARPS * 256 * 4;
__global__ void __launch_bounds__(SP_THREADS, 1280 / SP_THREADS)
    sort_pass_kernel(const uint64_t* __restrict__ kin, const uint32_t* __restrict__ vin, uint64_t* kout,
                     uint32_t* vout, int64_t n, int shift, const uint32_t* __restrict__ hist, uint32_t* ticket,
                     unsigned long long* words, unsigned epoch, WaitLimit lim) {
  constexpr int TILE = (int)kSortTile, ITEMS = SP_ITEMS, WARPS = SP_WARPS;
  extern __shared__ uint64_t ex[];                         // TILE keys in digit order
  uint32_t* exv = reinterpret_cast<uint32_t*>(ex + TILE);  // and their values
  uint32_t(*wc)[256] = reinterpret_cast<uint32_t(*)[256]>(exv + TILE);
  __shared__ uint32_t gbase[256], lofs[256];
  __shared__ unsigned s_tile;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
  const unsigned d0 = threadIdx.x;  // this thread's digit, of the first 256
  const uint32_t all = d0 < 256 ? hist[d0] : 0u;
  for (int j = threadIdx.x; j < WARPS * 256; j += SP_THREADS) (&wc[0][0])[j] = 0;
  __syncthreads();
  const unsigned tile = s_tile;
  const int64_t base = (int64_t)tile * TILE;
  const int valid = (int)min((int64_t)TILE, n - base);
  uint64_t k[ITEMS];
  uint32_t v[ITEMS];
  uint16_t rank[ITEMS];
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const int at = w * 32 * ITEMS + r * 32 + lane;
    k[r] = at < valid ? kin[base + at] : ~0ull;
    v[r] = at < valid ? vin[base + at] : 0u;
  }
  // ranks within the warp, in input order (warp w: 32 * ITEMS consecutive keys)
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const unsigned d = sort_digit(k[r], shift, 255u);
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const uint32_t c = wc[w][d];
    rank[r] = (uint16_t)(c + __popc(peers & lt));
    __syncwarp();
    if ((peers & lt) == 0u) wc[w][d] = c + __popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // digit d0: the warps in order, then the tiles before this one
  uint32_t count = 0;
  if (d0 < 256) {
#pragma unroll
    for (int j = 0; j < WARPS; ++j) {
      const uint32_t c = wc[j][d0];
      wc[j][d0] = count;
      count += c;
    }
    publish(words + (size_t)tile * 256 + d0, count, tile == 0 ? 2u : 1u, epoch);
  }
  unsigned long long total;
  const unsigned long long both = ((unsigned long long)all << 16) | count;  // a tile holds < 2^16 keys
  const unsigned long long before = block_scan<SP_THREADS, unsigned long long>(both, total);
  if (d0 < 256) {
    // the tiles before, from the nearest back to one whose sum is known
    uint32_t excl = 0;
    for (int64_t t = (int64_t)tile - 1; t >= 0; --t) {
      uint32_t c;
      const unsigned flag = await_word(words + (size_t)t * 256 + d0, epoch, c, lim);
      excl += c;
      if (flag == 2u) break;
    }
    if (tile) publish(words + (size_t)tile * 256 + d0, excl + count, 2u, epoch);
    const uint32_t local = (uint32_t)before & 0xFFFFu;
    lofs[d0] = local;
    gbase[d0] = (uint32_t)(before >> 16) + excl - local;
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const unsigned d = sort_digit(k[r], shift, 255u);
    const uint32_t at = lofs[d] + wc[w][d] + rank[r];
    ex[at] = k[r];
    exv[at] = v[r];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ITEMS; ++r) {
    const int at = r * SP_THREADS + threadIdx.x;
    const uint64_t key = ex[at];
    const uint32_t g = gbase[sort_digit(key, shift, 255u)] + (uint32_t)at;
    if (at < valid && (int64_t)g < n) {
      kout[g] = key;
      vout[g] = exv[at];
    }
  }
}

// Exclusive scan of one block of SC_BLOCK counts; block total to sums.
__global__ void __launch_bounds__(SC_THREADS) scan_block_kernel(const uint32_t* in, uint32_t* out,
                                                               int64_t n, uint32_t* sums) {
  __shared__ uint32_t ws[SC_THREADS / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * SC_BLOCK + (int64_t)threadIdx.x * SC_ITEMS;
  uint32_t x[SC_ITEMS], t = 0;
#pragma unroll
  for (int j = 0; j < SC_ITEMS; ++j) {
    x[j] = (base + j < n) ? in[base + j] : 0u;
    t += x[j];
  }
  uint32_t incl = t;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) ws[w] = incl;
  __syncthreads();
  if (w == 0) {
    uint32_t s = ws[lane];
    uint32_t si = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, si, o);
      if (lane >= o) si += y;
    }
    ws[lane] = si - s;
    if (lane == 31 && sums) sums[blockIdx.x] = si;
  }
  __syncthreads();
  uint32_t run = ws[w] + incl - t;
#pragma unroll
  for (int j = 0; j < SC_ITEMS; ++j) {
    if (base + j < n) out[base + j] = run;
    run += x[j];
  }
}

__global__ void scan_add_kernel(uint32_t* out, int64_t n, const uint32_t* __restrict__ block_off) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] += block_off[i / SC_BLOCK];
}

}  // namespace

size_t scan_scratch_words(int64_t n) {
  size_t w = 0;
  while (n > SC_BLOCK) {
    n = (n + SC_BLOCK - 1) / SC_BLOCK;
    w += (size_t)n;
  }
  return w + 1;
}

cudaError_t exclusive_scan_u32(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* scratch, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  int64_t blocks = (n + SC_BLOCK - 1) / SC_BLOCK;
  if (blocks == 1) {
    scan_block_kernel<<<1, SC_THREADS, 0, st>>>(in, out, n, nullptr);
    return cudaGetLastError();
  }
  uint32_t* sums = scratch;
  scan_block_kernel<<<(unsigned)blocks, SC_THREADS, 0, st>>>(in, out, n, sums);
  cudaError_t e = exclusive_scan_u32(sums, sums, blocks, scratch + blocks, st);
  if (e != cudaSuccess) return e;
  scan_add_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, n, sums);
  return cudaGetLastError();
}

cudaError_t launch_sort_pass(const kdop_ctx* ctx, const SortBuffers& b, int64_t n, int shift, const uint32_t* hist,
                             uint32_t* ticket, unsigned long long* words, unsigned epoch, WaitLimit lim) {
  const cudaError_t e =
      cudaFuncSetAttribute(sort_pass_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPassSmem);
  if (e != cudaSuccess) return e;
  const unsigned blocks = tile_blocks(ctx, STUCK_SORT, ticket, (unsigned)((n + kSortTile - 1) / kSortTile));
  sort_pass_kernel<<<blocks, SP_THREADS, kPassSmem, ctx->stream>>>(b.keys, b.vals, b.keys_tmp, b.vals_tmp, n, shift,
                                                                   hist, ticket, words, epoch, lim);
  return cudaGetLastError();
}

size_t radix_scratch_words(int64_t n) {
  const int64_t tiles = (std::max<int64_t>(n, 1) + kSortTile - 1) / kSortTile;
  return SortScratch::kHead / 4 + (size_t)tiles * 512;
}

}  // namespace kdop

// ---- reproducible order of a traversal's results ------------------------------
namespace kdop {
namespace {

// Sort key of a candidate row: (pair, tet of A, tet of B), the tets numbered
// within their meshes (`tb` bits each), so that a scene of 38 M tets in 1,024
// meshes sorts 45 bits instead of 96 and the sorted key alone gives the row
// back.
struct CandGen {
  const uint32_t *cA, *cB, *cP;
  const uint2* pairs;
  const uint32_t* t_off;
  int tb;
  __device__ uint64_t key(int64_t i) const {
    const uint32_t p = cP[i];
    const uint2 m = pairs[p];
    return ((uint64_t)p << (2 * tb)) | ((uint64_t)(cA[i] - t_off[m.x]) << tb) | (cB[i] - t_off[m.y]);
  }
  __device__ uint32_t val(int64_t i) const { return (uint32_t)i; }
};
// The same order in two sorts, least significant first, for keys wider than 64
// bits and for results whose pair list the scene no longer holds: tets by their
// global numbers, then pair indices (also where a replayed graph of the caller's
// may have put another list there).
struct TetGen {
  const uint32_t *cA, *cB;
  int tb;
  __device__ uint64_t key(int64_t i) const { return ((uint64_t)cA[i] << tb) | cB[i]; }
  __device__ uint32_t val(int64_t i) const { return (uint32_t)i; }
};
struct PairGen {
  const uint32_t *cP, *perm;
  int64_t n;
  __device__ uint64_t key(int64_t i) const { return cP[bounded(perm[i], n)]; }
  __device__ uint32_t val(int64_t i) const { return perm[i]; }
};

struct ApplyArgs {
  int64_t n;
  const uint64_t* keys;  // sorted keys, or NULL: rows are gathered by perm
  const uint32_t* perm;
  CandGen c;
  int64_t n_pairs;
  uint32_t *oA, *oB, *oP;
  const int4* rec;       // NULL without contacts
  int4* rec_out;
  uint32_t* src;         // first contact row of a sorted candidate before the sort
  uint32_t* ticket;
  unsigned long long* words;
  WaitLimit lim;
};

constexpr int AP_ITEMS = 4, AP_TILE = 256 * AP_ITEMS;

// Candidate rows in sorted order and, with contacts, their records with the
// rows' new places (a scan of the contact counts in the same pass).
__global__ void __launch_bounds__(256) sort_apply_kernel(ApplyArgs a) {
  __shared__ unsigned s_tile;
  if (threadIdx.x == 0) s_tile = a.rec ? atomicAdd(a.ticket, 1u) : blockIdx.x;
  __syncthreads();
  const unsigned tile = s_tile;
  const int64_t base = (int64_t)tile * AP_TILE + (int64_t)threadIdx.x * AP_ITEMS;
  int4 r[AP_ITEMS];
  uint32_t sum = 0;
#pragma unroll
  for (int j = 0; j < AP_ITEMS; ++j) {
    const int64_t k = base + j;
    r[j] = make_int4(-1, -1, 0, 0);
    if (k >= a.n) continue;
    if (a.keys) {
      const uint64_t key = a.keys[k];
      const uint32_t p = bounded((uint32_t)(key >> (2 * a.c.tb)), a.n_pairs), m = (1u << a.c.tb) - 1u;
      const uint2 mp = a.c.pairs[p];
      a.oA[k] = a.c.t_off[mp.x] + ((uint32_t)(key >> a.c.tb) & m);
      a.oB[k] = a.c.t_off[mp.y] + ((uint32_t)key & m);
      a.oP[k] = p;
    } else {
      const uint32_t o = bounded(a.perm[k], a.n);
      a.oA[k] = a.c.cA[o];
      a.oB[k] = a.c.cB[o];
      a.oP[k] = a.c.cP[o];
    }
    if (a.rec) {
      r[j] = a.rec[bounded(a.perm[k], a.n)];
      sum += (uint32_t)max(r[j].z, 0);
    }
  }
  if (!a.rec) return;
  uint32_t total;
  uint32_t run = block_scan<256, uint32_t>(sum, total);
  run += tile_prefix(a.words, tile, total, a.lim);
#pragma unroll
  for (int j = 0; j < AP_ITEMS; ++j) {
    const int64_t k = base + j;
    if (k >= a.n) continue;
    a.src[k] = (uint32_t)r[j].w;
    if (r[j].z > 0) {
      r[j].w = (int)run;
      run += (uint32_t)r[j].z;
    }
    a.rec_out[k] = r[j];
  }
}

__global__ void __launch_bounds__(256) candidate_rows_kernel(const uint32_t* __restrict__ cA,
                                                             const uint32_t* __restrict__ cB,
                                                             const uint32_t* __restrict__ cP,
                                                             const uint2* __restrict__ pairs, uint32_t n_pairs,
                                                             const uint32_t* __restrict__ t_off, int64_t n,
                                                             uint32_t* rows) {
  // thread per row, then the block's 768 words in order
  __shared__ uint32_t s[768];
  const int64_t base = (int64_t)blockIdx.x * 256, i = base + threadIdx.x;
  if (i < n) {
    const uint32_t p = cP[i];
    const uint2 m = p < n_pairs ? pairs[p] : make_uint2(0u, 0u);
    s[3 * threadIdx.x] = p;
    s[3 * threadIdx.x + 1] = cA[i] - t_off[m.x];
    s[3 * threadIdx.x + 2] = cB[i] - t_off[m.y];
  }
  __syncthreads();
  const int words = 3 * (int)min((int64_t)256, n - base);
  for (int k = threadIdx.x; k < words; k += 256) rows[3 * base + k] = s[k];
}

// Contact rows of sorted candidate k to rows r.w ..: eight lanes a candidate,
// 16 bytes a lane.  Records a timed-out sort left incomplete may name rows past
// the n_rows there are: nothing is copied for them.
__global__ void __launch_bounds__(256) contact_gather_kernel(int64_t n, const int4* __restrict__ rec,
                                                             const uint32_t* __restrict__ src,
                                                             const float4* __restrict__ rows, float4* rows_out,
                                                             int64_t n_rows) {
  const int64_t k = ((int64_t)blockIdx.x * 256 + threadIdx.x) >> 3;
  if (k >= n) return;
  const int4 r = rec[k];
  if (r.z <= 0) return;
  const uint32_t first = src[k];
  if ((int64_t)max(first, (uint32_t)r.w) + r.z > n_rows) return;
  const float4* from = rows + 2 * (size_t)first;
  float4* to = rows_out + 2 * (size_t)(uint32_t)r.w;
  for (int c = threadIdx.x & 7; c < 2 * r.z; c += 8) {
    float4 x = from[c];
    if (c & 1) x.w = __uint_as_float((uint32_t)k);  // the row's candidate
    to[c] = x;
  }
}

}  // namespace

cudaError_t launch_candidate_rows(kdop_scene* s, int64_t first, int64_t n, uint32_t* rows) {
  const uint32_t* c = s->cand + first;
  // the results' pair indices run over the list on the device, which is as long;
  // the library knows no more than its room when a replayed graph of the
  // caller's may have put another one there
  const int64_t n_pairs = s->ctl_replayed ? s->pairs_cap : s->result_pairs;
  candidate_rows_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s->ctx->stream>>>(
      c, c + s->cand_cap, c + 2 * s->cand_cap, s->pairs, (uint32_t)n_pairs, s->t_off_dev, n, rows);
  s->ctx->launches++;
  return cudaGetLastError();
}

// Work buffer of sort_results, every region 256-byte aligned.
struct SortWork {
  size_t head, words, keys, keys_tmp, vals, vals_tmp, cand_out, src, rec_out, rows_out, scratch, total;
  int64_t tiles;
  SortWork(int64_t n, int64_t n_contacts) {
    size_t at = 0;
    auto take = [&](size_t bytes) {
      size_t o = at;
      at += (bytes + 255) & ~(size_t)255;
      return o;
    };
    tiles = (n + AP_TILE - 1) / AP_TILE;
    head = take(256);
    words = take((size_t)tiles * 8);
    keys = take((size_t)n * 8);
    keys_tmp = take((size_t)n * 8);
    vals = take((size_t)n * 4);
    vals_tmp = take((size_t)n * 4);
    cand_out = take((size_t)n * 12);
    src = take((size_t)n * 4);
    rec_out = take((size_t)n * 16);
    rows_out = take((size_t)std::max<int64_t>(n_contacts, 1) * sizeof(kdop_contact));
    scratch = take(radix_scratch_words(n) * 4);
    total = at;
  }
};

cudaError_t sort_results(kdop_scene* s, int64_t n, int64_t n_contacts, void* work) {
  cudaStream_t st = s->ctx->stream;
  if (n <= 0) return cudaSuccess;
  char* w = static_cast<char*>(work);
  SortWork L(n, n_contacts);
  SortBuffers b{reinterpret_cast<uint64_t*>(w + L.keys), reinterpret_cast<uint64_t*>(w + L.keys_tmp),
                reinterpret_cast<uint32_t*>(w + L.vals), reinterpret_cast<uint32_t*>(w + L.vals_tmp)};
  int4* rec_out = reinterpret_cast<int4*>(w + L.rec_out);
  float4* rows_out = reinterpret_cast<float4*>(w + L.rows_out);
  uint32_t* cand_out = reinterpret_cast<uint32_t*>(w + L.cand_out);
  const WaitLimit lim(&s->ctl->error, s->ctx->wait_ns);
  CandGen gen{s->cand, s->cand + s->cand_cap, s->cand + 2 * s->cand_cap, s->pairs, s->t_off_dev, bits_of(std::max<int64_t>(s->most_tets, 1) - 1)};
  const int pair_bits = bits_of((uint64_t)std::max<int64_t>(s->result_pairs, 1) - 1);
  const bool packed = s->pairs_current && !s->ctl_replayed && pair_bits + 2 * gen.tb <= 64;
  cudaError_t e;
  if (packed) {
    e = radix_sort(s->ctx, gen, n, pair_bits + 2 * gen.tb, b, w + L.scratch, lim);
  } else {
    const int tb = bits_of(s->nt > 0 ? s->nt - 1 : 0);  // at most 30
    e = radix_sort(s->ctx, TetGen{gen.cA, gen.cB, tb}, n, 2 * tb, b, w + L.scratch, lim);
    if (e == cudaSuccess) e = radix_sort(s->ctx, PairGen{gen.cP, b.vals, n}, n, 32, b, w + L.scratch, lim);
  }
  if (e != cudaSuccess) return e;
  const bool with_contacts = s->contacted;
  ApplyArgs a;
  a.n = n;
  a.keys = packed ? b.keys : nullptr;
  a.perm = b.vals;
  a.c = gen;
  a.n_pairs = std::max<int64_t>(s->result_pairs, 1);
  // the sorted keys hold the rows: they go straight to the scene's columns
  a.oA = packed ? s->cand : cand_out;
  a.oB = packed ? s->cand + s->cand_cap : cand_out + n;
  a.oP = packed ? s->cand + 2 * s->cand_cap : cand_out + 2 * n;
  a.rec = with_contacts ? s->records : nullptr;
  a.rec_out = rec_out;
  a.src = reinterpret_cast<uint32_t*>(w + L.src);
  a.ticket = reinterpret_cast<uint32_t*>(w + L.head);
  a.words = reinterpret_cast<unsigned long long*>(w + L.words);
  a.lim = lim;
  if (with_contacts && (e = cudaMemsetAsync(w + L.head, 0, L.keys - L.head, st)) != cudaSuccess) return e;
  const unsigned tiles = with_contacts ? tile_blocks(s->ctx, STUCK_SCAN, a.ticket, (unsigned)L.tiles) : (unsigned)L.tiles;
  sort_apply_kernel<<<tiles, 256, 0, st>>>(a);
  s->ctx->launches++;
  if (!packed)
    for (int k = 0; k < 3; ++k) {
      e = cudaMemcpyAsync(s->cand + k * s->cand_cap, cand_out + k * n, (size_t)n * 4, cudaMemcpyDeviceToDevice, st);
      if (e != cudaSuccess) return e;
    }
  if (with_contacts) {
    contact_gather_kernel<<<(unsigned)((n + 31) / 32), 256, 0, st>>>(
        n, rec_out, a.src, reinterpret_cast<const float4*>(s->contacts), rows_out, n_contacts);
    s->ctx->launches++;
    e = cudaMemcpyAsync(s->records, rec_out, (size_t)n * sizeof(int4), cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess && n_contacts > 0)
      e = cudaMemcpyAsync(s->contacts, rows_out, (size_t)n_contacts * sizeof(kdop_contact), cudaMemcpyDeviceToDevice,
                          st);
    if (e != cudaSuccess) return e;
  }
  return cudaGetLastError();
}

size_t sort_results_bytes(int64_t n, int64_t n_contacts) { return SortWork(n, n_contacts).total; }

}  // namespace kdop
