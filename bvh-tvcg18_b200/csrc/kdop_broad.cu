// kdop_broad.cu -- broad phase: the mesh pairs worth a tandem traversal.
//
// Reference: broad::find_overlaps (SIMULATION/BROAD/BROAD/include/
// broad_find_overlaps.h:44-125 all-pair, :134- grid; both report the same
// set, lexicographically sorted, lower object first).  Each body's box is
// its position +- its bounding radius (prox_rigid_body.h:159-172), the
// radius of a tetramesh the largest |r0| over its rest vertices
// (narrow_shape_types.h:189-206), and two boxes overlap unless one's max is
// strictly below the other's min on some axis.
//
// Here: the radii once per scene (thread per vertex, float max by its bit
// pattern, exact for non-negative values); per query one kernel: a warp takes a
// body i, its lanes the bodies j > i, counts, learns its place from a one-pass
// scan over the blocks (bodies in order), and writes its pairs there in j order
// -- the sorted list without a sort.
// Bound: latency.  Count and write passes of a thread per body left the GPU
// idle (12 blocks for 1,500 bodies, each thread a chain of 1,500 loads): 281 us
// with the scan between them, now one launch of 17 us.
#include <algorithm>

#include "kdop_device.cuh"
#include "kdop_sort.cuh"

namespace kdop {

namespace {

__global__ void radius_kernel(const float4* __restrict__ rest, int64_t nv, unsigned* rbits) {
  int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  float4 r = __ldg(rest + v);
  f3 x = mk3(r.x, r.y, r.z);
  float n = fsqrt(dot3(x, x));  // tiny::norm
  if (n == n) atomicMax(rbits + __float_as_int(r.w), __float_as_uint(n));
}

struct BoxArgs {
  const float4* pos;     // per body: position (x, y, z)
  const unsigned* rbits; // per body: radius bits
  int n;
};

__device__ __forceinline__ void box(const BoxArgs& a, int i, float* lo, float* hi) {
  float4 p = __ldg(a.pos + i);
  float r = __uint_as_float(__ldg(a.rbits + i));
  lo[0] = fsub(p.x, r);
  lo[1] = fsub(p.y, r);
  lo[2] = fsub(p.z, r);
  hi[0] = fadd(p.x, r);
  hi[1] = fadd(p.y, r);
  hi[2] = fadd(p.z, r);
}

__device__ __forceinline__ bool boxes_overlap(const float* la, const float* ha, const float* lb, const float* hb) {
  return !(hb[0] < la[0]) && !(ha[0] < lb[0]) && !(hb[1] < la[1]) && !(ha[1] < lb[1]) && !(hb[2] < la[2]) &&
         !(ha[2] < lb[2]);
}

constexpr int BR_WARPS = 8;  // bodies per block

// Bodies' overlaps with later bodies, in order.  Pairs past `cap` are counted
// and not written; total gets the number found.
__global__ void __launch_bounds__(32 * BR_WARPS) broad_kernel(BoxArgs a, uint2* out, unsigned cap, unsigned* ticket,
                                                              unsigned long long* words, unsigned* total,
                                                              WaitLimit lim) {
  __shared__ unsigned s_tile, s_count[BR_WARPS];
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
  __syncthreads();
  const unsigned tile = s_tile;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int i = (int)tile * BR_WARPS + w;
  float la[3] = {0.f, 0.f, 0.f}, ha[3] = {0.f, 0.f, 0.f};
  unsigned n = 0;
  if (i < a.n) {
    box(a, i, la, ha);
#pragma unroll 4
    for (int j = i + 1 + lane; j < a.n; j += 32) {
      float lb[3], hb[3];
      box(a, j, lb, hb);
      n += boxes_overlap(la, ha, lb, hb) ? 1u : 0u;
    }
  }
  n = __reduce_add_sync(0xffffffffu, n);
  if (lane == 0) s_count[w] = n;
  __syncthreads();
  unsigned before = 0, sum = 0;
#pragma unroll
  for (int k = 0; k < BR_WARPS; ++k) {
    if (k < w) before += s_count[k];
    sum += s_count[k];
  }
  const unsigned first = tile_prefix(words, tile, sum, lim);
  if (threadIdx.x == 0 && (int)(tile + 1) * BR_WARPS >= a.n) *total = first + sum;
  if (n == 0) return;
  unsigned at = first + before;
  for (int j0 = i + 1; j0 < a.n; j0 += 32) {
    const int j = j0 + lane;
    bool hit = false;
    if (j < a.n) {
      float lb[3], hb[3];
      box(a, j, lb, hb);
      hit = boxes_overlap(la, ha, lb, hb);
    }
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    const unsigned p = at + __popc(m & ((1u << lane) - 1u));
    if (hit && p < cap) out[p] = make_uint2((unsigned)i, (unsigned)j);
    at += __popc(m);
  }
}

__global__ void pack_pos_kernel(const float* __restrict__ pos, int n, float4* out) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = make_float4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], 0.f);
}

}  // namespace

cudaError_t launch_mesh_radius(kdop_scene* s, unsigned* rbits) {
  cudaError_t e = cudaMemsetAsync(rbits, 0, (size_t)std::max(s->n_meshes, 1) * 4, s->ctx->stream);
  if (e != cudaSuccess || s->nv == 0) return e;
  radius_kernel<<<(unsigned)((s->nv + 255) / 256), 256, 0, s->ctx->stream>>>(s->rest, s->nv, rbits);
  s->ctx->launches++;
  return cudaGetLastError();
}

// Work buffer of a query: total, error word and ticket, the blocks' published
// sums, packed positions.
struct BroadWork {
  size_t head, words, packed, total;
  explicit BroadWork(int n) {
    size_t at = 0;
    auto take = [&](size_t b) {
      size_t o = at;
      at += (b + 255) & ~(size_t)255;
      return o;
    };
    head = take(16);
    words = take((size_t)((n + BR_WARPS - 1) / BR_WARPS) * 8);
    packed = take((size_t)n * 16);
    total = at;
  }
};

size_t broad_work_bytes(int n) { return BroadWork(std::max(n, 1)).total; }

// Overlapping body pairs; pos_dev: device n x 3 positions or NULL for the
// scene's poses.  *total = pairs found; the first cap of them go to `pairs`
// (device).  Synchronises.
cudaError_t broad_phase(kdop_scene* s, const unsigned* rbits, const float* pos_dev, void* work, uint2* pairs,
                        int64_t cap, int64_t* total) {
  cudaStream_t st = s->ctx->stream;
  const int n = s->n_meshes;
  *total = 0;
  if (n < 2) return cudaSuccess;
  char* w = static_cast<char*>(work);
  BroadWork L(n);
  unsigned* head = reinterpret_cast<unsigned*>(w + L.head);  // total, error, ticket
  float4* packed = reinterpret_cast<float4*>(w + L.packed);
  BoxArgs a;
  a.rbits = rbits;
  a.n = n;
  cudaError_t e = cudaMemsetAsync(w + L.head, 0, L.packed - L.head, st);
  if (e != cudaSuccess) return e;
  if (pos_dev) {
    pack_pos_kernel<<<(n + 255) / 256, 256, 0, st>>>(pos_dev, n, packed);
    a.pos = packed;
  } else {
    a.pos = s->pos;
  }
  const unsigned blocks = tile_blocks(s->ctx, STUCK_SCAN, head + 2, (unsigned)((n + BR_WARPS - 1) / BR_WARPS));
  broad_kernel<<<blocks, 32 * BR_WARPS, 0, st>>>(a, pairs, (unsigned)std::min<int64_t>(cap, 0xFFFFFFFFll), head + 2,
                                                 reinterpret_cast<unsigned long long*>(w + L.words), head,
                                                 WaitLimit(head + 1, s->ctx->wait_ns));
  s->ctx->launches += pos_dev ? 2 : 1;
  unsigned h[2];
  if ((e = cudaMemcpyAsync(h, head, sizeof(h), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
  if (h[1]) return cudaErrorLaunchTimeout;
  *total = h[0];
  return cudaGetLastError();
}

}  // namespace kdop
