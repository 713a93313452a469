// kdop_refit.cu -- bottom-up kDOP refit of every tree of a scene.
//
// Reference: kdop::refit_tree (SIMULATION/KDOP/KDOP/include/kdop_refit_tree.h:
// 24-115 per chunk, 120-162 per tree): a leaf gets make_dop of its tet's four
// vertices (FOUNDATION/GEOMETRY/GEOMETRY/include/types/geometry_dop.h:49-74),
// an internal node make_union of its two children (geometry_make_union.h:
// 10-24).  The OpenCL back-end did one work-group per object with retry loops
// (cl/kernels/kdop_cl_refit_tree.cl:17-168).
//
// Here one launch refits nine levels of every tree.  The index-median split
// makes a tree over n tets complete down to depth L = floor(log2 n), where a
// node holds one tet or two, so node i of depth d < L has the children 2 i and
// 2 i + 1 of depth d + 1, and the nodes of one depth of one tree are
// consecutive in memory.  A block takes 256 consecutive nodes of depth L: a
// thread projects its node's one or two tets (written as leaves of depth L + 1
// when there are two), and the block unites the 256 records in shared memory
// up to their common ancestor and writes each level's records as one
// consecutive range.  The next launch starts from the 1/256 as many ancestors.
// In pose or deform mode the refit first poses every vertex once
// (narrow_update_kdop_bvh.h:154-165 on the device, in the same call and the
// same graph) into a scene-owned array the leaves read: posing inside the leaf
// pass would transform each vertex once per tet that uses it (about 24 times
// in a lattice).
// Bound: the L1 data pipe (73 to 77 % of its peak at K = 14 and 18: the leaves'
// vertex gathers, the shared-memory unions, the records' stores), then HBM (47
// %).  Each node record is written once; a launch per level wrote every one, read it
// again for its parent and gathered a leaf's tet through the record's topology
// words, which now come from arrays in leaf order.  Steps before -> after: 64
// deforming pairs of 384 k tets (K = 18) 5.00 -> 3.53 ms (3.15 since the warps
// of large forests stop alone), one pair of 1.6 M tets (K = 26) 1.66 -> 1.36
// ms, 512 uneven pairs (K = 14) 13.2 -> 12.07 ms, one pair of 6,000 tets 273 ->
// 202 us.  Not kept: block barriers between the levels and a runtime walk over
// them (96 trees of 48,000 tets: 217 us against 185), one block fewer per SM
// (208).
#include <algorithm>

#include "kdop_device.cuh"

namespace kdop {

__device__ __forceinline__ void stg256(float4* p, const float* a, const float* b) {
  asm volatile("st.global.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "f"(a[0]), "f"(a[1]), "f"(a[2]),
               "f"(a[3]), "f"(b[0]), "f"(b[1]), "f"(b[2]), "f"(b[3])
               : "memory");
}

// Components of the unit corner and edge directions of the direction tables.
struct DirScale {
  float corner, edge;
};

// Projections of a point on the K/2 directions: dot3(d, p) = ((0 + d.x p.x) +
// d.y p.y) + d.z p.z for the axes, (1, +-1, +-1) corner and edge directions of
// the tables, with the products the directions share computed once (a product
// with -c is the negative of that with c; x * 1 is x; products with 0 stay,
// they carry infinities and NaN).  42 multiplications and additions become 20
// at K = 14.
template <int K>
__device__ __forceinline__ void project(float4 q, DirScale ds, float* p) {
  constexpr bool AXES = K == 6 || K == 14 || K == 18 || K == 26;
  constexpr bool CORNERS = K == 8 || K == 14 || K == 20 || K == 26;
  constexpr bool EDGES = K == 12 || K == 18 || K == 20 || K == 26;
  const float zy = fmul(q.y, 0.f), zz = fmul(q.z, 0.f), z0 = fadd(0.f, fmul(q.x, 0.f));
  int n = 0;
  if (AXES) {
    p[n++] = fadd(fadd(fadd(0.f, q.x), zy), zz);
    p[n++] = fadd(fadd(z0, q.y), zz);
    p[n++] = fadd(fadd(z0, zy), q.z);
  }
  if (CORNERS) {
    const float x = fadd(0.f, fmul(q.x, ds.corner)), y = fmul(q.y, ds.corner), z = fmul(q.z, ds.corner);
    const float a = fadd(x, y), b = fsub(x, y);
    p[n++] = fadd(a, z);
    p[n++] = fsub(a, z);
    p[n++] = fadd(b, z);
    p[n++] = fsub(b, z);
  }
  if (EDGES) {
    const float ex = fmul(q.x, ds.edge), y = fmul(q.y, ds.edge), z = fmul(q.z, ds.edge);
    const float x = fadd(0.f, ex);
    p[n++] = fadd(fadd(x, y), zz);
    p[n++] = fadd(fsub(x, y), zz);
    p[n++] = fadd(fadd(x, zy), z);
    p[n++] = fadd(fadd(z0, y), z);
    p[n++] = fadd(fadd(fsub(0.f, ex), zy), z);
    p[n++] = fadd(fsub(z0, y), z);
  }
}

// Slabs of a tet with vertices v (make_dop).  A projection is a sum that
// starts from +0, so it is never -0, and the running bounds start finite:
// fminf / fmaxf (one instruction; a NaN operand is dropped) give the values
// of the reference's std::min / std::max.
template <int K>
__device__ __forceinline__ void leaf_slabs(const float4* __restrict__ world, uint4 v, DirScale ds, float* w) {
  const float4 q[4] = {__ldg(world + v.x), __ldg(world + v.y), __ldg(world + v.z), __ldg(world + v.w)};
  float p[4][K / 2];
#pragma unroll
  for (int u = 0; u < 4; ++u) project<K>(q[u], ds, p[u]);
  constexpr float big = 3.40282346638528859812e+38f;
#pragma unroll
  for (int s = 0; s < K / 2; ++s) {
    w[2 * s] = fminf(fminf(fminf(big, p[0][s]), p[1][s]), fminf(p[2][s], p[3][s]));
    w[2 * s + 1] = fmaxf(fmaxf(fmaxf(-big, p[0][s]), p[1][s]), fmaxf(p[2][s], p[3][s]));
  }
}

constexpr int kRefitUp = 8;                    // levels a block unites above its nodes
constexpr int kRefitSlots = 1 << kRefitUp;     // nodes a block starts from
// From this many blocks on, the first launch's warps each stop at the ancestor
// of their own 32 nodes: a block's last three levels and its barrier keep seven
// of its eight warps' places taken while one works (96 trees of 48,000 tets,
// 12,288 blocks: K = 18 222 -> 211 us, K = 20 251 -> 229, K = 26 313 -> 287).
// Smaller forests keep the block's join, which saves levels of the next launch.
constexpr int64_t kWarpsAloneBlocks = 2048;
// Forests of trees smaller than this have blocks of one warp with the shared
// memory of 32 nodes: of 256 threads seven warps had nothing to do (20,000 trees
// of one tet, K = 26: 74 -> 20 us, a launch per level 52; 3,000 of 63, K = 14: 21 ->
// 11, 3,000 of 64 with blocks of 256 threads 22).
constexpr int64_t kTinyTets = 64;
// Shared-memory row of one record word: the block's nodes in heap order (root
// 1).  Rows are 8 banks apart, so that two slabs a lane group apart in a union
// fall on other halves of the banks, and a chunk's four rows are shifted by
// chunk_skew banks more, so that the chunks of consecutive twins, which the
// lanes of a store take, do not meet (rows of 514 words without the shift cost
// 6.4 M of 43 M shared-memory passes at K = 18).
template <int SLOTS>
__host__ __device__ constexpr int refit_row() {
  return 2 * SLOTS + 8;
}
template <int K>
__host__ __device__ constexpr int chunk_skew() {
  constexpr int NW = NodeLayout<K>::NW;
  return NW == 2 ? 16 : NW == 3 ? 10 : NW == 4 ? 8 : NW <= 6 ? 6 : 4;
}
template <int K, int SLOTS>
__device__ __forceinline__ float* word_row(float* T, int w) {
  return T + w * refit_row<SLOTS>() + chunk_skew<K>() * (w >> 2);
}
template <int K, int SLOTS>
__host__ __device__ constexpr int refit_words() {
  return (K * refit_row<SLOTS>() + chunk_skew<K>() * NodeLayout<K>::NW + 1) & ~1;  // slot_words follow, 8-byte aligned
}
template <int K, int SLOTS>
constexpr size_t refit_smem() {
  return (size_t)refit_words<K, SLOTS>() * 4 + SLOTS * 8;
}

struct RefitArgs {
  float4* nodes;
  const RefitBlock* blocks;
  const uint4* leaf_verts;
  const uint32_t* leaf_tet;
  const float4* world;
  DirScale ds;
};

// Slab x of node U of the block's heap: the union of its children (make_union;
// slabs hold no NaN and no -0, so fminf / fmaxf are the reference's choices).
template <int K, int SLOTS>
__device__ __forceinline__ void unite_slab(float* T, uint32_t U, int x) {
  float* row = word_row<K, SLOTS>(T, 2 * x);
  const float2 lo = *reinterpret_cast<const float2*>(row + 2 * U);
  const float2 hi = *reinterpret_cast<const float2*>(row + refit_row<SLOTS>() + 2 * U);
  row[U] = fminf(lo.x, lo.y);
  row[refit_row<SLOTS>() + U] = fmaxf(hi.x, hi.y);
}
// The 2^M nodes M levels below `root`, a slab of a node per lane.
template <int K, int SLOTS, int M>
__device__ __forceinline__ void unite_level(float* T, uint32_t root, int lane) {
  constexpr int N = (K / 2) << M;
#pragma unroll
  for (int it = 0; it * 32 < N; ++it)
    if ((it + 1) * 32 <= N || it * 32 + lane < N)
      unite_slab<K, SLOTS>(T, (root << M) + (uint32_t)(lane & ((1 << M) - 1)), (lane >> M) + it * (32 >> M));
  __syncwarp();
}

// Chunk j of the twin of the children of heap node U to `to`; the topology
// words of its two nodes are we, wo.
template <int K, int SLOTS>
__device__ __forceinline__ void put_chunk(const float* T, uint32_t U, int j, uint2 we, uint2 wo, float4* to) {
  const float* col = T + j * (4 * refit_row<SLOTS>() + chunk_skew<K>()) + 2 * U;
  float e[4], o[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    e[c] = o[c] = 0.f;
    if (4 * j + c < K) {
      const float2 x = *reinterpret_cast<const float2*>(col + c * refit_row<SLOTS>());
      e[c] = x.x;
      o[c] = x.y;
    }
  }
  if (j == NodeLayout<K>::TOPO_CHUNK) {
    constexpr int c = K % 4;
    e[c] = __uint_as_float(we.x);
    e[c + 1] = __uint_as_float(we.y);
    o[c] = __uint_as_float(wo.x);
    o[c + 1] = __uint_as_float(wo.y);
  }
  stg256(to, e, o);
}
// Chunk j of heap node U alone.
template <int K, int SLOTS>
__device__ __forceinline__ float4 half_chunk(float* T, uint32_t U, int j, uint2 words) {
  float e[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int w = 4 * j + c;
    e[c] = w < K ? word_row<K, SLOTS>(T, w)[U]
                 : w == K ? __uint_as_float(words.x) : w == K + 1 ? __uint_as_float(words.y) : 0.f;
  }
  return make_float4(e[0], e[1], e[2], e[3]);
}
// The twins of the children of the 2^M nodes M levels below heap node `root`,
// which is the at-th of its level: consecutive records from node `first` on; a
// chunk per lane, so that a warp writes 1 KB in a row.  kids: first child of
// the first of them; words: their topology words instead, where they are the
// block's own nodes.
template <int K, int SLOTS, int M>
__device__ __forceinline__ void put_level(float4* nodes, const float* T, uint32_t root, uint32_t first, uint32_t kids,
                                          const uint2* words, int lane) {
  constexpr int NW = NodeLayout<K>::NW, N = NW << M;
  float4* to = nodes + NodeLayout<K>::at(first, 0) + 2 * lane;
#pragma unroll
  for (int it = 0; it * 32 < N; ++it) {
    if ((it + 1) * 32 > N && it * 32 + lane >= N) continue;
    constexpr bool pow2 = (NW & (NW - 1)) == 0;
    constexpr int sh = NW == 1 ? 0 : NW == 2 ? 1 : 2;
    const int r = pow2 ? (lane >> sh) + it * (32 >> sh) : (it * 32 + lane) / NW;
    const int j = pow2 ? lane & (NW - 1) : (it * 32 + lane) % NW;
    const uint32_t k = kids + 4u * (uint32_t)r;
    uint2 we = make_uint2(k, k + 1u), wo = make_uint2(k + 2u, k + 3u);
    if (words) {
      we = words[2 * r];
      wo = words[2 * r + 1];
    }
    put_chunk<K, SLOTS>(T, (root << M) + (uint32_t)r, j, we, wo, to + 64 * it);
  }
}

// BOTTOM: from the tets of the nodes of depth L; else from the records of the
// block's nodes, written by the launch before.  A warp unites its 32 nodes and
// writes their levels by itself (no block barrier); the first warp does the
// last levels from the warps' ancestors.
template <int K, bool BOTTOM, int SLOTS>
__global__ void __launch_bounds__(SLOTS, SLOTS == 32 ? (K <= 20 ? 32 : 24) : K <= 8 ? 6 : K <= 14 ? 5 : K <= 20 ? 4 : 3)
    refit_kernel(const __grid_constant__ RefitArgs a) {
  using L = NodeLayout<K>;
  constexpr int NW = L::NW, NS = L::NS;
  extern __shared__ float T[];  // word_row(T, w)[heap index]
  uint2* slot_words = reinterpret_cast<uint2*>(T + refit_words<K, SLOTS>());
  const RefitBlock& b = a.blocks[blockIdx.x];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int hd = b.levels;             // levels above the block's nodes in this block
  const int cnt = 1 << hd;             // its nodes
  const int wl = min(hd, 5);           // levels within a warp
  const int warps = cnt >> wl;         // warps with nodes
  const uint32_t root = (uint32_t)(warps + wib);  // this warp's ancestor in the block's heap
  if (wib < warps) {
    const int t = (wib << wl) + lane;  // this thread's node of the block
    if (BOTTOM) {
      const bool act = lane < (1 << wl);
      // The left half takes the odd tet at every split, so of 2^h nodes below
      // an ancestor with r tets more than nodes the j-th in bit-reversed order
      // holds two when j < r: the block's extra tets over its warps, then the
      // warp's over its lanes.
      const uint32_t extra = b.tets - (uint32_t)cnt;
      const int wb = hd - wl;  // bits of a warp's number
      uint32_t before = 0, mine = extra;
      if (wb) {
#pragma unroll
        for (int w = 0; w < SLOTS / 32; ++w) {
          const uint32_t x = (extra + (1u << wb) - 1u - (__brev((uint32_t)w) >> (32 - wb))) >> wb;
          if (w < wib) before += x;
          if (w == wib) mine = x;
        }
      }
      const uint32_t rev = wl ? __brev((uint32_t)lane) >> (32 - wl) : 0u;
      const bool two = act && rev < mine;
      const unsigned twos = __ballot_sync(0xffffffffu, two);
      before += __popc(twos & ((1u << lane) - 1u));  // two-tet nodes of the block before this one
      if (act) {
        // a node of one tet takes it twice (the union with itself)
        const size_t at = (size_t)b.first_leaf + t + before;
        const uint4 va = __ldg(a.leaf_verts + at), vb = __ldg(a.leaf_verts + at + (two ? 1 : 0));
        const uint32_t t0 = __ldg(a.leaf_tet + at), t1 = __ldg(a.leaf_tet + at + (two ? 1 : 0));
        float w[4 * NW], v[4 * NW];
#pragma unroll
        for (int c = 0; c < 4 * NW; ++c) w[c] = v[c] = 0.f;
        leaf_slabs<K>(a.world, va, a.ds, w);
        leaf_slabs<K>(a.world, vb, a.ds, v);
        uint2 words = make_uint2(LEAF_BIT | (t0 & SURF_BIT) | (b.node[hd] + t), t0 & NODE_MASK);
        if (two) {
          // two leaves: their twin of depth L + 1
          const uint32_t c = b.leaf_twin + 2u * before;
          w[K] = __uint_as_float(LEAF_BIT | (t0 & SURF_BIT) | c);
          w[K + 1] = __uint_as_float(t0 & NODE_MASK);
          v[K] = __uint_as_float(LEAF_BIT | (t1 & SURF_BIT) | (c + 1u));
          v[K + 1] = __uint_as_float(t1 & NODE_MASK);
          float4* to = a.nodes + L::at(c, 0);
#pragma unroll
          for (int j = 0; j < NW; ++j) stg256(to + 2 * j, w + 4 * j, v + 4 * j);
          words = make_uint2(c, c + 1u);
        }
        slot_words[t] = words;
#pragma unroll
        for (int k = 0; k < K; k += 2) {
          word_row<K, SLOTS>(T, k)[cnt + t] = fminf(w[k], v[k]);
          word_row<K, SLOTS>(T, k + 1)[cnt + t] = fmaxf(w[k + 1], v[k + 1]);
        }
      }
    } else {
      // records of the warp's 2^wl >= 2 consecutive nodes (whole twins)
      const float4* from = a.nodes + L::at(b.node[hd] + (wib << wl), 0);
      for (int q = lane; q < (NW << wl); q += 32) {
        const float4 x = from[q];
        const int i = (wib << wl) + 2 * (q / (2 * NW)) + (q & 1), j = (q % (2 * NW)) >> 1;
        const float e[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (4 * j + c < K) word_row<K, SLOTS>(T, 4 * j + c)[cnt + i] = e[c];
      }
    }
    __syncwarp();
    if (wl == 5) {
      unite_level<K, SLOTS, 4>(T, root, lane);
      unite_level<K, SLOTS, 3>(T, root, lane);
      unite_level<K, SLOTS, 2>(T, root, lane);
      unite_level<K, SLOTS, 1>(T, root, lane);
      unite_level<K, SLOTS, 0>(T, root, lane);
      // levels from the block's own nodes up: those M + 1 levels below the
      // warp's ancestor start at node 2^(M + 1) wib of their level
      const uint32_t w = (uint32_t)wib;
      if (BOTTOM)
        put_level<K, SLOTS, 4>(a.nodes, T, root, b.node[hd] + 32u * w, 0u, slot_words + 32 * wib, lane);
      put_level<K, SLOTS, 3>(a.nodes, T, root, b.node[hd - 1] + 16u * w, b.node[hd] + 32u * w, nullptr, lane);
      put_level<K, SLOTS, 2>(a.nodes, T, root, b.node[hd - 2] + 8u * w, b.node[hd - 1] + 16u * w, nullptr, lane);
      put_level<K, SLOTS, 1>(a.nodes, T, root, b.node[hd - 3] + 4u * w, b.node[hd - 2] + 8u * w, nullptr, lane);
      put_level<K, SLOTS, 0>(a.nodes, T, root, b.node[hd - 4] + 2u * w, b.node[hd - 3] + 4u * w, nullptr, lane);
      if (b.warps_alone && lane < NW) {
        // the next launch starts from the warps' ancestors
        const uint32_t kids = b.node[hd - 4] + 2u * w;
        a.nodes[L::at(b.node[hd - 5] + w, lane)] = half_chunk<K, SLOTS>(T, root, lane, make_uint2(kids, kids + 1u));
      }
    } else {
      // a tree of fewer than 64 tets (or its last levels): one warp, level by level
      for (int m = wl - 1; m >= 0; --m) {
        for (int x = lane; x < (NS << m); x += 32) unite_slab<K, SLOTS>(T, (1u << m) + (x & ((1 << m) - 1)), x >> m);
        __syncwarp();
      }
      for (int m = BOTTOM ? wl - 1 : wl - 2; m >= 0; --m)
        for (int q = lane; q < (NW << m); q += 32) {
          const uint32_t r = (uint32_t)(q / NW);
          const uint32_t k = m + 2 <= hd ? b.node[m + 2] + 4u * r : 0u;
          uint2 we = make_uint2(k, k + 1u), wo = make_uint2(k + 2u, k + 3u);
          if (m + 1 == hd) {
            we = slot_words[2 * r];
            wo = slot_words[2 * r + 1];
          }
          put_chunk<K, SLOTS>(T, (1u << m) + r, q % NW, we, wo, a.nodes + L::at(b.node[m + 1], 0) + 2 * q);
        }
    }
  }
  if (b.warps_alone) return;
  __syncthreads();
  if (wib > 0) return;
  for (int n = warps >> 1; n >= 1; n >>= 1) {
    for (int x = lane; x < n * NS; x += 32) unite_slab<K, SLOTS>(T, (uint32_t)(n + x % n), x / n);
    __syncwarp();
  }
  for (int q = lane; q < (warps - 1) * NW; q += 32) {
    // the twin below heap node U
    const uint32_t U = (uint32_t)(q / NW) + 1u;
    const int l = 32 - __clz(U);
    const uint32_t i = 2 * U - (1u << l), k = b.node[l + 1] + 2u * i;
    const int j = q % NW;
    put_chunk<K, SLOTS>(T, U, j, make_uint2(k, k + 1u), make_uint2(k + 2u, k + 3u), a.nodes + L::at(b.node[l] + i, j));
  }
  // the common ancestor: one half of a twin
  if (lane < NW) {
    const uint2 words = (BOTTOM && hd == 0) ? slot_words[0] : make_uint2(b.node[1], b.node[1] + 1u);
    a.nodes[L::at(b.node[0], lane)] = half_chunk<K, SLOTS>(T, 1u, lane, words);
    if (b.pad_node != NO_NODE) {
      // the root level's padding node: the root again (a leaf under its own index)
      const uint32_t own = (words.x & LEAF_BIT) ? (words.x & (LEAF_BIT | SURF_BIT)) | b.pad_node : words.x;
      a.nodes[L::at(b.pad_node, lane)] = half_chunk<K, SLOTS>(T, 1u, lane, make_uint2(own, words.y));
    }
  }
}

// Tets in leaf order, from the topology words of the nodes of depth L and
// L + 1: vertex indices, and the tet with its surface bit.  A block per block
// of the refit's first launch.
template <int K>
__global__ void __launch_bounds__(kRefitSlots) leaf_table_kernel(const float4* __restrict__ nodes,
                                                                 const RefitBlock* __restrict__ blocks,
                                                                 const uint4* __restrict__ tets, uint4* leaf_verts,
                                                                 uint32_t* leaf_tet) {
  using L = NodeLayout<K>;
  const RefitBlock& b = blocks[blockIdx.x];
  if ((int)threadIdx.x >= (1 << b.levels)) return;
  uint32_t f = 0, s = b.tets;
  for (int k = b.levels - 1; k >= 0; --k) {
    const uint32_t left = s - (s >> 1);
    if ((threadIdx.x >> k) & 1u) f += left;
    s = ((threadIdx.x >> k) & 1u) ? s >> 1 : left;
  }
  const float4 x = nodes[L::at(b.node[b.levels] + threadIdx.x, L::TOPO_CHUNK)];
  const uint32_t node = L::word0(x) & NODE_MASK;  // a leaf's own index, or its first child
  for (uint32_t c = 0; c < s; ++c) {
    const float4 y = nodes[L::at(node + c, L::TOPO_CHUNK)];
    const uint32_t tet = L::word1(y);
    leaf_verts[(size_t)b.first_leaf + f + c] = tets[tet];
    leaf_tet[(size_t)b.first_leaf + f + c] = tet | (L::word0(y) & SURF_BIT);
  }
}

// Topology words into the node records, slabs zeroed.  topo holds the
// reference's (m_start, m_end) per node (leaf <=> start == end = tet).
template <int K>
__global__ void write_topology_kernel(float4* nodes, int64_t nn, const uint32_t* __restrict__ topo,
                                      const uint8_t* __restrict__ surf) {
  using L = NodeLayout<K>;
  int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nn * L::NW) return;
  int64_t node = 2 * (t / (2 * L::NW)) + (t & 1);
  int j = (int)((t % (2 * L::NW)) >> 1);
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  if (j == L::TOPO_CHUNK) {
    uint32_t st = topo[2 * node], en = topo[2 * node + 1];
    if (st == en) {
      en = st;
      st = LEAF_BIT | (surf[en] ? SURF_BIT : 0u) | (uint32_t)node;
    }
    float a = __uint_as_float(st), b = __uint_as_float(en);
    if (L::TOPO_ZW) {
      o.z = a;
      o.w = b;
    } else {
      o.x = a;
      o.y = b;
    }
  }
  nodes[t] = o;
}

// One tree in the reference's preorder: thread per node h of depths 0 .. L in
// heap numbering, which also takes the two leaves below a two-tet node.  The
// left half of s tets fills 2 left - 1 places after its parent's.  Only the
// places [first, first + count) are written (a window of the caller's buffer).
struct TreeBase {
  uint32_t base[32];  // first node of each depth
};
template <int K>
__device__ __forceinline__ void put_node(const float4* __restrict__ nodes, uint32_t node, int64_t at, int64_t count,
                                         uint32_t t_off, float* vol, int64_t* tet) {
  using L = NodeLayout<K>;
  if (at < 0 || at >= count) return;
  uint32_t w0 = 0, w1 = 0;
#pragma unroll
  for (int j = 0; j < L::NW; ++j) {
    const float4 x = nodes[L::at(node, j)];
    const float e[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int c = 0; c < 4; ++c)
      if (4 * j + c < K) vol[at * K + 4 * j + c] = e[c];
    if (j == L::TOPO_CHUNK) {
      w0 = L::word0(x);
      w1 = L::word1(x);
    }
  }
  tet[at] = (w0 & LEAF_BIT) ? (int64_t)w1 - (int64_t)t_off : -1;
}
template <int K>
__global__ void __launch_bounds__(256) preorder_kernel(const float4* __restrict__ nodes, TreeBase b, uint32_t n_tets,
                                                       int depth, uint32_t t_off, int64_t first, int64_t count,
                                                       float* vol, int64_t* tet) {
  const uint32_t h = blockIdx.x * 256 + threadIdx.x + 1;
  if (h >= (2u << depth)) return;
  const int d = 31 - __clz(h);
  uint32_t s = n_tets;
  int64_t at = -first;
  for (int k = d - 1; k >= 0; --k) {
    const uint32_t left = s - (s >> 1);
    if ((h >> k) & 1u) {
      at += 2 * (int64_t)left;
      s >>= 1;
    } else {
      at += 1;
      s = left;
    }
  }
  const uint32_t node = b.base[d] + (h - (1u << d));
  put_node<K>(nodes, node, at, count, t_off, vol, tet);
  if (d == depth && s == 2u) {
    using L = NodeLayout<K>;
    const uint32_t c = L::word0(nodes[L::at(node, L::TOPO_CHUNK)]);
    put_node<K>(nodes, c, at + 1, count, t_off, vol, tet);
    put_node<K>(nodes, c + 1, at + 2, count, t_off, vol, tet);
  }
}

// World positions of all vertices (pose / deform modes), for read-back.
__global__ void world_kernel(int64_t nv, VertexSource vs, float4* out) {
  int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= nv) return;
  f3 x = world_vertex(vs, (uint32_t)v);
  out[v] = make_float4(x.x, x.y, x.z, 0.f);
}

// One step of rigid motion per mesh and of the deformation phase:
// p += v, q = normalise(q + 0.5 (0, w) q).
__global__ void motion_kernel(int n_meshes, float4* quat, float4* pos, const float4* __restrict__ lin,
                              const float4* __restrict__ ang, float* phase, float phase_rate) {
  int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m == 0) *phase = *phase + phase_rate;
  if (m >= n_meshes) return;
  float4 p = pos[m], v = lin[m], q = quat[m], w = ang[m];
  p.x += v.x;
  p.y += v.y;
  p.z += v.z;
  // dq = 0.5 * (0, w) (x) q
  float dw = -(w.x * q.y + w.y * q.z + w.z * q.w);
  float dx = w.x * q.x + (w.y * q.w - w.z * q.z);
  float dy = w.y * q.x + (w.z * q.y - w.x * q.w);
  float dz = w.z * q.x + (w.x * q.z - w.y * q.y);
  q.x += 0.5f * dw;
  q.y += 0.5f * dx;
  q.z += 0.5f * dy;
  q.w += 0.5f * dz;
  float inv = rsqrtf(q.x * q.x + q.y * q.y + q.z * q.z + q.w * q.w);
  q.x *= inv;
  q.y *= inv;
  q.z *= inv;
  q.w *= inv;
  quat[m] = q;
  pos[m] = p;
}

// xyz triples -> float4 (w = mesh index bits when with_mesh_id >= 0, else 0)
__global__ void pack3_kernel(const float* __restrict__ in, float4* out, int64_t n, const float4* __restrict__ keep_w,
                             int keep) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float w = keep ? keep_w[i].w : 0.f;
  out[i] = make_float4(in[3 * i], in[3 * i + 1], in[3 * i + 2], w);
}

__global__ void pack_poses_kernel(const float* __restrict__ q, const float* __restrict__ p, float4* quat, float4* pos,
                                  int64_t n) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  quat[i] = make_float4(q[4 * i], q[4 * i + 1], q[4 * i + 2], q[4 * i + 3]);
  pos[i] = make_float4(p[3 * i], p[3 * i + 1], p[3 * i + 2], 0.f);
}

cudaError_t launch_pack3(kdop_scene* s, const float* in, float4* out, int64_t n, int with_mesh_id) {
  if (n <= 0) return cudaSuccess;
  pack3_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s->ctx->stream>>>(in, out, n, s->rest, with_mesh_id >= 0);
  s->ctx->launches++;
  return cudaGetLastError();
}
cudaError_t launch_pack_poses(kdop_scene* s, const float* quat, const float* pos) {
  const int64_t n = s->n_meshes;
  if (n <= 0) return cudaSuccess;
  pack_poses_kernel<<<(unsigned)((n + 127) / 128), 128, 0, s->ctx->stream>>>(quat, pos, s->quat, s->pos, n);
  s->ctx->launches++;
  return cudaGetLastError();
}

static VertexSource vertex_source(kdop_scene* s, int mode) {
  VertexSource vs;
  vs.rest = s->rest;
  vs.world = s->world;
  vs.quat = s->quat;
  vs.pos = s->pos;
  vs.deform.amp = s->amp;
  vs.deform.w = s->w;
  vs.deform.phase = s->phase_dev;
  vs.mode = mode;
  return vs;
}


template <int K>
static cudaError_t refit_impl(kdop_scene* s, int mode) {
  VertexSource vs = vertex_source(s, mode);
  const float4* world = s->world;
  if (mode != KDOP_REFIT_VERTICES && s->nv > 0) {
    // pose (and deform) every vertex once; the leaves then read world
    // positions instead of transforming each vertex once per tet using it
    world_kernel<<<(unsigned)((s->nv + 255) / 256), 256, 0, s->ctx->stream>>>(s->nv, vs, s->posed);
    s->ctx->launches++;
    world = s->posed;
  }
  // the direction tables list axes, corners, edges (K = 14: 3 axes, 4 corners)
  constexpr int axes = (K == 6 || K == 14 || K == 18 || K == 26) ? 3 : 0;
  constexpr int corners = (K == 8 || K == 14 || K == 20 || K == 26) ? 4 : 0;
  RefitArgs a;
  a.nodes = s->nodes;
  a.leaf_verts = s->leaf_verts;
  a.leaf_tet = s->leaf_tet;
  a.world = world;
  a.ds.corner = corners ? s->dirs.d[axes][0] : 0.f;
  a.ds.edge = axes + corners < K / 2 ? s->dirs.d[axes + corners][0] : 0.f;
  if (s->most_tets < kTinyTets) {
    // one launch: no tree has more than 32 nodes of depth L
    const unsigned n = s->refit_stage.size() > 1 ? (unsigned)s->refit_stage[1] : 0u;
    a.blocks = s->refit_blocks;
    if (n) {
      refit_kernel<K, true, 32><<<n, 32, refit_smem<K, 32>(), s->ctx->stream>>>(a);
      s->ctx->launches++;
    }
    return cudaGetLastError();
  }
  constexpr size_t smem = refit_smem<K, kRefitSlots>();
  cudaError_t e =
      cudaFuncSetAttribute(refit_kernel<K, true, kRefitSlots>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(refit_kernel<K, false, kRefitSlots>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
  if (e != cudaSuccess) return e;
  for (size_t i = 0; i + 1 < s->refit_stage.size(); ++i) {
    const unsigned n = (unsigned)(s->refit_stage[i + 1] - s->refit_stage[i]);
    a.blocks = s->refit_blocks + s->refit_stage[i];
    if (i == 0)
      refit_kernel<K, true, kRefitSlots><<<n, kRefitSlots, smem, s->ctx->stream>>>(a);
    else
      refit_kernel<K, false, kRefitSlots><<<n, kRefitSlots, smem, s->ctx->stream>>>(a);
    s->ctx->launches++;
  }
  return cudaGetLastError();
}

// Blocks of each launch of a refit (launch i: blocks stage[i] .. stage[i + 1]):
// one per 256 nodes of depth L of every tree, then of depth L - 8, L - 16 and so
// on.  In a large forest the first launch's warps stop at their own ancestors
// and the depths are L, L - 5, L - 13, ...: its blocks then have no barrier and
// no last levels that one warp works on while the other seven's place stays
// taken (12,288 blocks: kWarpsAloneBlocks); in a small
// one the launch that this can add costs more.  pre: nodes of the trees before
// m at depth d; t_off: first tet of a mesh.
void refit_blocks(const ForestBuild& fb, const std::vector<int64_t>& pre, const std::vector<int32_t>& lg,
                  const std::vector<int64_t>& n_tets, const std::vector<int64_t>& t_off,
                  std::vector<RefitBlock>& blocks, std::vector<int64_t>& stage) {
  blocks.clear();
  stage.assign(1, 0);
  const size_t nm = lg.size();
  const int levels = (int)fb.level_off.size() - 1;
  auto base = [&](size_t m, int d) -> uint32_t {
    return d < levels ? (uint32_t)(fb.level_off[d] + pre[(size_t)d * (nm + 1) + m]) : 0u;
  };
  // the root level holds one padding node after the real roots when their
  // count is odd: the first tree's root again
  int64_t n_roots = 0;
  for (size_t m = 0; m < nm; ++m) n_roots += lg[m] >= 0 ? 1 : 0;
  uint32_t pad = NO_NODE;
  if (n_roots > 0 && fb.level_off[1] - fb.level_off[0] > n_roots) pad = (uint32_t)(fb.level_off[1] - 1);
  size_t first = 0;
  while (first < nm && lg[first] < 0) ++first;
  int64_t bottom = 0;
  for (size_t m = 0; m < nm; ++m) bottom += lg[m] >= 0 ? int64_t(1) << std::max(lg[m] - kRefitUp, 0) : 0;
  const bool alone = bottom >= kWarpsAloneBlocks;
  std::vector<std::pair<uint32_t, uint32_t>> range, next;  // tets [f, f + s) of the nodes of one depth
  for (int i = 0;; ++i) {
    const int above = kRefitUp * i - (alone && i > 0 ? kRefitUp - 5 : 0);
    for (size_t m = 0; m < nm; ++m) {
      const int d = lg[m] - above;  // depth 0 is done by the launch before, or is a single node
      if (lg[m] < 0 || d < 0 || (i > 0 && d == 0)) continue;
      const int hd = std::min(d, kRefitUp), d0 = d - hd;
      range.assign(1, std::make_pair(0u, (uint32_t)n_tets[m]));
      for (int k = 0; k < d0; ++k) {
        next.clear();
        for (const auto& r : range) {
          const uint32_t left = r.second - (r.second >> 1);
          next.push_back(std::make_pair(r.first, left));
          next.push_back(std::make_pair(r.first + left, r.second - left));
        }
        range.swap(next);
      }
      for (size_t j = 0; j < range.size(); ++j) {
        RefitBlock b;
        b.first_leaf = (uint32_t)t_off[m] + range[j].first;
        b.tets = range[j].second;
        // two-tet nodes before the block's: its first tet less its first node
        b.leaf_twin = base(m, lg[m] + 1) + 2u * (range[j].first - (uint32_t)(j << hd));
        b.levels = hd;
        for (int l = 0; l <= kRefitUp; ++l) b.node[l] = l <= hd ? base(m, d0 + l) + (uint32_t)(j << l) : 0u;
        b.pad_node = (d0 == 0 && m == first) ? pad : NO_NODE;
        b.warps_alone = alone && i == 0 && hd > 5;
        b.pad = 0;
        blocks.push_back(b);
      }
    }
    if ((int64_t)blocks.size() == stage.back()) break;
    stage.push_back((int64_t)blocks.size());
  }
}

template <int K>
static cudaError_t leaf_tables_impl(kdop_scene* s) {
  if (s->refit_stage.size() < 2) return cudaSuccess;
  leaf_table_kernel<K><<<(unsigned)s->refit_stage[1], kRefitSlots, 0, s->ctx->stream>>>(
      s->nodes, s->refit_blocks, s->tets, s->leaf_verts, s->leaf_tet);
  s->ctx->launches++;
  return cudaGetLastError();
}

template <int K>
static cudaError_t preorder_impl(kdop_scene* s, int mesh, int64_t first, int64_t count, float* vol, int64_t* tet) {
  // nodes of a tree at depth d: 2^d down to L = floor(log2 n), then two per
  // two-tet node
  TreeBase b;
  int depth = 0;
  const int64_t n = s->t_off[mesh + 1] - s->t_off[mesh];
  while ((int64_t(2) << depth) <= n) ++depth;
  for (int d = 0; d <= depth; ++d) {
    int64_t at = s->level_off[d];
    for (int m = 0; m < mesh; ++m) {
      const int64_t k = s->t_off[m + 1] - s->t_off[m], full = int64_t(1) << d;
      at += k >= full ? full : std::max<int64_t>(0, 2 * k - full);
    }
    b.base[d] = (uint32_t)at;
  }
  const unsigned threads = (2u << depth) - 1u;
  preorder_kernel<K><<<(threads + 255) / 256, 256, 0, s->ctx->stream>>>(s->nodes, b, (uint32_t)n, depth,
                                                                       (uint32_t)s->t_off[mesh], first, count, vol, tet);
  s->ctx->launches++;
  return cudaGetLastError();
}

cudaError_t launch_preorder(kdop_scene* s, int mesh, int64_t first, int64_t count, float* vol, int64_t* tet) {
  switch (s->K) {
    case 6: return preorder_impl<6>(s, mesh, first, count, vol, tet);
    case 8: return preorder_impl<8>(s, mesh, first, count, vol, tet);
    case 12: return preorder_impl<12>(s, mesh, first, count, vol, tet);
    case 14: return preorder_impl<14>(s, mesh, first, count, vol, tet);
    case 18: return preorder_impl<18>(s, mesh, first, count, vol, tet);
    case 20: return preorder_impl<20>(s, mesh, first, count, vol, tet);
    case 26: return preorder_impl<26>(s, mesh, first, count, vol, tet);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_leaf_tables(kdop_scene* s) {
  switch (s->K) {
    case 6: return leaf_tables_impl<6>(s);
    case 8: return leaf_tables_impl<8>(s);
    case 12: return leaf_tables_impl<12>(s);
    case 14: return leaf_tables_impl<14>(s);
    case 18: return leaf_tables_impl<18>(s);
    case 20: return leaf_tables_impl<20>(s);
    case 26: return leaf_tables_impl<26>(s);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_refit(kdop_scene* s, int mode) {
  switch (s->K) {
    case 6: return refit_impl<6>(s, mode);
    case 8: return refit_impl<8>(s, mode);
    case 12: return refit_impl<12>(s, mode);
    case 14: return refit_impl<14>(s, mode);
    case 18: return refit_impl<18>(s, mode);
    case 20: return refit_impl<20>(s, mode);
    case 26: return refit_impl<26>(s, mode);
  }
  return cudaErrorInvalidValue;
}

template <int K>
static cudaError_t topo_impl(kdop_scene* s, const uint32_t* topo) {
  int64_t items = s->nn * NodeLayout<K>::NW;
  if (items == 0) return cudaSuccess;
  write_topology_kernel<K><<<(unsigned)((items + 255) / 256), 256, 0, s->ctx->stream>>>(s->nodes, s->nn, topo, s->surf);
  s->ctx->launches++;
  return cudaGetLastError();
}

cudaError_t launch_write_topology(kdop_scene* s, const uint32_t* topo) {
  switch (s->K) {
    case 6: return topo_impl<6>(s, topo);
    case 8: return topo_impl<8>(s, topo);
    case 12: return topo_impl<12>(s, topo);
    case 14: return topo_impl<14>(s, topo);
    case 18: return topo_impl<18>(s, topo);
    case 20: return topo_impl<20>(s, topo);
    case 26: return topo_impl<26>(s, topo);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_world(kdop_scene* s, int mode, float4* out) {
  if (s->nv == 0) return cudaSuccess;
  VertexSource vs = vertex_source(s, mode);
  world_kernel<<<(unsigned)((s->nv + 255) / 256), 256, 0, s->ctx->stream>>>(s->nv, vs, out);
  s->ctx->launches++;
  return cudaGetLastError();
}

cudaError_t launch_motion(kdop_scene* s) {
  int n = s->n_meshes > 0 ? s->n_meshes : 1;
  motion_kernel<<<(n + 127) / 128, 128, 0, s->ctx->stream>>>(s->n_meshes, s->quat, s->pos, s->lin_vel, s->ang_vel,
                                                              s->phase_dev, s->phase_rate);
  s->ctx->launches++;
  return cudaGetLastError();
}

}  // namespace kdop
