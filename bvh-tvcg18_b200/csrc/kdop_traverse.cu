// kdop_traverse.cu -- tandem (BVTT) traversal of mesh-pair trees.
//
// Reference semantics: kdop::details::traversal and kdop::tandem_traversal
// (SIMULATION/KDOP/KDOP/include/kdop_tandem_traversal.h:19-196): test the two
// root kDOPs (:164), then descend simultaneously; an overlapping pair of
// internal nodes expands into its 2 x 2 child pairs, an internal/leaf pair into
// 1 x 2 (:122-155); an overlapping leaf pair whose tets both have a boundary
// face (:56-88) goes to contact generation.  Overlap is the strict slab test
// of geometry_overlap_dop_dop.h:13-25 / geometry_overlap_interval_interval.h:
// 12-20.  The set of emitted tet pairs and the number of kDOP tests equal the
// reference's; only the emission order differs (sort for a canonical order).
//
// B200 design (replacing the OpenCL backlog kernel, cl/kernels/
// kdop_cl_tandem_traversal.cl:19-233, and the gProximity queues,
// cl/kernels/gproximity/*.cl):
//   * one persistent launch sized to the resident-block count; each warp owns
//     a node-pair deque in shared memory;
//   * "test on expand": a popped entry is a pair already known to overlap;
//     a few lanes take one entry together and read the children of both sides
//     as whole twin records (siblings' chunks interleaved, so one 256-bit load
//     per lane and chunk pair), test the four child pairs slab by slab, and
//     keep the overlapping ones (see traverse_kernel);
//   * ballot compaction: prefix sums over per-lane push counts pack the kept
//     pairs into the deque, and emitted leaf pairs reserve rows with one
//     atomic per warp;
//   * load balance: a seed pass expands the pairs (largest first) breadth first
//     into thousands of node pairs, which the warps claim a few at a time; a
//     warp whose deque is deep while other warps wait gives its oldest
//     (largest) entries to a global queue -- any deque with work gives half
//     while many warps wait; a deque overflow spills there too;
//   * termination: a global count of outstanding work units reaches zero;
//     every wait is bounded by a time limit after which the kernel records
//     DEV_ERR_TIMEOUT and returns (no unbounded spin).
#include <algorithm>
#include <cstring>
#include <mutex>

#include "kdop_device.cuh"
#include "kdop_sort.cuh"

namespace kdop {

struct TravArgs {
  const float4* __restrict__ nodes;
  const uint32_t* __restrict__ root;
  const uint2* __restrict__ pairs;
  uint32_t* candA;
  uint32_t* candB;
  uint32_t* candP;
  unsigned cand_cap;
  uint4* q_items;
  uint32_t* q_tags;
  unsigned q_cap;
  TravCtl* ctl;
  int stack_cap;  // power of two
  int init_chunk;
  int donate_min;
  int surface_filter;
  long long timeout_ns;
  unsigned n_meshes;
  const uint32_t* __restrict__ order;  // root pair i -> pair index (NULL: identity)
  const uint4* __restrict__ entries;   // when set: initial work = these deque entries (A, B, pair)
  int stuck;           // test hook: outstanding work units nobody completes
  unsigned poll_mask;  // queue counters polled on steps with (step & poll_mask) == 0
};

// Device buffers one traversal works in: pairs (input), candidates (output),
// work queue and control block (scratch).
struct TravBuffers {
  const uint2* pairs;
  const uint32_t* order;  // processing order of the pairs, or NULL
  const uint4* entries = nullptr;  // initial deque entries instead of root pairs (n_init of them)
  uint32_t* cand;  // 3 * cand_cap: A tets | B tets | pair ids
  int64_t cand_cap;
  uint4* q_items;
  uint32_t* q_tags;
  int64_t q_cap;
  TravCtl* ctl;
  uint4* seeds = nullptr;  // room for the seed pass's entries (seed_entries), or NULL: start from the root pairs
};

// 256-bit read-only load of two consecutive float4 chunks (p 32-byte aligned).
__device__ __forceinline__ void ldg256(const float4* p, float4& x, float4& y) {
  asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w), "=f"(y.x), "=f"(y.y), "=f"(y.z), "=f"(y.w)
               : "l"(p));
}
__device__ __forceinline__ unsigned ld_volatile(const unsigned* p) { return *(const volatile unsigned*)p; }
__device__ __forceinline__ int ld_volatile(const int* p) { return *(const volatile int*)p; }

// Overlap of two single nodes by one lane (the root test of a mesh pair): both
// records chunk by chunk; wa, wb get the records' word 0.
template <int K>
__device__ __forceinline__ bool node_overlap(const float4* __restrict__ nodes, uint32_t na, uint32_t nb,
                                             uint32_t& wa, uint32_t& wb) {
  using L = NodeLayout<K>;
  bool sep = false;
  wa = wb = 0;
#pragma unroll
  for (int j = 0; j < L::NW; ++j) {
    float4 A = __ldg(nodes + L::at(na, j)), B = __ldg(nodes + L::at(nb, j));
    if (2 * j < L::NS) sep |= (A.y < B.x) || (B.y < A.x);
    if (2 * j + 1 < L::NS) sep |= (A.w < B.z) || (B.w < A.z);
    if (j == L::TOPO_CHUNK) {
      wa = L::word0(A);
      wb = L::word0(B);
    }
  }
  return !sep;
}

// Waiting warps from which on every deque with work donates (tail mode).
constexpr int kTailWaiting = 512;

// Warp total and exclusive prefix of per-lane counts below 2^BITS, one
// ballot per bit.
template <int BITS>
__device__ __forceinline__ void warp_prefix(int v, unsigned lt_mask, int& total, int& excl) {
  total = excl = 0;
#pragma unroll
  for (int k = 0; k < BITS; ++k) {
    unsigned m = __ballot_sync(0xffffffffu, (v >> k) & 1);
    total += __popc(m) << k;
    excl += __popc(m & lt_mask) << k;
  }
}

// Tet of a leaf node (word 1 of its record).
template <int K>
__device__ __forceinline__ uint32_t leaf_tet(const float4* __restrict__ nodes, uint32_t w) {
  using L = NodeLayout<K>;
  return L::word1(__ldg(nodes + L::at(w & NODE_MASK, L::TOPO_CHUNK)));
}

// Lanes per deque entry: chunk pairs of a record over C chunks per lane,
// rounded up to a power of two so that entries sit on aligned lane groups.
template <int K, int C>
struct Coop {
  static constexpr int NW = NodeLayout<K>::NW;
  static constexpr int Q0 = (NW + C - 1) / C;
  static constexpr int Q = Q0 <= 1 ? 1 : Q0 <= 2 ? 2 : Q0 <= 4 ? 4 : 8;
  static constexpr int E = 32 / Q;             // entries per sub-batch
  static constexpr int PM = (4 + Q - 1) / Q;   // child pairs per lane
};

// The slab tests of one lane: on the lane's chunks of both children of each
// side, separation of child pairs (0,0), (0,1), (1,0), (1,1) in s, and word 0
// of the four children (A0, A1, B0, B1) in t on the lane holding the topology
// chunk.
template <int K, int C>
__device__ __forceinline__ void test_twins(const float4 (&A0)[C], const float4 (&A1)[C], const float4 (&B0)[C],
                                           const float4 (&B1)[C], int gq, bool (&s)[4], uint32_t (&t)[4]) {
  using L = NodeLayout<K>;
  constexpr int Q = Coop<K, C>::Q, TR = L::TOPO_CHUNK / Q;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    s[c] = false;
    t[c] = 0u;
  }
#pragma unroll
  for (int r = 0; r < C; ++r) {
    const int j = gq + Q * r;
    const float4 a0 = A0[r], a1 = A1[r], b0 = B0[r], b1 = B1[r];
    if (2 * j < L::NS) {
      s[0] = s[0] || (a0.y < b0.x) || (b0.y < a0.x);
      s[1] = s[1] || (a0.y < b1.x) || (b1.y < a0.x);
      s[2] = s[2] || (a1.y < b0.x) || (b0.y < a1.x);
      s[3] = s[3] || (a1.y < b1.x) || (b1.y < a1.x);
    }
    if (2 * j + 1 < L::NS) {
      s[0] = s[0] || (a0.w < b0.z) || (b0.w < a0.z);
      s[1] = s[1] || (a0.w < b1.z) || (b1.w < a0.z);
      s[2] = s[2] || (a1.w < b0.z) || (b0.w < a1.z);
      s[3] = s[3] || (a1.w < b1.z) || (b1.w < a1.z);
    }
    if (r == TR) {
      t[0] = L::word0(a0);
      t[1] = L::word0(a1);
      t[2] = L::word0(b0);
      t[3] = L::word0(b1);
    }
  }
}

// What becomes of a lane's child pairs c = gq + Q r (c = 2 i + k: child i of
// A, child k of B) of the entry (xa, xb): pushed, emitted, counted.  A single
// side is the node itself, which is side (x & 1) of the twin loaded: the
// pairs with the other side are absent.  The verdicts of the entry's lanes
// come together by one ballot per child pair (a shuffle would go through the
// L1 data pipe, the kernel's busiest unit).  Called by whole warps.
template <int K, int C>
__device__ __forceinline__ void child_pairs(uint32_t xa, uint32_t xb, bool valid, const bool (&s)[4],
                                            const uint32_t (&t)[4], int ge, int gq, unsigned group_mask, uint32_t need,
                                            bool* push, bool* emit, uint32_t* pushA, uint32_t* pushB,
                                            unsigned& tests32, unsigned& lo32) {
  using L = NodeLayout<K>;
  using CP = Coop<K, C>;
  constexpr int Q = CP::Q, PM = CP::PM;
  constexpr int TQ = L::TOPO_CHUNK % Q;  // lane holding topology
  const unsigned m0 = __ballot_sync(0xffffffffu, s[0]), m1 = __ballot_sync(0xffffffffu, s[1]);
  const unsigned m2 = __ballot_sync(0xffffffffu, s[2]), m3 = __ballot_sync(0xffffffffu, s[3]);
  // word 0 of the four children, from the lane holding the topology chunk
  const int src = ge * Q + TQ;
  const uint32_t wA0 = __shfl_sync(0xffffffffu, t[0], src);
  const uint32_t wA1 = __shfl_sync(0xffffffffu, t[1], src);
  uint32_t wB0, wB1;
  if (Q == 2) {
    // lane gq only handles child gq of B: the topology lane keeps its own
    // word, the other lane gets the other child's
    const uint32_t wo = __shfl_sync(0xffffffffu, TQ ? t[2] : t[3], src);
    wB0 = wB1 = (gq == TQ) ? (TQ ? t[3] : t[2]) : wo;
  } else {
    wB0 = __shfl_sync(0xffffffffu, t[2], src);
    wB1 = __shfl_sync(0xffffffffu, t[3], src);
  }
  const bool singleA = (xa & LEAF_BIT) != 0, singleB = (xb & LEAF_BIT) != 0;
#pragma unroll
  for (int r = 0; r < PM; ++r) {
    const int c = gq + Q * r;
    const int ci = (Q == 2) ? r : (c >> 1), ck = (Q == 2) ? gq : (c & 1);
    const uint32_t wa = ci ? wA1 : wA0, wb = ck ? wB1 : wB0;
    const unsigned mc = ci ? (ck ? m3 : m2) : (ck ? m1 : m0);
    const bool there = valid && (Q * r + Q - 1 < 4 || c < 4) && !(singleA && (int)(xa & 1u) != ci) &&
                       !(singleB && (int)(xb & 1u) != ck);
    const bool ok = there && (mc & group_mask) == 0u;
    const uint32_t both = wa & wb;
    const bool leaf = ok && (both & LEAF_BIT);
    if (there) tests32 += 1u;
    if (leaf) lo32 += 1u;
    push[r] = ok && !(both & LEAF_BIT);
    emit[r] = leaf && (both & need) == need;
    pushA[r] = wa;
    pushB[r] = wb;
  }
}

// A candidate row for the leaves of words wa, wb at position `at`.
template <int K>
__device__ __forceinline__ void put_candidate(const TravArgs& a, unsigned at, uint32_t wa, uint32_t wb, uint32_t pid) {
  if (at < a.cand_cap) {
    a.candA[at] = leaf_tet<K>(a.nodes, wa);
    a.candB[at] = leaf_tet<K>(a.nodes, wb);
    a.candP[at] = pid;
  }
}

// Root test of mesh pair pid (kdop_tandem_traversal.h:164), then the
// traversal's own test of the root pair (:42), both counted as the reference
// does.  True when the pair is to be expanded (wa, wb its entry).
template <int K>
__device__ __forceinline__ bool root_pair(const TravArgs& a, uint32_t pid, uint32_t& wa, uint32_t& wb,
                                          unsigned& tests32, unsigned& lo32) {
  const uint2 mp = a.pairs[pid];
  if (mp.x >= a.n_meshes || mp.y >= a.n_meshes) {
    atomicOr(&a.ctl->error, DEV_ERR_BAD_INDEX);
    return false;
  }
  const uint32_t ra = a.root[mp.x], rb = a.root[mp.y];
  if (ra == NO_NODE || rb == NO_NODE) return false;
  const bool ov = node_overlap<K>(a.nodes, ra, rb, wa, wb);
  tests32 += ov ? 2u : 1u;
  if (!ov || !(wa & wb & LEAF_BIT)) return ov;
  lo32 += 1u;
  if (!a.surface_filter || (wa & wb & SURF_BIT)) put_candidate<K>(a, atomicAdd(&a.ctl->n_cand, 1u), wa, wb, pid);
  return false;
}

// Claims of the seed pass's entries: this many at most per claim (a deque
// takes them in one go), fewer towards the end (guided self-scheduling).
// Claims of one entry cost small launches an atomic per expansion (a pair of
// 6,000 tets: 114 us, 81 us with up to 4), claims of up to 16 leave long tails
// (256 touching pairs: 500 against 435 us; a pair of 1.6 M tets: 979 against
// 886 us).
constexpr unsigned kMaxClaim = 4;
__device__ __forceinline__ unsigned claim_size(unsigned left, unsigned warps) {
  return min(max(left / (2u * warps), 1u), kMaxClaim);
}

// Deque entries (X, Y, pair): X and Y overlap and their children are to be
// tested.  A side with LEAF_BIT is the single node X & NODE_MASK (a leaf);
// otherwise X is the first child of an internal node, whose children X, X + 1
// form one twin record.  Word 0 of a child's record is its entry value.
//
// Cooperative expansion: Q lanes take one entry (E = 32 / Q entries per
// sub-batch).  Lane q reads chunks j = q, q + Q, ... (C of them) of both
// children of each side, one 256-bit load per chunk and side (twin records
// interleave the siblings' chunks), so the lanes of an entry read whole
// 128-byte lines (k = 14) and a warp-wide load touches E lines instead of 32.
// The lane tests its slabs for the four child pairs; a ballot over the
// entry's lanes combines the verdicts; the lane holding the topology chunk
// broadcasts the children's word 0; lane q then handles child pairs q, q + Q.
// Bound: the L1 data pipe (82 % of its peak at k = 14; a 256-bit load passes
// each 128-byte line it touches twice), then the ALU pipe (56 %); 3.1 warp
// instructions per node-pair test, 4.6 before.  A deque holding one pair
// only (no pair index beside its entries: 8 instead of 12 bytes of shared
// memory, the rest of the array caches records), verdicts combined by ballots
// instead of shuffles, and the refill, root test and donation polls outside
// the step took the batched workload (1.96 G tests, k = 14) from 11.28 to 9.6
// ms, and to 9.4 with the lanes beyond the last entry repeating its loads.
// S sub-batches are loaded together per step, and one compaction per step
// packs the pushes of all of them.
//
// SEEDED: starts from the seed pass's entries.  Otherwise a warp claims
// init_chunk root pairs (tested one per lane) or entries of a caller's frontier
// at a time.  They lie at the bottom of its deque, each with a pair index of its
// own beside it, until they are begun, so that waiting warps can be given them
// like any other entry.  (Held back one by one instead, a claim of 32 took 64
// touching pairs of 6,000 tets from 213 to 1,322 us, and used up the queue of
// the call that cannot grow it.)
template <int K, int C, int S, bool SEEDED>
__global__ void __launch_bounds__(512, (C * S >= 4) ? 1 : 2) traverse_kernel(TravArgs a) {
  using L = NodeLayout<K>;
  using CP = Coop<K, C>;
  constexpr int NW = L::NW;
  constexpr int Q = CP::Q, E = CP::E, PM = CP::PM;
  constexpr int SLOTS = PM * S;                     // pushes per lane per step
  constexpr int CBITS = SLOTS <= 1 ? 1 : SLOTS <= 3 ? 2 : SLOTS <= 7 ? 3 : 4;  // bits of a lane's emit count
  extern __shared__ uint32_t smem[];
  __shared__ uint2 s_claim[SEEDED ? 16 : 1];  // per warp: claimed initial work not yet taken [x, y)
  __shared__ unsigned s_first;
  __shared__ uint32_t s_pair[SEEDED ? 1 : 16 * 32];  // per warp: pairs of the claimed entries, by deque position
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int ge = lane / Q, gq = lane % Q;  // entry and chunk lane of this lane
  const float4* __restrict__ nodes_q = a.nodes + 2 * gq;  // chunk gq of twin 0
  const unsigned lt_mask = (1u << lane) - 1u;
  const unsigned group_mask = ((1u << Q) - 1u) << (ge * Q);  // lanes of this lane's entry
  const int CAP = a.stack_cap;
  const int MASK = CAP - 1;
  uint2* sAB = reinterpret_cast<uint2*>(smem) + (size_t)wib * CAP;  // this warp's deque
  TravCtl* ctl = a.ctl;
  if (SEEDED && ctl->n_init == 0u && a.stuck == 0) return;  // the seed pass finished every pair
  // A block that starts takes a first claim of the seeded entries for each of its
  // warps at once (an atomic per block, not per warp).  All claims come off the
  // one counter, so that entries belong to running warps only: a block that
  // waits for a place on an SM another stream uses owns nothing the running ones
  // would wait for.
  auto first_claim = [&](unsigned n_init) {
    return max(claim_size(n_init, gridDim.x * (blockDim.x >> 5)), (unsigned)a.init_chunk);
  };
  bool init_done = false;
  if (SEEDED) {
    const unsigned n_init = ctl->n_init, first = first_claim(n_init);
    if (threadIdx.x == 0) s_first = atomicAdd(&ctl->init_head, first * (blockDim.x >> 5));
    __syncthreads();
    const unsigned own = min(s_first + (unsigned)wib * first, n_init);
    if (lane == 0) s_claim[wib] = make_uint2(own, min(own + first, n_init));
    __syncwarp();
    init_done = own >= n_init;
  }

  int top = 0, bot = 0;  // deque [bot, top) in virtual positions
  int begun = 0;         // not SEEDED: [bot, begun) are claimed entries of a pair each
  int release = 0;       // work units taken and not yet released
  unsigned claim = 0xFFFFFFFFu;
  // per-lane counts, added to the control block's 64-bit totals every 1024
  // steps and at the end (at most 4 per lane and step: no overflow)
  unsigned tests32 = 0, lo32 = 0;
  auto fold_counts = [&]() {
    unsigned t = tests32, l = lo32;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      t += __shfl_down_sync(0xffffffffu, t, o);
      l += __shfl_down_sync(0xffffffffu, l, o);
    }
    if (lane == 0) {
      if (t) atomicAdd(&ctl->tests, (unsigned long long)t);
      if (l) atomicAdd(&ctl->leaf_overlaps, (unsigned long long)l);
    }
    tests32 = lo32 = 0;
  };
  // Pair index of the deque's entries (from `begun` on).  A deque is filled from
  // one root pair, one queue item or frontier entries of one pair, and entries
  // inherit their parent's pair, so it holds a single pair at any time
  // (warp-uniform).
  uint32_t curP = 0;
  const uint32_t need = a.surface_filter ? SURF_BIT : 0u;  // word bits an emitted leaf pair has to share

  unsigned step = 0;
  for (;;) {
    if (!SEEDED) ++step;
    if (top == bot) {
      // Work handed to the queue was counted before it was published, so the
      // release needs no fence.
      if (release) {
        if (lane == 0) atomicSub(&ctl->work, release);
        release = 0;
      }
      if (SEEDED && !init_done) {
        uint2 r = s_claim[wib];
        __syncwarp();
        if (r.x == r.y) {
          // what is left when every block has its first claim, at most
          const unsigned n_init = ctl->n_init, warps = gridDim.x * (blockDim.x >> 5);
          const unsigned left = n_init - min(n_init, max(r.y, warps * first_claim(n_init)));
          const unsigned chunk = max((unsigned)a.init_chunk, claim_size(left, warps));
          unsigned base = 0;
          if (lane == 0) base = atomicAdd(&ctl->init_head, chunk);
          base = min(__shfl_sync(0xffffffffu, base, 0), n_init);
          init_done = base >= n_init;
          r = make_uint2(base, min(base + chunk, n_init));
        }
        if (!init_done) {
          // pending node pairs of a frontier (their tests are counted already):
          // the claim's leading run of one pair
          const bool in = r.x + lane < r.y;
          uint4 e = make_uint4(0u, 0u, 0u, 0u);
          if (in) e = a.entries[r.x + lane];
          curP = __shfl_sync(0xffffffffu, e.z, 0);
          const unsigned same = __ballot_sync(0xffffffffu, in && e.z == curP);
          const int run = (same == 0xffffffffu) ? 32 : __ffs(~same) - 1;
          if (lane < run) sAB[(top + lane) & MASK] = make_uint2(e.x, e.y);
          top += run;
          release += run;
          r.x += (unsigned)run;
          if (lane == 0) s_claim[wib] = r;
          __syncwarp();
          continue;
        }
      }
      if (!SEEDED && !init_done) {
        unsigned first = 0;
        if (lane == 0) first = atomicAdd(&ctl->init_head, (unsigned)a.init_chunk);
        first = __shfl_sync(0xffffffffu, first, 0);
        const unsigned n_init = ctl->n_init;
        init_done = first >= n_init;
        if (!init_done) {
          const int n = (int)min((unsigned)a.init_chunk, n_init - first);
          uint32_t wa = 0, wb = 0, pid = 0;
          bool there = lane < n;
          if (there && a.entries) {
            const uint4 e = a.entries[first + lane];
            wa = e.x;
            wb = e.y;
            pid = e.z;
          } else if (there) {
            pid = ctl->pair_base + first + lane;
            if (a.order) pid = a.order[pid];
            there = root_pair<K>(a, pid, wa, wb, tests32, lo32);
          }
          const unsigned m = __ballot_sync(0xffffffffu, there);
          if (there) {
            const int at = top + __popc(m & lt_mask);
            sAB[at & MASK] = make_uint2(wa, wb);
            s_pair[wib * 32 + (at & 31)] = pid;
          }
          release += n;
          top += __popc(m);
          begun = top;
          __syncwarp();
          continue;
        }
      }
      // wait for a queue item or the end of all work
      if (claim == 0xFFFFFFFFu) {
        unsigned c = 0;
        if (lane == 0) c = atomicAdd(&ctl->q_head, 1u);
        claim = __shfl_sync(0xffffffffu, c, 0);
      }
      unsigned long long t0 = global_ns();
      unsigned backoff = 64;
      int got = 0, failed = 0;
      for (unsigned it = 0;; ++it) {
        if (claim < a.q_cap && ld_volatile(&a.q_tags[claim]) != 0u) {
          got = 1;
          break;
        }
        // the end-of-work counter is polled by every waiting warp: every
        // 4th round only, to keep its line free for the workers' atomics
        if ((it & 3u) == 0u && ld_volatile(&ctl->work) == 0) break;
        if ((long long)(global_ns() - t0) > a.timeout_ns) {
          failed = 1;
          break;
        }
        __nanosleep(backoff);
        backoff = min(backoff * 2u, 2048u);
      }
      got = __shfl_sync(0xffffffffu, got, 0);
      failed = __shfl_sync(0xffffffffu, failed, 0);
      if (failed && lane == 0) atomicOr(&ctl->error, DEV_ERR_TIMEOUT);
      if (failed || !got) break;
      __threadfence();
      uint4 it = __ldcg(a.q_items + claim);
      if (lane == 0) {
        a.q_tags[claim] = 0u;
        sAB[top & MASK] = make_uint2(it.x, it.y);
      }
      curP = it.z;  // the deque was empty: one pair
      top += 1;
      release += 1;
      claim = 0xFFFFFFFFu;
      __syncwarp();
      continue;
    }

    // ---- one step: expand up to E * S entries from the top of the deque ----
    // this step's pushes (entry words) and emitted leaf pairs (node words)
    bool push[SLOTS], emit[SLOTS];
    uint32_t pushA[SLOTS], pushB[SLOTS];
    const bool had_two = SEEDED || top - bot >= 2;
    {
      if (!SEEDED && top == begun) curP = s_pair[wib * 32 + (--begun & 31)];
      const int n = min(E * S, top - (SEEDED ? bot : begun));
      top -= n;
      uint2 eab[S];
      float4 A0[S][C], A1[S][C], B0[S][C], B1[S][C];
#pragma unroll
      for (int b = 0; b < S; ++b) {
        // a lane without an entry loads the last one's records again (no line
        // of its own) and its verdicts are not used
        eab[b] = sAB[(top + min(b * E + ge, n - 1)) & MASK];
        const float4* pa = nodes_q + (size_t)((eab[b].x & NODE_MASK) >> 1) * (2 * NW);
        const float4* pb = nodes_q + (size_t)((eab[b].y & NODE_MASK) >> 1) * (2 * NW);
#pragma unroll
        for (int r = 0; r < C; ++r) {
          const int j = gq + Q * r;
          if (j < NW) {
            ldg256(pa + 2 * Q * r, A0[b][r], A1[b][r]);
            ldg256(pb + 2 * Q * r, B0[b][r], B1[b][r]);
          }
        }
      }
      __syncwarp();  // entries read before this step's pushes overwrite them
#pragma unroll
      for (int b = 0; b < S; ++b) {
        const bool valid = b * E + ge < n;
        const uint32_t xa = eab[b].x, xb = eab[b].y;
        bool sep[4];
        uint32_t words[4];
        test_twins<K, C>(A0[b], A1[b], B0[b], B1[b], gq, sep, words);
        child_pairs<K, C>(xa, xb, valid, sep, words, ge, gq, group_mask, need, push + b * PM, emit + b * PM,
                          pushA + b * PM, pushB + b * PM, tests32, lo32);
      }
    }

    // ---- emits (rare): leaf pairs to candidate rows, one atomic per warp ----
    bool any_emit = false;
#pragma unroll
    for (int k = 0; k < SLOTS; ++k) any_emit |= emit[k];
    if (__any_sync(0xffffffffu, any_emit)) {
      int ne = 0, tot_e = 0, off_e = 0;
#pragma unroll
      for (int k = 0; k < SLOTS; ++k) ne += emit[k] ? 1 : 0;
      warp_prefix<CBITS>(ne, lt_mask, tot_e, off_e);
      unsigned base = 0;
      if (lane == 0) base = atomicAdd(&ctl->n_cand, (unsigned)tot_e);
      base = __shfl_sync(0xffffffffu, base, 0) + (unsigned)off_e;
#pragma unroll
      for (int k = 0; k < SLOTS; ++k) {
        if (emit[k]) put_candidate<K>(a, base++, pushA[k], pushB[k], curP);
      }
    }
    // ---- pushes: deque (or the global queue), slot-major: every lane's
    // slot-0 push, then every slot-1 push, ..., so that the lanes of one store
    // instruction write consecutive positions (one ballot per slot) ----
    {
      unsigned pm[SLOTS];
      int pbase[SLOTS];
      int tot_p = 0;
#pragma unroll
      for (int k = 0; k < SLOTS; ++k) {
        pm[k] = __ballot_sync(0xffffffffu, push[k]);
        pbase[k] = tot_p;
        tot_p += __popc(pm[k]);
      }
      if (top - bot + tot_p <= CAP) {
#pragma unroll
        for (int k = 0; k < SLOTS; ++k)
          if (push[k])
            sAB[(top + pbase[k] + __popc(pm[k] & lt_mask)) & MASK] = make_uint2(pushA[k], pushB[k]);
        top += tot_p;
      } else {
        // deque full: the new entries go to the global queue
        unsigned t0 = 0;
        if (lane == 0) t0 = atomicAdd(&ctl->q_tail, (unsigned)tot_p);
        t0 = __shfl_sync(0xffffffffu, t0, 0);
        int room = (int)min((unsigned long long)tot_p,
                            (t0 < a.q_cap) ? (unsigned long long)(a.q_cap - t0) : 0ull);
        if (room < tot_p && lane == 0) atomicOr(&ctl->error, DEV_ERR_QUEUE_FULL);
        if (room > 0 && lane == 0) atomicAdd(&ctl->work, room);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < SLOTS; ++k) {
          const unsigned slot = t0 + (unsigned)(pbase[k] + __popc(pm[k] & lt_mask));
          if (push[k] && slot < t0 + (unsigned)room) a.q_items[slot] = make_uint4(pushA[k], pushB[k], curP, 0u);
        }
        __threadfence();
        __syncwarp();
#pragma unroll
        for (int k = 0; k < SLOTS; ++k) {
          const unsigned slot = t0 + (unsigned)(pbase[k] + __popc(pm[k] & lt_mask));
          if (push[k] && slot < t0 + (unsigned)room) atomicExch(&a.q_tags[slot], 1u);
        }
      }
    }

    // ---- donation: give the oldest entries to waiting warps ----
    // The queue counters are polled on every (poll_mask + 1)-th step.  A deep
    // deque gives to any waiting warp; while many warps wait (the tail of the
    // traversal) any deque with two or more entries gives half.
    if (SEEDED) ++step;
    if ((step & a.poll_mask) == 0u) {
      if ((step & 1023u) == 0u) fold_counts();
      const int depth = top - bot;
      if (depth >= 2 && had_two) {
        int waiting = 0;
        if (lane == 0) {
          const unsigned q_h = ld_volatile(&ctl->q_head), q_t = ld_volatile(&ctl->q_tail);
          waiting = (q_h > q_t) ? (int)min(q_h - q_t, 1024u) : 0;
        }
        waiting = __shfl_sync(0xffffffffu, waiting, 0);
        int d = (depth >= a.donate_min || waiting >= kTailWaiting) ? min(min(waiting, 32), depth / 2) : 0;
        if (d > 0) {
          __syncwarp();  // this step's pushes, before other lanes read them
          unsigned t0 = 0;
          if (lane == 0) t0 = atomicAdd(&ctl->q_tail, (unsigned)d);
          t0 = __shfl_sync(0xffffffffu, t0, 0);
          int room = (int)min((unsigned long long)d, (t0 < a.q_cap) ? (unsigned long long)(a.q_cap - t0) : 0ull);
          if (room < d && lane == 0) atomicOr(&ctl->error, DEV_ERR_QUEUE_FULL);
          if (room > 0 && lane == 0) atomicAdd(&ctl->work, room);
          __syncwarp();
          if (lane < room) {
            uint2 ab = sAB[(bot + lane) & MASK];
            const uint32_t pid = SEEDED || bot + lane >= begun ? curP : s_pair[wib * 32 + ((bot + lane) & 31)];
            a.q_items[t0 + lane] = make_uint4(ab.x, ab.y, pid, 0u);
          }
          __threadfence();
          __syncwarp();
          if (lane < room) atomicExch(&a.q_tags[t0 + lane], 1u);
          // entries that found no room stay lost only with DEV_ERR_QUEUE_FULL set
          bot += d;
          begun = max(begun, bot);
        }
      }
    }
    __syncwarp();
  }

  // ---- totals ----
  fold_counts();
}

// ---- seed pass ----------------------------------------------------------------
// Breadth-first expansion of the top of the node-pair trees, so that the
// persistent traversal starts from thousands of node pairs instead of the root
// pairs.  Starting from few roots, the traversal hands work on through the
// global queue one donation at a time, a chain of atomics, polls and record
// loads per generation: a launch of one pair of 6,000 tets spent most of its
// 149 us on that, with 4,700 of its 4,736 warps waiting.  Here a block takes
// `group` pairs (their root tests one per thread) or, in the second pass,
// an even share of the first pass's node pairs, and expands them level by
// level in shared memory until at least kSeedStop are pending, which it
// appends to the frontier; a block whose pairs end earlier leaves nothing.
// The traversal claims the frontier's entries in order.  Tests, leaf pairs
// and candidates are those of the same expansions done by the traversal.
// Measured, whole traversal call without -> with this pass and the loop below:
// one pair of 6,000 tets 149 -> 81 us, of 24,576 tets in touch 138 -> 51 us,
// 64 deforming pairs of 384 k tets 1,027 -> 477 us, 256 touching pairs of 48 k
// tets 668 -> 435 us.  Stopping at 128 or 1024 pending pairs instead of 512:
// 537 and 578 us on the 64 pairs, 490 and 472 us on the 256.
constexpr unsigned kSeedStop = 512;
constexpr unsigned kSeedCap = 4 * kSeedStop;  // most a level of fewer than kSeedStop pairs leaves
constexpr int kSeedThreads = 512;
constexpr int64_t kSeedTwiceMax = 64, kSeedTwiceTets = 4096;

// ---- order of the root pairs ----------------------------------------------------
// Pairs by decreasing size (tets of both meshes), equal sizes in list order.
struct PairSizeGen {
  const uint2* pairs;
  const uint32_t* t_off;
  uint32_t most;  // tets of the two largest meshes at least
  __device__ uint64_t key(int64_t i) const {
    const uint2 m = pairs[i];
    return most - (t_off[m.x + 1] - t_off[m.x]) - (t_off[m.y + 1] - t_off[m.y]);
  }
  __device__ uint32_t val(int64_t i) const { return (uint32_t)i; }
};
// Work of that sort, in the seed pass's buffer (free until the traversal).
struct PairOrderWork {
  size_t keys, keys_tmp, vals, vals_tmp, scratch, total;
  explicit PairOrderWork(int64_t n) {
    size_t at = 0;
    auto take = [&](size_t b) {
      size_t o = at;
      at += (b + 255) & ~(size_t)255;
      return o;
    };
    keys = take((size_t)n * 8);
    keys_tmp = take((size_t)n * 8);
    vals = take((size_t)n * 4);
    vals_tmp = take((size_t)n * 4);
    scratch = take(radix_scratch_words(n) * 4);
    total = at;
  }
};

cudaError_t launch_pair_order(kdop_scene* s, int64_t n, uint32_t most, long long wait_ns) {
  char* w = reinterpret_cast<char*>(s->seeds);
  const PairOrderWork L(n);
  SortBuffers b{reinterpret_cast<uint64_t*>(w + L.keys), reinterpret_cast<uint64_t*>(w + L.keys_tmp),
                reinterpret_cast<uint32_t*>(w + L.vals), reinterpret_cast<uint32_t*>(w + L.vals_tmp)};
  // a sort wait that gave up leaves an incomplete order: every place starts as
  // a valid pair index, and the traversals over this order report the error
  cudaError_t e = cudaMemsetAsync(&s->ctl->order_error, 0, 4, s->ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(w + L.vals, 0, L.scratch - L.vals, s->ctx->stream);
  if (e == cudaSuccess)
    e = radix_sort(s->ctx, PairSizeGen{s->pairs, s->t_off_dev, most}, n, bits_of(most), b, w + L.scratch,
                   WaitLimit(&s->ctl->order_error, wait_ns));
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(s->pair_order, b.vals, (size_t)n * 4, cudaMemcpyDeviceToDevice, s->ctx->stream);
  return e;
}

// Pairs per block of the first pass: four blocks per SM until a group fills
// a block's list.
static int64_t seed_group(int sm_count, int64_t n_pairs) {
  const int64_t blocks = 4 * (int64_t)sm_count;
  return std::min<int64_t>(std::max<int64_t>((n_pairs + blocks - 1) / blocks, 1), kSeedCap);
}
// Few pairs leave too few node pairs for 4,736 warps after one pass: they are
// expanded once more, over two blocks per SM (one pair of 1.6 M tets 1,250 us
// with one pass, 1,022 with two; 64 pairs 601 and 560 us, 256 pairs 455 and
// 471 us, each against the same loop).
// Pairs of fewer than kSeedTwiceTets tets in all end in the first pass or soon
// after it (a touching pair of 384 tets 198 -> 187 us without the second launch
// and with the poses packed by one).
static int seed_blocks2(int sm_count, int64_t n_pairs, int64_t tets) {
  return n_pairs <= kSeedTwiceMax && tets >= kSeedTwiceTets ? 2 * sm_count : 0;
}

// Entries the first pass can leave: kSeedCap per group of pairs.
static int64_t seed_entries1(int sm_count, int64_t n) {
  return std::max(std::min<int64_t>(n, 4 * (int64_t)sm_count), (n + kSeedCap - 1) / kSeedCap) * kSeedCap;
}
int64_t seed_entries(int sm_count, int64_t n) {
  const int64_t seeds = seed_entries1(sm_count, n) + (int64_t)seed_blocks2(sm_count, 1, kSeedTwiceTets) * kSeedCap;
  return std::max(seeds, (int64_t)(PairOrderWork(n).total / sizeof(uint4)) + 1);  // the pair order's work, before
}

template <int K>
__global__ void __launch_bounds__(kSeedThreads) seed_kernel(TravArgs a, unsigned n_pairs, unsigned group,
                                                            const uint4* __restrict__ in,
                                                            const unsigned* __restrict__ in_count, uint4* out,
                                                            unsigned* out_count) {
  constexpr int C = 2;
  using CP = Coop<K, C>;
  constexpr int NW = NodeLayout<K>::NW, Q = CP::Q, E = CP::E, PM = CP::PM;
  extern __shared__ uint32_t smem[];
  __shared__ unsigned cnt[2], flush_at;
  // two lists of (A, B) words and of pair indices, read and written in turn
  uint2* const AB = reinterpret_cast<uint2*>(smem);
  uint32_t* const P = smem + 4 * kSeedCap;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const unsigned lt_mask = (1u << lane) - 1u;
  const int ge = lane / Q, gq = lane % Q;
  const unsigned group_mask = ((1u << Q) - 1u) << (ge * Q);
  const float4* __restrict__ nodes_q = a.nodes + 2 * gq;
  const uint32_t need = a.surface_filter ? SURF_BIT : 0u;
  TravCtl* ctl = a.ctl;
  unsigned tests32 = 0, lo32 = 0;
  unsigned n_src = n_pairs;
  if (in) {
    n_src = *in_count;
    group = min((n_src + gridDim.x - 1) / gridDim.x, kSeedCap);
  }
  for (unsigned long long base = (unsigned long long)blockIdx.x * group; base < n_src;
       base += (unsigned long long)gridDim.x * group) {
    const unsigned n = (unsigned)min((unsigned long long)group, n_src - base);
    if (threadIdx.x < 2) cnt[threadIdx.x] = (in && threadIdx.x == 0) ? n : 0u;
    __syncthreads();
    for (unsigned i = threadIdx.x; i < n; i += blockDim.x) {
      if (in) {
        const uint4 e = in[base + i];
        AB[i] = make_uint2(e.x, e.y);
        P[i] = e.z;
      } else {
        const uint32_t pid = a.order[base + i];
        uint32_t wa = 0, wb = 0;
        if (root_pair<K>(a, pid, wa, wb, tests32, lo32)) {
          const unsigned at = atomicAdd(&cnt[0], 1u);
          AB[at] = make_uint2(wa, wb);
          P[at] = pid;
        }
      }
    }
    __syncthreads();
    unsigned cur = 0, c = cnt[0];
    while (c > 0 && c < kSeedStop) {
      const unsigned nx = cur ^ 1u;
      for (unsigned i0 = wib * E; i0 < c; i0 += nw * E) {
        const unsigned i = i0 + ge;
        const bool valid = i < c;
        const uint2 x = AB[cur * kSeedCap + min(i, c - 1)];
        const uint32_t pid = P[cur * kSeedCap + min(i, c - 1)];
        const float4* pa = nodes_q + (size_t)((x.x & NODE_MASK) >> 1) * (2 * NW);
        const float4* pb = nodes_q + (size_t)((x.y & NODE_MASK) >> 1) * (2 * NW);
        float4 A0[C], A1[C], B0[C], B1[C];
#pragma unroll
        for (int r = 0; r < C; ++r)
          if (gq + Q * r < NW) {
            ldg256(pa + 2 * Q * r, A0[r], A1[r]);
            ldg256(pb + 2 * Q * r, B0[r], B1[r]);
          }
        bool sep[4], push[PM], emit[PM];
        uint32_t words[4], pa_w[PM], pb_w[PM];
        test_twins<K, C>(A0, A1, B0, B1, gq, sep, words);
        child_pairs<K, C>(x.x, x.y, valid, sep, words, ge, gq, group_mask, need, push, emit, pa_w, pb_w, tests32,
                          lo32);
#pragma unroll
        for (int r = 0; r < PM; ++r) {
          const unsigned pm = __ballot_sync(0xffffffffu, push[r]);
          if (pm) {
            unsigned at = 0;
            if (lane == 0) at = atomicAdd(&cnt[nx], (unsigned)__popc(pm));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(pm & lt_mask);
            if (push[r]) {
              AB[nx * kSeedCap + at] = make_uint2(pa_w[r], pb_w[r]);
              P[nx * kSeedCap + at] = pid;
            }
          }
          const unsigned em = __ballot_sync(0xffffffffu, emit[r]);
          if (em) {
            unsigned at = 0;
            if (lane == 0) at = atomicAdd(&ctl->n_cand, (unsigned)__popc(em));
            at = __shfl_sync(0xffffffffu, at, 0) + __popc(em & lt_mask);
            if (emit[r]) put_candidate<K>(a, at, pa_w[r], pb_w[r], pid);
          }
        }
      }
      __syncthreads();
      cur = nx;
      c = cnt[cur];
      if (threadIdx.x == 0) cnt[cur ^ 1u] = 0;
      __syncthreads();
    }
    if (c > 0) {
      if (threadIdx.x == 0) {
        flush_at = atomicAdd(out_count, c);
        if (out_count == &ctl->n_init) atomicAdd(&ctl->work, (int)c);  // the traversal's work units
      }
      __syncthreads();
      for (unsigned i = threadIdx.x; i < c; i += blockDim.x) {
        const uint2 x = AB[cur * kSeedCap + i];
        out[flush_at + i] = make_uint4(x.x, x.y, P[cur * kSeedCap + i], 0u);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    tests32 += __shfl_down_sync(0xffffffffu, tests32, o);
    lo32 += __shfl_down_sync(0xffffffffu, lo32, o);
  }
  if (lane == 0) {
    if (tests32) atomicAdd(&ctl->tests, (unsigned long long)tests32);
    if (lo32) atomicAdd(&ctl->leaf_overlaps, (unsigned long long)lo32);
  }
}

__global__ void trav_init_kernel(TravCtl* c, unsigned n_init, unsigned pair_base, int reset_totals, int stuck) {
  if (threadIdx.x != 0) return;
  if (reset_totals) {
    c->tests = 0;
    c->leaf_overlaps = 0;
    c->n_cand = 0;
    c->error = c->order_error;
    c->n_seed = 0;
    c->n_contacts = 0;
    c->n_mid = 0;
  }
  c->init_head = 0;
  c->q_head = 0;
  c->q_tail = 0;
  c->work = (int)n_init + stuck;
  c->n_init = n_init;
  c->pair_base = pair_base;
}

int traverse_block_threads(int block_warps) { return 32 * block_warps; }
size_t traverse_smem_bytes(int block_warps, int stack_cap) {
  return (size_t)block_warps * (size_t)stack_cap * sizeof(uint2);
}
// The kernels' limit, one for every shape: the attribute is the function's, and a
// host thread that set a shape's own could lower it between another thread's
// setting and its launch.  Options allow no shape above it.
size_t traverse_smem_limit(size_t smem_optin) { return smem_optin / 12 * sizeof(uint2); }

template <int K, int C, int S>
static cudaError_t prepare_shape(size_t smem) {
  cudaError_t e = cudaFuncSetAttribute(traverse_kernel<K, C, S, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(traverse_kernel<K, C, S, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return e;
}
template <int K>
static cudaError_t prepare_k(size_t smem) {
  cudaError_t e = prepare_shape<K, 1, 1>(smem);
  if (e == cudaSuccess) e = prepare_shape<K, 1, 2>(smem);
  if (e == cudaSuccess) e = prepare_shape<K, 2, 1>(smem);
  if (e == cudaSuccess) e = prepare_shape<K, 2, 2>(smem);
  return e;
}

cudaError_t traverse_prepare(int K, size_t smem) {
  switch (K) {
    case 6: return prepare_k<6>(smem);
    case 8: return prepare_k<8>(smem);
    case 12: return prepare_k<12>(smem);
    case 14: return prepare_k<14>(smem);
    case 18: return prepare_k<18>(smem);
    case 20: return prepare_k<20>(smem);
    case 26: return prepare_k<26>(smem);
  }
  return cudaErrorInvalidValue;
}

template <int K, int C, int S>
static cudaError_t traverse_impl(kdop_scene* s, int64_t n_pairs, const TravBuffers& b, const TravParams& p,
                                 int plain) {
  cudaStream_t st = s->ctx->stream;
  int threads = traverse_block_threads(p.block_warps);
  size_t smem = traverse_smem_bytes(p.block_warps, p.stack_cap);
  const bool seeded = b.seeds && !plain && p.wave_pairs <= 0 && n_pairs > 0;
  const auto kernel = seeded ? traverse_kernel<K, C, S, true> : traverse_kernel<K, C, S, false>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)traverse_smem_limit(s->ctx->smem_optin));
  if (e != cudaSuccess) return e;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                           p.smem_carveout > 0 ? p.smem_carveout : -1);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  unsigned grid = (unsigned)(per_sm * s->ctx->sm_count);
  TravArgs a;
  a.nodes = s->nodes;
  a.root = s->root_dev;
  a.pairs = b.pairs;
  a.order = b.order;
  a.entries = b.entries;
  a.candA = b.cand;
  a.candB = b.cand + b.cand_cap;
  a.candP = b.cand + 2 * b.cand_cap;
  a.cand_cap = (unsigned)b.cand_cap;
  a.q_items = b.q_items;
  a.q_tags = b.q_tags;
  a.q_cap = (unsigned)b.q_cap;
  a.ctl = b.ctl;
  a.n_meshes = (unsigned)s->n_meshes;
  a.stack_cap = p.stack_cap;
  a.init_chunk = p.init_chunk;
  a.donate_min = p.donate_min;
  a.surface_filter = p.surface_filter;
  a.timeout_ns = p.timeout_ns;
  // Donations reach waiting warps only through polls.  A batched launch keeps
  // most warps busy with root pairs and polls every 16th step (config 3: 10.49
  // ms vs 10.65 ms every 4th step); a one-pair launch leaves most warps
  // waiting for donations and polls every 4th step (config 3, one launch per
  // pair: 88 ms vs 103 ms every 16th).
  a.poll_mask = plain ? 3u : 15u;
  a.stuck = p.stuck_work;
  if (seeded) {
    const int sms = s->ctx->sm_count;
    const int64_t group = seed_group(sms, n_pairs), groups = (n_pairs + group - 1) / group;
    const unsigned blocks2 = (unsigned)seed_blocks2(sms, n_pairs, s->pairs_tets);
    constexpr size_t seed_smem = kSeedCap * 24;
    e = cudaFuncSetAttribute(seed_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)seed_smem);
    if (e != cudaSuccess) return e;
    uint4* seeds2 = b.seeds + seed_entries1(sms, n_pairs);
    trav_init_kernel<<<1, 32, 0, st>>>(b.ctl, 0u, 0u, 1, p.stuck_work);
    seed_kernel<K><<<(unsigned)std::min<int64_t>(groups, 4 * sms), kSeedThreads, seed_smem, st>>>(
        a, (unsigned)n_pairs, (unsigned)group, nullptr, nullptr, b.seeds,
        blocks2 ? &b.ctl->n_seed : &b.ctl->n_init);
    if (blocks2)
      seed_kernel<K><<<blocks2, kSeedThreads, seed_smem, st>>>(a, 0u, 0u, b.seeds, &b.ctl->n_seed, seeds2,
                                                              &b.ctl->n_init);
    a.entries = blocks2 ? seeds2 : b.seeds;
    kernel<<<grid, threads, smem, st>>>(a);
    s->ctx->launches += blocks2 ? 4 : 3;
    return cudaGetLastError();
  }
  if (b.entries) {
    // seeded by a frontier: its tests and leaf pairs are in the totals already
    trav_init_kernel<<<1, 32, 0, st>>>(b.ctl, (unsigned)n_pairs, 0u, 0, p.stuck_work);
    kernel<<<grid, threads, smem, st>>>(a);
    s->ctx->launches += 2;
  } else if (!plain) {
    // waves of wave_pairs root pairs (largest first), or all at once
    int64_t wave = p.wave_pairs > 0 ? p.wave_pairs : n_pairs;
    if (wave < 1) wave = 1;
    for (int64_t off = 0; off < n_pairs || off == 0; off += wave) {
      int64_t n = std::min<int64_t>(wave, n_pairs - off);
      trav_init_kernel<<<1, 32, 0, st>>>(b.ctl, (unsigned)std::max<int64_t>(n, 0), (unsigned)off, off == 0,
                                         p.stuck_work);
      kernel<<<grid, threads, smem, st>>>(a);
      s->ctx->launches += 2;
      if (n_pairs == 0) break;
    }
  } else {
    for (int64_t i = 0; i < n_pairs; ++i) {
      trav_init_kernel<<<1, 32, 0, st>>>(b.ctl, 1u, (unsigned)i, i == 0 ? 1 : 0, p.stuck_work);
      kernel<<<grid, threads, smem, st>>>(a);
      s->ctx->launches += 2;
    }
    if (n_pairs == 0) {
      trav_init_kernel<<<1, 32, 0, st>>>(b.ctl, 0u, 0u, 1, 0);
      s->ctx->launches += 1;
    }
  }
  return cudaGetLastError();
}

template <int K>
static cudaError_t traverse_group(kdop_scene* s, int64_t n_pairs, const TravBuffers& b, const TravParams& p,
                                  int plain) {
  // load_group: 1 = one chunk pair per lane, one sub-batch per step;
  // 2 = two sub-batches per step; 4 = two chunk pairs per lane (half the
  // lanes per entry, twice the entries per sub-batch); 8 = two chunk pairs
  // per lane and two sub-batches per step (twice the registers, one block
  // per SM)
  switch (p.load_group) {
    case 1: return traverse_impl<K, 1, 1>(s, n_pairs, b, p, plain);
    case 4: return traverse_impl<K, 2, 1>(s, n_pairs, b, p, plain);
    case 8: return traverse_impl<K, 2, 2>(s, n_pairs, b, p, plain);
    default: return traverse_impl<K, 1, 2>(s, n_pairs, b, p, plain);
  }
}

static cudaError_t traverse_buffers(kdop_scene* s, int64_t n_pairs, const TravBuffers& b, const TravParams& p,
                                    int plain) {
  switch (s->K) {
    case 6: return traverse_group<6>(s, n_pairs, b, p, plain);
    case 8: return traverse_group<8>(s, n_pairs, b, p, plain);
    case 12: return traverse_group<12>(s, n_pairs, b, p, plain);
    case 14: return traverse_group<14>(s, n_pairs, b, p, plain);
    case 18: return traverse_group<18>(s, n_pairs, b, p, plain);
    case 20: return traverse_group<20>(s, n_pairs, b, p, plain);
    case 26: return traverse_group<26>(s, n_pairs, b, p, plain);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_traverse(kdop_scene* s, int64_t n_pairs, const uint2* pairs, const TravParams& p, int plain) {
  TravBuffers b;
  b.pairs = pairs;
  b.order = s->pair_order;
  b.seeds = s->seeds;
  b.cand = s->cand;
  b.cand_cap = s->cand_cap;
  b.q_items = s->q_items;
  b.q_tags = s->q_tags;
  b.q_cap = s->queue_cap;
  b.ctl = s->ctl;
  return traverse_buffers(s, n_pairs, b, p, plain);
}

// ---- frontier-seeded and sharded traversal ----------------------------------
// The node-pair tree is expanded breadth first, one launch per level, until
// enough pairs are pending; every test and leaf pair of that expansion is the
// reference's own (the same rule, in breadth-first order).  The pending pairs
// are sorted (a deterministic list on every rank) and dealt round-robin to the
// shards; each shard's persistent traversal starts from its share.
namespace {

template <int K>
__device__ void frontier_emit(const TravArgs& a, uint32_t wa, uint32_t wb, uint32_t pid) {
  unsigned at = atomicAdd(&a.ctl->n_cand, 1u);
  if (at < a.cand_cap) {
    a.candA[at] = leaf_tet<K>(a.nodes, wa);
    a.candB[at] = leaf_tet<K>(a.nodes, wb);
    a.candP[at] = pid;
  }
}

__device__ void frontier_push(uint4* out, unsigned* count, unsigned cap, uint32_t wa, uint32_t wb, uint32_t pid,
                              unsigned* error) {
  unsigned at = atomicAdd(count, 1u);
  if (at < cap)
    out[at] = make_uint4(wa, wb, pid, 0u);
  else
    atomicOr(error, DEV_ERR_QUEUE_FULL);
}

// root test of each mesh pair (kdop_tandem_traversal.h:164, then :42)
template <int K>
__global__ void frontier_root_kernel(TravArgs a, unsigned n_pairs, uint4* out, unsigned* count, unsigned cap) {
  // count: level 0's count (the frontier state's first word)
  unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n_pairs) return;
  uint2 mp = a.pairs[p];
  if (mp.x >= a.n_meshes || mp.y >= a.n_meshes) {
    atomicOr(&a.ctl->error, DEV_ERR_BAD_INDEX);
    return;
  }
  uint32_t ra = a.root[mp.x], rb = a.root[mp.y];
  if (ra == NO_NODE || rb == NO_NODE) return;
  uint32_t wa, wb;
  bool ov = node_overlap<K>(a.nodes, ra, rb, wa, wb);
  atomicAdd(&a.ctl->tests, ov ? 2ull : 1ull);
  if (!ov) return;
  if (wa & wb & LEAF_BIT) {
    atomicAdd(&a.ctl->leaf_overlaps, 1ull);
    if (!a.surface_filter || (wa & wb & SURF_BIT)) frontier_emit<K>(a, wa, wb, p);
  } else {
    frontier_push(out, count, cap, wa, wb, p, &a.ctl->error);
  }
}

// Frontier state: level counts fs[0 .. kMaxLevels], then the frozen flag,
// the final level and the final count.
constexpr int kMaxLevels = 20;
constexpr int FS_FROZEN = kMaxLevels + 1, FS_LEVEL = kMaxLevels + 2, FS_COUNT = kMaxLevels + 3, FS_WORDS = 32;

// one level: every pending pair's child pairs.  The level stops the expansion
// (freezes) when its input is empty, large enough, or could overflow the
// next buffer; all later levels then do nothing.  Every thread reads the
// same counts, so they all take the same decision.
template <int K>
__global__ void frontier_level_kernel(TravArgs a, int level, const uint4* __restrict__ in, uint4* out, unsigned* fs,
                                      unsigned cap, unsigned fmin) {
  if (fs[FS_FROZEN]) return;
  const unsigned n_in = min(fs[level], cap);
  if (n_in == 0 || n_in >= fmin || 4ull * n_in > cap) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      fs[FS_FROZEN] = 1u;
      fs[FS_LEVEL] = (unsigned)level;
      fs[FS_COUNT] = n_in;
    }
    return;
  }
  unsigned* count = fs + level + 1;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n_in; i += gridDim.x * blockDim.x) {
  uint4 e = in[i];
  uint32_t A[2], B[2];
  int na = 2, nb = 2;
  if (e.x & LEAF_BIT) {
    A[0] = e.x & NODE_MASK;
    na = 1;
  } else {
    A[0] = e.x;
    A[1] = e.x + 1;
  }
  if (e.y & LEAF_BIT) {
    B[0] = e.y & NODE_MASK;
    nb = 1;
  } else {
    B[0] = e.y;
    B[1] = e.y + 1;
  }
  unsigned long long lo = 0;
  for (int x = 0; x < na; ++x)
    for (int y = 0; y < nb; ++y) {
      uint32_t wa, wb;
      if (!node_overlap<K>(a.nodes, A[x], B[y], wa, wb)) continue;
      if (wa & wb & LEAF_BIT) {
        ++lo;
        if (!a.surface_filter || (wa & wb & SURF_BIT)) frontier_emit<K>(a, wa, wb, e.z);
      } else {
        frontier_push(out, count, cap, wa, wb, e.z, &a.ctl->error);
      }
    }
  atomicAdd(&a.ctl->tests, (unsigned long long)(na * nb));
  if (lo) atomicAdd(&a.ctl->leaf_overlaps, lo);
  }
}

__global__ void frontier_final_kernel(unsigned* fs, unsigned cap) {
  if (threadIdx.x == 0 && !fs[FS_FROZEN]) {
    fs[FS_FROZEN] = 1u;
    fs[FS_LEVEL] = kMaxLevels;
    fs[FS_COUNT] = min(fs[kMaxLevels], cap);
  }
}

// Frontier order: by (A, B) words, then, stably, by pair.
struct EntryGen {
  const uint4* f;
  __device__ uint64_t key(int64_t i) const { return ((uint64_t)f[i].x << 32) | f[i].y; }
  __device__ uint32_t val(int64_t i) const { return (uint32_t)i; }
};
struct EntryPairGen {
  const uint4* f;
  const uint32_t* order;
  int64_t n;
  __device__ uint64_t key(int64_t i) const { return f[bounded(order[i], n)].z; }
  __device__ uint32_t val(int64_t i) const { return order[i]; }
};

// this shard's entries: sorted positions rank, rank + n_ranks, ...
__global__ void deal_kernel(const uint4* __restrict__ f, const uint32_t* __restrict__ order, unsigned n, int rank,
                            int n_ranks, uint4* mine) {
  unsigned j = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned src = (unsigned)rank + j * (unsigned)n_ranks;
  if (src < n) mine[j] = f[bounded(order[src], n)];
}

__global__ void clear_totals_kernel(TravCtl* c) {
  if (threadIdx.x == 0) {
    c->tests = 0;
    c->leaf_overlaps = 0;
    c->n_cand = 0;
  }
}

template <int K>
TravArgs frontier_args(kdop_scene* s, const uint2* pairs, const TravParams& p) {
  TravArgs a;
  std::memset(&a, 0, sizeof(a));
  a.nodes = s->nodes;
  a.root = s->root_dev;
  a.pairs = pairs;
  a.candA = s->cand;
  a.candB = s->cand + s->cand_cap;
  a.candP = s->cand + 2 * s->cand_cap;
  a.cand_cap = (unsigned)s->cand_cap;
  a.ctl = s->ctl;
  a.n_meshes = (unsigned)s->n_meshes;
  a.surface_filter = p.surface_filter;
  return a;
}

// Work buffer of a sharded traversal: frontier state, two frontiers, the
// sort (keys, values, scratch), this shard's entries; 256-byte regions.
struct ShardWork {
  size_t fs, f0, f1, k, kt, v, vt, sc, mine, total;
  explicit ShardWork(int64_t cap) {
    size_t at = 0;
    auto take = [&](size_t b) {
      size_t o = at;
      at += (b + 255) & ~(size_t)255;
      return o;
    };
    fs = take(FS_WORDS * 4);
    f0 = take((size_t)cap * 16);
    f1 = take((size_t)cap * 16);
    k = take((size_t)cap * 8);
    kt = take((size_t)cap * 8);
    v = take((size_t)cap * 4);
    vt = take((size_t)cap * 4);
    sc = take(radix_scratch_words(cap) * 4);
    mine = take((size_t)cap * 16);
    total = at;
  }
};

template <int K>
cudaError_t shard_impl(kdop_scene* s, int64_t n_pairs, const uint2* pairs, const TravParams& p, int rank,
                       int n_ranks, int64_t frontier_min, char* w, int64_t cap, int64_t* n_entries) {
  cudaStream_t st = s->ctx->stream;
  ShardWork L(cap);
  unsigned* fs = reinterpret_cast<unsigned*>(w + L.fs);
  uint4* F[2] = {reinterpret_cast<uint4*>(w + L.f0), reinterpret_cast<uint4*>(w + L.f1)};
  SortBuffers b{reinterpret_cast<uint64_t*>(w + L.k), reinterpret_cast<uint64_t*>(w + L.kt),
                reinterpret_cast<uint32_t*>(w + L.v), reinterpret_cast<uint32_t*>(w + L.vt)};
  uint4* mine = reinterpret_cast<uint4*>(w + L.mine);
  TravArgs a = frontier_args<K>(s, pairs, p);
  cudaError_t e;
  trav_init_kernel<<<1, 32, 0, st>>>(s->ctl, 0u, 0u, 1, 0);  // totals and queue state to zero
  if ((e = cudaMemsetAsync(fs, 0, FS_WORDS * 4, st)) != cudaSuccess) return e;
  if (n_pairs > 0)
    frontier_root_kernel<K><<<(unsigned)((n_pairs + 255) / 256), 256, 0, st>>>(a, (unsigned)n_pairs, F[0], fs,
                                                                                (unsigned)cap);
  const unsigned g = (unsigned)std::min<int64_t>((cap / 4 + 255) / 256, 4 * (int64_t)s->ctx->sm_count);
  for (int level = 0; level < kMaxLevels; ++level)
    frontier_level_kernel<K><<<g, 256, 0, st>>>(a, level, F[level & 1], F[(level + 1) & 1], fs, (unsigned)cap,
                                               (unsigned)frontier_min);
  frontier_final_kernel<<<1, 32, 0, st>>>(fs, (unsigned)cap);
  s->ctx->launches += 3 + kMaxLevels;
  unsigned hfs[FS_WORDS];
  if ((e = cudaMemcpyAsync(hfs, fs, sizeof(hfs), cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
  const unsigned n = hfs[FS_COUNT];
  const uint4* fin = F[hfs[FS_LEVEL] & 1];
  // deterministic order: by (A, B), then by pair
  if (n > 0) {
    const unsigned gn = (n + 255) / 256;
    const WaitLimit lim(&s->ctl->error, p.timeout_ns);
    if ((e = radix_sort(s->ctx, EntryGen{fin}, n, 64, b, w + L.sc, lim)) != cudaSuccess) return e;
    if ((e = radix_sort(s->ctx, EntryPairGen{fin, b.vals, n}, n, bits_of((uint64_t)std::max<int64_t>(n_pairs, 1) - 1), b,
                        w + L.sc, lim)) != cudaSuccess)
      return e;
    deal_kernel<<<gn, 256, 0, st>>>(fin, b.vals, n, rank, n_ranks, mine);
    s->ctx->launches += 1;
  }
  // the expansion's tests and leaf pairs belong to shard 0
  if (rank != 0) {
    clear_totals_kernel<<<1, 32, 0, st>>>(s->ctl);
    s->ctx->launches++;
  }
  const int64_t m = n > (unsigned)rank ? ((int64_t)n - rank + n_ranks - 1) / n_ranks : 0;
  *n_entries = m;
  TravBuffers t;
  t.pairs = pairs;
  t.order = nullptr;
  t.entries = mine;
  t.cand = s->cand;
  t.cand_cap = s->cand_cap;
  t.q_items = s->q_items;
  t.q_tags = s->q_tags;
  t.q_cap = s->queue_cap;
  t.ctl = s->ctl;
  return traverse_group<K>(s, m, t, p, 0);
}

}  // namespace

cudaError_t launch_traverse_shard(kdop_scene* s, int64_t n_pairs, const uint2* pairs, const TravParams& p, int rank,
                                  int n_ranks, int64_t frontier_min, void** work, size_t* work_bytes,
                                  int64_t* n_entries) {
  const int64_t cap = std::max<int64_t>(8 * std::max<int64_t>(frontier_min, 1), n_pairs) + 1024;
  const size_t need = ShardWork(cap).total;
  if (*work_bytes < need) {
    if (*work) cudaFree(*work);
    *work = nullptr;
    *work_bytes = 0;
    cudaError_t e = cudaMalloc(work, need);
    if (e != cudaSuccess) return e;
    *work_bytes = need;
  }
  char* w = static_cast<char*>(*work);
  switch (s->K) {
    case 6: return shard_impl<6>(s, n_pairs, pairs, p, rank, n_ranks, frontier_min, w, cap, n_entries);
    case 8: return shard_impl<8>(s, n_pairs, pairs, p, rank, n_ranks, frontier_min, w, cap, n_entries);
    case 12: return shard_impl<12>(s, n_pairs, pairs, p, rank, n_ranks, frontier_min, w, cap, n_entries);
    case 14: return shard_impl<14>(s, n_pairs, pairs, p, rank, n_ranks, frontier_min, w, cap, n_entries);
    case 18: return shard_impl<18>(s, n_pairs, pairs, p, rank, n_ranks, frontier_min, w, cap, n_entries);
    case 20: return shard_impl<20>(s, n_pairs, pairs, p, rank, n_ranks, frontier_min, w, cap, n_entries);
    case 26: return shard_impl<26>(s, n_pairs, pairs, p, rank, n_ranks, frontier_min, w, cap, n_entries);
  }
  return cudaErrorInvalidValue;
}

}  // namespace kdop

// ---- traversal that allocates no device memory -------------------------------
// Its scratch -- the traversal's control block and work queue -- lives in this
// file-scope device array instead of the scene's allocated buffers.  Every GPU
// that loads the library holds the array until the process exits.
namespace kdop {
namespace {

constexpr int64_t kStaticQueueEntries = 65536;
constexpr size_t kStaticCtlBytes = 1024;
constexpr size_t kStaticTagBytes = (size_t)kStaticQueueEntries * sizeof(uint32_t);
constexpr size_t kStaticScratchBytes = kStaticCtlBytes + kStaticTagBytes + (size_t)kStaticQueueEntries * sizeof(uint4);
static_assert(sizeof(TravCtl) <= kStaticCtlBytes, "control block does not fit");

__device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

// Device address of g_static_scratch per device, found once per device with
// that device current.  In host code the array's name only stands in for the
// symbol; it is not a device address.
constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
void* g_static_addr[kMaxDevices] = {nullptr};

cudaError_t static_scratch(int device, unsigned char** out) {
  if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (!g_static_addr[device]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
    if (e != cudaSuccess) return e;
    g_static_addr[device] = p;
  }
  *out = static_cast<unsigned char*>(g_static_addr[device]);
  return cudaSuccess;
}

__global__ void static_counters_kernel(const TravCtl* c, unsigned long long* out) {
  if (threadIdx.x != 0) return;
  out[0] = c->n_cand;
  out[1] = c->tests;
  out[2] = c->leaf_overlaps;
  out[3] = c->error;
}

}  // namespace
}  // namespace kdop

extern "C" int kdop_traverse_noalloc(kdop_scene* s, int64_t n_pairs, const uint32_t* pairs, uint32_t* candidates,
                                     int64_t cap, unsigned long long* counters, const kdop_traverse_opts* opts) {
  using namespace kdop;
  if (!s || n_pairs < 0 || (n_pairs > 0 && !pairs) || !candidates || cap <= 0 || !counters) return KDOP_ERR_INVALID;
  if (cap > (int64_t)0xFFFFFFF0ll || n_pairs >= (int64_t)0x7FFFFFFF) return KDOP_ERR_CAPACITY;
  TravParams p;
  int mode = 0;
  if (kdop_resolve_traverse_opts(s, opts, p, mode) != KDOP_OK) return KDOP_ERR_INVALID;
  if (cudaSetDevice(s->ctx->device) != cudaSuccess) return KDOP_ERR_CUDA;
  unsigned char* base = nullptr;
  if (static_scratch(s->ctx->device, &base) != cudaSuccess) {
    cudaGetLastError();
    return KDOP_ERR_CUDA;
  }
  TravBuffers b;
  b.pairs = reinterpret_cast<const uint2*>(pairs);
  b.order = nullptr;
  b.cand = candidates;
  b.cand_cap = cap;
  b.ctl = reinterpret_cast<TravCtl*>(base);
  b.q_tags = reinterpret_cast<uint32_t*>(base + kStaticCtlBytes);
  b.q_items = reinterpret_cast<uint4*>(base + kStaticCtlBytes + kStaticTagBytes);
  b.q_cap = kStaticQueueEntries;
  cudaStream_t st = s->ctx->stream;
  // the array keeps the previous call's contents: the control block and the
  // queue tags must start at zero
  if (cudaMemsetAsync(base, 0, kStaticCtlBytes + kStaticTagBytes, st) != cudaSuccess) {
    cudaGetLastError();
    return KDOP_ERR_CUDA;
  }
  cudaError_t e = traverse_buffers(s, n_pairs, b, p, mode == KDOP_TRAVERSE_PLAIN);
  if (e == cudaSuccess) {
    static_counters_kernel<<<1, 32, 0, st>>>(b.ctl, counters);
    s->ctx->launches += 1;
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return KDOP_ERR_CUDA;
  }
  return KDOP_OK;
}
