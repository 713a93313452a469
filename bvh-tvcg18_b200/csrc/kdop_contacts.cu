// kdop_contacts.cu -- tet-tet contact generation and its adjoint.
//
// Reference: contacts_tetrahedron_tetrahedron(A, B, cb, sA, sB,
// MOST_OPPOSING_SURFACES) (FOUNDATION/GEOMETRY/GEOMETRY/include/contacts/
// geometry_contacts_tetrahedron_tetrahedron.h:1313-1345), the default of
// kdop_select_contact_point_algorithm.h:30:
//   1. exact SAT overlap of the two tets (overlap/
//      geometry_overlap_tetrahedron_tetrahedron.h:51-290),
//   2. contact normal = unit normal of A's boundary face in the most opposing
//      pair of boundary faces (:465-533),
//   3. candidates = vertices of one tet inside the other and edge/face-plane
//      crossings inside the other tet (:544-620), depth = min - max of p.n over
//      all candidates, points projected on the mid plane, near-duplicates
//      (max-norm < 10 FLT_EPSILON) dropped, reported in order (:622-681).
//
// Three passes over the candidate tet pairs.  A contact needs an admissible
// pair of boundary faces (step 2) and overlapping tets (step 1), so the order
// of the two tests is free: the first pass looks for an admissible face pair,
// which of a deep overlap's candidates almost none has, and lists the pairs
// that go on; the second runs the 44 SAT axes on that list; the third runs step
// 2's argmin and step 3 for the pairs that overlap, in the reference's order
// (face pairs, then the 56 candidates in generation order), so the reported
// rows and every value equal the reference's FP32 results.  All passes evaluate
// the same functions on the same inputs, so their decisions agree.  Vertex
// positions are the world positions the last refit used (after a pose / deform
// refit, the array it computed).
//
// A thread takes a candidate, except that the second and third pass give a
// short list (kWarpCands, kWarpPairs) a warp per candidate: lanes over SAT
// axes, faces, face pairs and contact points, ballots keeping the order.  A
// thread's pass over 44 axes or 56 points is a chain of 15 and 28 us however
// few candidates there are; a warp's takes 6 and 9 us for a thousand, and about
// 2 ns more for each further one (30,000: 60 and 71 us, against 15 and 37).
// Measured before -> after: three passes of 512 uneven pairs (2.2 M candidates,
// 1.4 % with an admissible face pair) 520 -> 152 us, of 256 touching pairs (1.3 M
// candidates, half of them) 733 -> 515 us, of a touching pair of 384 tets 54 ->
// 23 us.
#include "kdop_device.cuh"

namespace kdop {

// geometry_tetrahedron.h:231-257: face opposite vertex v, outward for a
// positively oriented tet.
__constant__ int8_t c_face[4][3] = {{1, 2, 3}, {0, 3, 2}, {0, 1, 3}, {0, 2, 1}};
// edge table of geometry_contacts_tetrahedron_tetrahedron.h:584-591
__constant__ int8_t c_edge[6][2] = {{0, 1}, {0, 2}, {0, 3}, {1, 2}, {1, 3}, {2, 3}};
// The face and edge tables as compile-time values, and the 36 edge x edge
// axes of geometry_overlap_tetrahedron_tetrahedron.h:109-287 in order (A
// edge, B edge, A vertex left out, B vertex left out of SAT_line): in loops
// unrolled over faces, edges or SAT axes the indices fold to constants, so a
// tet's vertices and planes stay in registers instead of an indexed array in
// local memory (the passes over 2.2 M candidates, in their earlier order: 0.17
// -> 0.14 ms and 0.39 -> 0.32 ms).
__device__ __forceinline__ int face_vtx(int f, int k) {
  constexpr int8_t t[4][3] = {{1, 2, 3}, {0, 3, 2}, {0, 1, 3}, {0, 2, 1}};
  return t[f][k];
}
__device__ __forceinline__ int edge_vtx(int e, int k) {
  constexpr int8_t t[6][2] = {{0, 1}, {0, 2}, {0, 3}, {1, 2}, {1, 3}, {2, 3}};
  return t[e][k];
}
__device__ __forceinline__ int sat_entry(int e, int k) {
  constexpr int8_t t[36][4] = {
      {0, 0, 0, 0}, {0, 1, 0, 2}, {0, 2, 0, 3}, {0, 3, 0, 2}, {0, 4, 0, 3}, {0, 5, 0, 3},
      {1, 0, 0, 0}, {1, 1, 0, 0}, {1, 2, 0, 3}, {1, 3, 0, 2}, {1, 4, 0, 3}, {1, 5, 0, 3},
      {2, 0, 0, 0}, {2, 1, 0, 0}, {2, 2, 0, 0}, {2, 3, 0, 2}, {2, 4, 0, 3}, {2, 5, 0, 3},
      {3, 0, 2, 0}, {3, 1, 2, 0}, {3, 2, 2, 0}, {3, 3, 2, 2}, {3, 4, 2, 3}, {3, 5, 2, 3},
      {4, 0, 3, 0}, {4, 1, 3, 0}, {4, 2, 3, 0}, {4, 3, 3, 2}, {4, 4, 3, 3}, {4, 5, 3, 3},
      {5, 0, 3, 0}, {5, 1, 3, 0}, {5, 2, 3, 0}, {5, 3, 3, 2}, {5, 4, 3, 3}, {5, 5, 3, 3}};
  return t[e][k];
}

struct UPlane {
  f3 n, p;
};

// make_unscaled_plane (…_tetrahedron_tetrahedron.h:31-62)
__device__ __forceinline__ UPlane unscaled_plane(f3 p0, f3 p1, f3 p2) {
  f3 m0 = cross3(sub3(p1, p0), sub3(p2, p0));
  f3 m1 = cross3(sub3(p2, p1), sub3(p0, p1));
  f3 m2 = cross3(sub3(p0, p2), sub3(p1, p2));
  float l0 = dot3(m0, m0), l1 = dot3(m1, m1), l2 = dot3(m2, m2);
  UPlane pl{m0, p0};
  if (l0 >= l1 && l0 >= l2) pl = UPlane{m0, p0};
  if (l1 >= l0 && l1 >= l2) pl = UPlane{m1, p1};
  if (l2 >= l1 && l2 >= l0) pl = UPlane{m2, p2};
  return pl;
}
__device__ __forceinline__ float sdist(f3 q, const UPlane& pl) { return dot3(pl.n, sub3(q, pl.p)); }
__device__ __forceinline__ f3 intersect(f3 a, f3 b, const UPlane& pl) {
  float dA = fabsf(sdist(a, pl)), dB = fabsf(sdist(b, pl));
  float t = fdiv(dA, fadd(dA, dB));
  return add3(a, scl3(sub3(b, a), t));
}

// One of the 44 SAT tests; true = separating.
__device__ __forceinline__ bool sat_test(int t, const f3* A, const f3* B) {
  if (t < 8) {
    const f3* X = (t < 4) ? A : B;  // plane owner
    const f3* Y = (t < 4) ? B : A;  // tested points
    int f = t & 3;
    f3 p0 = X[face_vtx(f, 0)], p1 = X[face_vtx(f, 1)], p2 = X[face_vtx(f, 2)];
    // make_plane (geometry_plane.h:102-111) and get_signed_distance (:171-175)
    f3 nrm = unit3(cross3(sub3(p1, p0), sub3(p2, p0)));
    float w = dot3(p0, nrm);
    float d0 = fsub(dot3(nrm, Y[0]), w), d1 = fsub(dot3(nrm, Y[1]), w);
    float d2 = fsub(dot3(nrm, Y[2]), w), d3 = fsub(dot3(nrm, Y[3]), w);
    return d0 > 0.f && d1 > 0.f && d2 > 0.f && d3 > 0.f;
  }
  int e = t - 8;
  int ea = sat_entry(e, 0), eb = sat_entry(e, 1), xa = sat_entry(e, 2), xb = sat_entry(e, 3);
  f3 axis = cross3(sub3(A[edge_vtx(ea, 1)], A[edge_vtx(ea, 0)]), sub3(B[edge_vtx(eb, 1)], B[edge_vtx(eb, 0)]));
  // SAT_line (geometry_overlap_tetrahedron_tetrahedron.h:14-47) over the 3
  // vertices of each tet other than the one left out, in index order
  float s[3], u[3];
  int k = 0;
#pragma unroll
  for (int v = 0; v < 4; ++v)
    if (v != xa) s[k++] = dot3(axis, A[v]);
  k = 0;
#pragma unroll
  for (int v = 0; v < 4; ++v)
    if (v != xb) u[k++] = dot3(axis, B[v]);
  float lo_s = smin(smin(s[0], s[1]), s[2]), hi_s = smax(smax(s[0], s[1]), s[2]);
  float lo_u = smin(smin(u[0], u[1]), u[2]), hi_u = smax(smax(u[0], u[1]), u[2]);
  return (hi_s < lo_u) || (lo_s > hi_u);
}

struct ContactArgs {
  const uint32_t* candA;
  const uint32_t* candB;
  uint32_t* surv;  // candidates that overlap and have an admissible face pair (n_surv of them)
  uint32_t* mid;   // candidates with an admissible face pair (n_mid of them)
  unsigned cand_cap;
  const uint4* __restrict__ tets;
  const uint8_t* __restrict__ surf;
  VertexSource vs;
  kdop_contact* out;
  int4* rec;
  unsigned out_cap;
  TravCtl* ctl;
};

constexpr unsigned kWarpCands = 4096;   // second pass: up to this many candidates, a warp each
constexpr unsigned kWarpPairs = 6144;   // third pass: likewise

// A tet pair's values in shared memory, word `w` of a thread's (or a warp's)
// pair at base[w * stride]: an index that differs between lanes costs no bank
// conflict, where an indexed register array would live in local memory and
// fetch a line per lane.  Words: vertices (A 0-3, B 4-7), then the normals of
// the face planes (A 0-3, B 4-7); a plane's point is one of its vertices.
struct PairStore {
  float* base;
  int stride;
  __device__ __forceinline__ f3 get(int w) const {
    return mk3(base[w * stride], base[(w + 1) * stride], base[(w + 2) * stride]);
  }
  __device__ __forceinline__ void put(int w, f3 v) const {
    base[w * stride] = v.x;
    base[(w + 1) * stride] = v.y;
    base[(w + 2) * stride] = v.z;
  }
  __device__ __forceinline__ f3 vertex(int v) const { return get(3 * v); }       // v: tet * 4 + local vertex
  __device__ __forceinline__ f3 normal(int f) const { return get(24 + 3 * f); }  // f: tet * 4 + face
};
constexpr int kPairWords = 48;

// Vertex k of face f and of edge e, at run time.
__device__ __forceinline__ int face_at(int f, int k) {
  // {1, 2, 3}, {0, 3, 2}, {0, 1, 3}, {0, 2, 1}: two bits each, six per face
  return (int)((0x634B39u >> (6 * f + 2 * k)) & 3u);
}
__device__ __forceinline__ int edge_at(int e, int k) {
  // {0, 1}, {0, 2}, {0, 3}, {1, 2}, {1, 3}, {2, 3}: two bits each, four per edge
  return (int)((0xED9C84u >> (4 * e + 2 * k)) & 3u);
}

// make_unscaled_plane of face f (tet * 4 + face) from the stored vertices.
__device__ __forceinline__ UPlane stored_face_plane(const PairStore& s, int f) {
  const int t = f & 4;
  return unscaled_plane(s.vertex(t + face_at(f & 3, 0)), s.vertex(t + face_at(f & 3, 1)),
                        s.vertex(t + face_at(f & 3, 2)));
}

// Tets ta and tb of a candidate, posed.
__device__ __forceinline__ void candidate_tets(const ContactArgs& a, uint32_t ta, uint32_t tb, f3* A, f3* B) {
  const uint4 qa = __ldg(a.tets + ta), qb = __ldg(a.tets + tb);
  A[0] = world_vertex(a.vs, qa.x);
  A[1] = world_vertex(a.vs, qa.y);
  A[2] = world_vertex(a.vs, qa.z);
  A[3] = world_vertex(a.vs, qa.w);
  B[0] = world_vertex(a.vs, qb.x);
  B[1] = world_vertex(a.vs, qb.y);
  B[2] = world_vertex(a.vs, qb.z);
  B[3] = world_vertex(a.vs, qb.w);
}
// The same into a warp's store: a lane per vertex.
__device__ __forceinline__ void warp_tets(const ContactArgs& a, uint32_t ta, uint32_t tb, const PairStore& s,
                                          int lane) {
  if (lane < 8) {
    const uint32_t* q = reinterpret_cast<const uint32_t*>(a.tets + (lane < 4 ? ta : tb));
    s.put(3 * lane, world_vertex(a.vs, __ldg(q + (lane & 3))));
  }
  __syncwarp();
}

// Face pair admissible as the most opposing pair (…_tetrahedron_
// tetrahedron.h:465-533) besides being boundary faces: opposing unit normals
// (test, nA), and each tet's opposite vertex not behind the other's face
// plane.
__device__ __forceinline__ bool planes_oppose(const UPlane& pa, const UPlane& pb, f3 oppA, f3 oppB, float& test,
                                              f3& nA) {
  const float tA = dot3(pa.n, sub3(oppB, pa.p));
  const float tB = dot3(pb.n, sub3(oppA, pb.p));
  if ((tA < 0.f) || (tB < 0.f)) return false;
  nA = unit3(pa.n);
  test = dot3(nA, unit3(pb.n));
  return test < 0.f;
}

// Appends the warp's kept candidates to a list (one atomic per warp).
__device__ __forceinline__ void warp_append(bool keep, unsigned ci, unsigned* counter, uint32_t* list, unsigned cap,
                                            int lane) {
  const unsigned m = __ballot_sync(0xffffffffu, keep);
  if (m) {
    unsigned at = 0;
    if (lane == 0) at = atomicAdd(counter, (unsigned)__popc(m));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
    if (keep && at < cap) list[at] = ci;
  }
}

// Pass 1: thread per candidate, the search for an admissible face pair over the
// boundary faces (one or two of a tet, mostly).  A pair without one gets its
// empty record here; the others are listed.
__global__ void __launch_bounds__(256) contacts_filter_kernel(ContactArgs a) {
  __shared__ float store[24 * 256];
  const PairStore s{store + threadIdx.x, 256};
  const int lane = threadIdx.x & 31;
  const unsigned n_cand = min(*(volatile unsigned*)&a.ctl->n_cand, a.cand_cap);
  const unsigned stride = gridDim.x * blockDim.x;
  // counters of the later passes (n_mid, this pass's own, is zeroed by the
  // traversal and by pass 3)
  if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl->n_surv = a.ctl->n_contacts = 0u;
  for (unsigned base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n_cand; base += stride) {
    const unsigned ci = base + lane;
    bool keep = false;
    if (ci < n_cand) {
      const uint32_t ta = a.candA[ci], tb = a.candB[ci];
      const uint32_t sa = a.surf[ta] & 15u, sb = a.surf[tb] & 15u;
      if (sa && sb) {
        f3 A[4], B[4];
        candidate_tets(a, ta, tb, A, B);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          s.put(3 * v, A[v]);
          s.put(12 + 3 * v, B[v]);
        }
        for (uint32_t ma = sa; ma && !keep; ma &= ma - 1u) {
          const int fa = __ffs(ma) - 1;
          const UPlane pa = stored_face_plane(s, fa);
          const f3 oppA = s.vertex(fa);
          for (uint32_t mb = sb; mb && !keep; mb &= mb - 1u) {
            const int fb = __ffs(mb) - 1;
            float test;
            f3 nA;
            keep = planes_oppose(pa, stored_face_plane(s, 4 + fb), oppA, s.vertex(4 + fb), test, nA);
          }
        }
      }
      if (!keep) a.rec[ci] = make_int4(-1, -1, 0, 0);
    }
    warp_append(keep, ci, &a.ctl->n_mid, a.mid, a.cand_cap, lane);
  }
}

// SAT axis t (0..43) at run time, from the stored vertices; true = separating.
__device__ __forceinline__ bool stored_sat_test(int t, const PairStore& s) {
  if (t < 8) {
    const int Y = (t < 4) ? 4 : 0;  // plane owner: A for t < 4
    const int X = 4 - Y, f = t & 3;
    const f3 p0 = s.vertex(X + face_at(f, 0)), p1 = s.vertex(X + face_at(f, 1)), p2 = s.vertex(X + face_at(f, 2));
    const f3 nrm = unit3(cross3(sub3(p1, p0), sub3(p2, p0)));
    const float w = dot3(p0, nrm);
    bool out = true;
#pragma unroll
    for (int v = 0; v < 4; ++v) out = out && fsub(dot3(nrm, s.vertex(Y + v)), w) > 0.f;
    return out;
  }
  const int e = t - 8, ea = e / 6, eb = e % 6;
  // the vertices left out (the table of sat_entry)
  const int xa = ea < 3 ? 0 : ea == 3 ? 2 : 3;
  const int xb = eb == 0 ? 0 : eb == 1 ? (ea == 0 ? 2 : 0) : eb == 2 ? (ea < 2 ? 3 : 0) : eb == 3 ? 2 : 3;
  const f3 axis = cross3(sub3(s.vertex(edge_at(ea, 1)), s.vertex(edge_at(ea, 0))),
                         sub3(s.vertex(4 + edge_at(eb, 1)), s.vertex(4 + edge_at(eb, 0))));
  float p[3], u[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    p[k] = dot3(axis, s.vertex(k + (k >= xa ? 1 : 0)));
    u[k] = dot3(axis, s.vertex(4 + k + (k >= xb ? 1 : 0)));
  }
  const float lo_s = smin(smin(p[0], p[1]), p[2]), hi_s = smax(smax(p[0], p[1]), p[2]);
  const float lo_u = smin(smin(u[0], u[1]), u[2]), hi_u = smax(smax(u[0], u[1]), u[2]);
  return (hi_s < lo_u) || (lo_s > hi_u);
}

// Pass 2: the SAT axes of the listed candidates, the 8 face axes, then the 36
// edge axes.  A separated pair gets its empty record here; the others are
// listed for pass 3.
__global__ void __launch_bounds__(256) contacts_edge_kernel(ContactArgs a) {
  __shared__ float store[8][24];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const unsigned n_mid = min(*(volatile unsigned*)&a.ctl->n_mid, a.cand_cap);
  if (n_mid <= kWarpCands) {
    const PairStore s{store[wib], 1};
    for (unsigned k = blockIdx.x * 8u + wib; k < n_mid; k += gridDim.x * 8u) {
      const unsigned ci = a.mid[k];
      warp_tets(a, a.candA[ci], a.candB[ci], s, lane);
      bool sep = stored_sat_test(lane, s);
      if (lane < 12) sep = sep || stored_sat_test(lane + 32, s);
      sep = __any_sync(0xffffffffu, sep);
      if (lane == 0) {
        if (sep)
          a.rec[ci] = make_int4(-1, -1, 0, 0);
        else
          a.surv[atomicAdd(&a.ctl->n_surv, 1u)] = ci;
      }
      __syncwarp();
    }
    return;
  }
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n_mid; base += stride) {
    const unsigned k = base + lane;
    bool keep = false;
    unsigned ci = 0;
    if (k < n_mid) {
      ci = a.mid[k];
      f3 A[4], B[4];
      candidate_tets(a, a.candA[ci], a.candB[ci], A, B);
      bool sep = false;
#pragma unroll
      for (int t = 0; t < 44; ++t)
        if (!sep) sep = sat_test(t, A, B);
      keep = !sep;
      if (!keep) a.rec[ci] = make_int4(-1, -1, 0, 0);
    }
    warp_append(keep, ci, &a.ctl->n_surv, a.surv, a.cand_cap, lane);
  }
}

// The face planes of a pair whose vertices and plane normals are stored; the
// points are vertices: corner codes, two bits per face (face_at's index).
struct Planes {
  PairStore s;
  uint32_t corners;
  __device__ __forceinline__ UPlane operator[](int f) const {
    const int k = (int)((corners >> (2 * f)) & 3u);
    return UPlane{s.normal(f), s.vertex((f & 4) + face_at(f & 3, k))};
  }
};
// Corner whose cross product make_unscaled_plane takes.
__device__ __forceinline__ UPlane corner_plane(f3 p0, f3 p1, f3 p2, uint32_t& corner) {
  f3 m0 = cross3(sub3(p1, p0), sub3(p2, p0));
  f3 m1 = cross3(sub3(p2, p1), sub3(p0, p1));
  f3 m2 = cross3(sub3(p0, p2), sub3(p1, p2));
  float l0 = dot3(m0, m0), l1 = dot3(m1, m1), l2 = dot3(m2, m2);
  corner = 0u;
  UPlane pl{m0, p0};
  if (l1 >= l0 && l1 >= l2) {
    pl = UPlane{m1, p1};
    corner = 1u;
  }
  if (l2 >= l1 && l2 >= l0) {
    pl = UPlane{m2, p2};
    corner = 2u;
  }
  return pl;
}

__device__ __forceinline__ bool inside_planes(f3 q, const Planes& P, int t) {
  bool in = true;
#pragma unroll
  for (int f = 0; f < 4; ++f) in = in && !(sdist(q, P[t + f]) > 0.f);
  return in;
}
// Crossing point of contact candidate c >= 8 (edge (c - 8) / 8 of B, of A when
// c is odd, with face plane ((c - 8) / 2) % 4 of the other tet), known to
// cross; true when it lies inside that tet.
__device__ __forceinline__ bool crossing_point(int c, const PairStore& s, const Planes& P, f3& q) {
  const int e = (c - 8) >> 3, p = ((c - 8) >> 1) & 3;
  const int E = (c & 1) ? 0 : 4, T = 4 - E;
  q = intersect(s.vertex(E + edge_at(e, 0)), s.vertex(E + edge_at(e, 1)), P[T + p]);
  return inside_planes(q, P, T);
}

// Which side of each face plane of tet T (4: B, 0: A) the other tet's vertices
// lie on: bit 4 v + f of `ge` (distance >= 0), `le` (<= 0), `gt` (> 0).
struct Sides {
  uint32_t ge, le, gt;
};
__device__ __forceinline__ void add_side(Sides& d, int v, int f, float dist) {
  const int b = 4 * v + f;
  d.ge |= (dist >= 0.f ? 1u : 0u) << b;
  d.le |= (dist <= 0.f ? 1u : 0u) << b;
  d.gt |= (dist > 0.f ? 1u : 0u) << b;
}
__device__ __forceinline__ uint32_t spread4(uint32_t x) {  // bit k to bit 2 k
  return (x & 1u) | ((x & 2u) << 1) | ((x & 4u) << 2) | ((x & 8u) << 3);
}
// Contact candidates that are there, bit c (0..55) in the reference's
// generation order: vertices inside the other tet, edges that cross a face
// plane (whose crossing may still lie outside).  b: B's vertices against A's
// planes, a: A's against B's.
__device__ __forceinline__ uint64_t candidate_bits(const Sides& b, const Sides& a) {
  uint64_t m = 0;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    if (((b.gt >> (4 * v)) & 15u) == 0u) m |= 1ull << (2 * v);
    if (((a.gt >> (4 * v)) & 15u) == 0u) m |= 2ull << (2 * v);
  }
#pragma unroll
  for (int e = 0; e < 6; ++e) {
    const int i = 4 * edge_vtx(e, 0), j = 4 * edge_vtx(e, 1);
    const uint32_t xb = ~((b.ge >> i) & (b.ge >> j)) & ~((b.le >> i) & (b.le >> j)) & 15u;
    const uint32_t xa = ~((a.ge >> i) & (a.ge >> j)) & ~((a.le >> i) & (a.le >> j)) & 15u;
    m |= (uint64_t)(spread4(xb) | (spread4(xa) << 1)) << (8 + 8 * e);
  }
  return m;
}

constexpr float kContactEps = 1.1920928955078125e-06f;  // 10 * FLT_EPSILON
__device__ __forceinline__ bool near_points(f3 p, f3 q) {
  return smax(smax(fabsf(fsub(p.x, q.x)), fabsf(fsub(p.y, q.y))), fabsf(fsub(p.z, q.z))) < kContactEps;
}
__device__ __forceinline__ void put_row(const ContactArgs& a, unsigned r, f3 p, f3 n, float depth, unsigned ci) {
  if (r >= a.out_cap) return;
  float4* o = reinterpret_cast<float4*>(a.out + r);
  o[0] = make_float4(p.x, p.y, p.z, n.x);
  o[1] = make_float4(n.y, n.z, depth, __uint_as_float(ci));
}
// Projection on the mid plane (mid: its point on n).
__device__ __forceinline__ f3 on_mid_plane(f3 q, f3 n, f3 mid) {
  const float k = dot3(n, sub3(q, mid));
  return sub3(q, mk3(fmul(k, n.x), fmul(k, n.y), fmul(k, n.z)));
}
__device__ __forceinline__ f3 mid_point(f3 n, float mn, float mx) {
  const float sum = fadd(mx, mn);
  return mk3(fmul(fmul(n.x, sum), 0.5f), fmul(fmul(n.y, sum), 0.5f), fmul(fmul(n.z, sum), 0.5f));
}

// Smallest (first: SIGN 1) or largest (SIGN -1) d over the lanes' values, two a
// lane (candidates lane and lane + 32), the first of equal ones; as a running
// minimum takes it: a first value that is NaN stays, later ones are passed
// over.  `there`: the candidates' mask.
template <int SIGN>
__device__ __forceinline__ void warp_extreme(float d0, float d1, uint64_t there, int lane, float& best, int& code) {
  best = 0.f;
  code = 64;
  auto take = [&](float d, int c) {
    const bool less = SIGN > 0 ? d < best : best < d;
    if (code == 64 || less || (d == best && c < code)) {
      best = d;
      code = c;
    }
  };
  if (((there >> lane) & 1ull) && d0 == d0) take(d0, lane);
  if (((there >> (lane + 32)) & 1ull) && d1 == d1) take(d1, lane + 32);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float d = __shfl_xor_sync(0xffffffffu, best, o);
    const int c = __shfl_xor_sync(0xffffffffu, code, o);
    if (c != 64) take(d, c);
  }
  const int first = __ffsll((long long)there) - 1;
  const float df = first < 32 ? __shfl_sync(0xffffffffu, d0, first) : __shfl_sync(0xffffffffu, d1, first - 32);
  if (!(df == df)) {
    best = df;
    code = first;
  }
}

// Pass 3, a warp per listed pair.  pts: room for 56 points.
__device__ __forceinline__ void warp_contacts(const ContactArgs& a, unsigned ci, const PairStore& s, float* pts,
                                              int lane) {
  const uint32_t ta = a.candA[ci], tb = a.candB[ci];
  warp_tets(a, ta, tb, s, lane);
  uint32_t corner = 0;
  if (lane < 8) {
    const int t = lane & 4, f = lane & 3;
    s.put(24 + 3 * lane, corner_plane(s.vertex(t + face_at(f, 0)), s.vertex(t + face_at(f, 1)),
                                      s.vertex(t + face_at(f, 2)), corner).n);
  }
  Planes P{s, 0u};
  P.corners = __reduce_or_sync(0xffffffffu, lane < 8 ? corner << (2 * lane) : 0u);
  __syncwarp();
  // face pair l = 4 fa + fb on lane l: the smallest test, the first of equal ones
  const uint32_t sa = a.surf[ta], sb = a.surf[tb];
  float test = 3.0e38f;
  f3 n = mk3(0.f, 0.f, 0.f);
  int l = 16;
  if (lane < 16 && ((sa >> (lane >> 2)) & 1u) && ((sb >> (lane & 3)) & 1u)) {
    float t;
    f3 nA;
    if (planes_oppose(P[lane >> 2], P[4 + (lane & 3)], s.vertex(lane >> 2), s.vertex(4 + (lane & 3)), t, nA)) {
      test = t;
      n = nA;
      l = lane;
    }
  }
  const f3 mine = n;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    const float t = __shfl_xor_sync(0xffffffffu, test, o);
    const int k = __shfl_xor_sync(0xffffffffu, l, o);
    if (k < 16 && (l == 16 || t < test || (t == test && k < l))) {
      test = t;
      l = k;
    }
  }
  l = __shfl_sync(0xffffffffu, l, 0);
  if (l == 16) {  // not with pass 1's list
    if (lane == 0) a.rec[ci] = make_int4(-1, -1, 0, 0);
    return;
  }
  n = mk3(__shfl_sync(0xffffffffu, mine.x, l), __shfl_sync(0xffffffffu, mine.y, l), __shfl_sync(0xffffffffu, mine.z, l));
  // sides: vertex lane / 4 against plane lane % 4, B's vertices on the lower
  // half of the warp, A's on the upper
  const int v = (lane >> 2) & 3, f = lane & 3, half = lane >> 4;
  const float dist = sdist(s.vertex((half ? 0 : 4) + v), P[(half ? 4 : 0) + f]);
  const unsigned ge = __ballot_sync(0xffffffffu, dist >= 0.f), le = __ballot_sync(0xffffffffu, dist <= 0.f);
  const unsigned gt = __ballot_sync(0xffffffffu, dist > 0.f);
  const uint64_t maybe = candidate_bits(Sides{ge & 0xFFFFu, le & 0xFFFFu, gt & 0xFFFFu}, Sides{ge >> 16, le >> 16, gt >> 16});
  f3 q0 = mk3(0.f, 0.f, 0.f), q1 = q0;
  bool in0 = (maybe >> lane) & 1ull, in1 = (maybe >> (lane + 32)) & 1ull;
  if (in0) {
    if (lane < 8)
      q0 = s.vertex(((lane & 1) ? 0 : 4) + (lane >> 1));
    else
      in0 = crossing_point(lane, s, P, q0);
  }
  if (in1) in1 = crossing_point(lane + 32, s, P, q1);
  const unsigned b0 = __ballot_sync(0xffffffffu, in0), b1 = __ballot_sync(0xffffffffu, in1);
  const uint64_t there = (uint64_t)b0 | ((uint64_t)b1 << 32);
  int4 record = make_int4(l >> 2, 0, 0, 0);
  if (there) {
    const float d0 = dot3(q0, n), d1 = dot3(q1, n);
    float mn, mx;
    int cmn, cmx;
    warp_extreme<1>(d0, d1, there, lane, mn, cmn);
    warp_extreme<-1>(d0, d1, there, lane, mx, cmx);
    const float depth = fsub(mn, mx);
    const f3 mid = mid_point(n, mn, mx);
    q0 = on_mid_plane(q0, n, mid);
    q1 = on_mid_plane(q1, n, mid);
    // points in order; a point near an earlier one is dropped
    const unsigned lt = (1u << lane) - 1u;
    const int i0 = __popc(b0 & lt), i1 = __popc(b0) + __popc(b1 & lt), nq = __popc(b0) + __popc(b1);
    if (in0) {
      pts[3 * i0] = q0.x;
      pts[3 * i0 + 1] = q0.y;
      pts[3 * i0 + 2] = q0.z;
    }
    if (in1) {
      pts[3 * i1] = q1.x;
      pts[3 * i1 + 1] = q1.y;
      pts[3 * i1 + 2] = q1.z;
    }
    __syncwarp();
    bool u0 = in0, u1 = in1;
    for (int j = 0; j < nq; ++j) {
      const f3 p = mk3(pts[3 * j], pts[3 * j + 1], pts[3 * j + 2]);
      if (j < i0 && near_points(p, q0)) u0 = false;
      if (j < i1 && near_points(p, q1)) u1 = false;
    }
    const unsigned k0 = __ballot_sync(0xffffffffu, u0), k1 = __ballot_sync(0xffffffffu, u1);
    const int nu = __popc(k0) + __popc(k1);
    unsigned row = 0;
    if (lane == 0) row = atomicAdd(&a.ctl->n_contacts, (unsigned)nu);
    row = __shfl_sync(0xffffffffu, row, 0);
    if (u0) put_row(a, row + __popc(k0 & lt), q0, n, depth, ci);
    if (u1) put_row(a, row + __popc(k0) + __popc(k1 & lt), q1, n, depth, ci);
    record.y = (cmn & 0xFF) | ((cmx & 0xFF) << 8);
    record.z = nu;
    record.w = (int)row;
  }
  if (lane == 0) a.rec[ci] = record;
  __syncwarp();
}

// Pass 3, thread per listed pair (or warp, above): the argmin over the face
// pairs by a strict < in loop order (first occurrence), the candidate points in
// generation order with running min / max of p.n (first occurrence), projection
// on the mid plane, and the duplicate test of each point against every earlier
// one.  The distances of the 8 vertices to the other tet's planes are taken
// once and say which vertices lie inside and which edges cross; a thread then
// goes from one of its crossings to the next instead of over all 48 (449 -> 296
// us for 640,000 pairs; six blocks per SM at 80 registers, with four at 127 338
// us, with eight 367).  Rows of a warp are placed with one atomic.
constexpr int CT_THREADS = 128;
__global__ void __launch_bounds__(CT_THREADS, 6) contacts_thread_kernel(ContactArgs a) {
  __shared__ float store[kPairWords * CT_THREADS];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const unsigned n_surv = min(*(volatile unsigned*)&a.ctl->n_surv, a.cand_cap);
  if (blockIdx.x == 0 && threadIdx.x == 0) a.ctl->n_mid = 0u;  // for the next call (pass 2 has read it)
  if (n_surv <= kWarpPairs) {
    float* mine = store + wib * (kPairWords + 3 * 56);
    for (unsigned k = blockIdx.x * (CT_THREADS / 32) + wib; k < n_surv; k += gridDim.x * (CT_THREADS / 32))
      warp_contacts(a, a.surv[k], PairStore{mine, 1}, mine + kPairWords, lane);
    return;
  }
  const PairStore s{store + threadIdx.x, CT_THREADS};
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n_surv; base += stride) {
    const unsigned k = base + lane;
    const bool act = k < n_surv;
    unsigned ci = 0;
    int4 record = make_int4(-1, -1, 0, 0);
    int nq = 0, nu = 0;
    float depth = 0.f;
    f3 n = mk3(0.f, 0.f, 0.f);
    float px[56], py[56], pz[56];
    uint64_t kept = 0;
    if (act) {
      ci = a.surv[k];
      const uint32_t ta = a.candA[ci], tb = a.candB[ci];
      const uint32_t sa = a.surf[ta] & 15u, sb = a.surf[tb] & 15u;
      Planes P{s, 0u};
      Sides dB{0u, 0u, 0u}, dA{0u, 0u, 0u};
      {
        f3 A[4], B[4];
        candidate_tets(a, ta, tb, A, B);
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          s.put(3 * v, A[v]);
          s.put(12 + 3 * v, B[v]);
        }
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          uint32_t ca, cb;
          const UPlane pa = corner_plane(A[face_vtx(f, 0)], A[face_vtx(f, 1)], A[face_vtx(f, 2)], ca);
          const UPlane pb = corner_plane(B[face_vtx(f, 0)], B[face_vtx(f, 1)], B[face_vtx(f, 2)], cb);
          s.put(24 + 3 * f, pa.n);
          s.put(36 + 3 * f, pb.n);
          P.corners |= (ca << (2 * f)) | (cb << (8 + 2 * f));
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            add_side(dB, v, f, sdist(B[v], pa));
            add_side(dA, v, f, sdist(A[v], pb));
          }
        }
      }
      float bv = 3.0e38f;
      int bl = -1;
      for (uint32_t ma = sa; ma; ma &= ma - 1u)
        for (uint32_t mb = sb; mb; mb &= mb - 1u) {
          const int fa = __ffs(ma) - 1, fb = __ffs(mb) - 1;
          float t;
          f3 nA;
          if (planes_oppose(P[fa], P[4 + fb], s.vertex(fa), s.vertex(4 + fb), t, nA) && t < bv) {
            bv = t;
            bl = 4 * fa + fb;
            n = nA;
          }
        }
      if (bl >= 0) {
        record.x = bl >> 2;
        record.y = 0;
        float mnv = 0.f, mxv = 0.f;
        int mnc = -1, mxc = -1;
        for (uint64_t m = candidate_bits(dB, dA); m; m &= m - 1ull) {
          const int c = __ffsll((long long)m) - 1;
          f3 q;
          if (c < 8)
            q = s.vertex(((c & 1) ? 0 : 4) + (c >> 1));
          else if (!crossing_point(c, s, P, q))
            continue;
          const float d = dot3(q, n);
          if (nq == 0 || d < mnv) { mnv = d; mnc = c; }
          if (nq == 0 || mxv < d) { mxv = d; mxc = c; }
          px[nq] = q.x;
          py[nq] = q.y;
          pz[nq] = q.z;
          ++nq;
        }
        if (nq > 0) {
          depth = fsub(mnv, mxv);
          const f3 mid = mid_point(n, mnv, mxv);
          for (int i = 0; i < nq; ++i) {
            const f3 q = on_mid_plane(mk3(px[i], py[i], pz[i]), n, mid);
            px[i] = q.x;
            py[i] = q.y;
            pz[i] = q.z;
            bool u = true;
            for (int j = 0; j < i && u; ++j) u = !near_points(mk3(px[j], py[j], pz[j]), q);
            if (u) {
              kept |= 1ull << i;
              ++nu;
            }
          }
          record.y = (mnc & 0xFF) | ((mxc & 0xFF) << 8);
          record.z = nu;
        }
      }
    }
    // rows of the warp: one atomic
    int incl = nu;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    unsigned wbase = 0;
    if (lane == 0 && total > 0) wbase = atomicAdd(&a.ctl->n_contacts, (unsigned)total);
    wbase = __shfl_sync(0xffffffffu, wbase, 0);
    if (act) {
      if (nu > 0) {
        unsigned r = wbase + (unsigned)(incl - nu);
        record.w = (int)r;
        for (int i = 0; i < nq; ++i)
          if ((kept >> i) & 1ull) put_row(a, r++, mk3(px[i], py[i], pz[i]), n, depth, ci);
      }
      a.rec[ci] = record;
    }
  }
}

// ---- adjoint -------------------------------------------------------------------
// Frozen-decision depth d = q_min . n - q_max . n with n = m / |m|, m the
// cross product of A's chosen face; q a vertex or an edge/plane crossing
// a + (b - a) t, t = |sA| / (|sA| + |sB|), s = m_p . (x - F0) for the face
// plane p of the other tet.  In exact arithmetic the three corner cross
// products of make_unscaled_plane coincide and every corner lies on the
// plane, so the first corner stands for the chosen one.  The inputs and the
// gradient are float; the chain rule runs in double, because near-parallel
// edge/plane crossings (dA + dB small) amplify rounding by orders of
// magnitude.
struct d3 {
  double x, y, z;
};
__device__ __forceinline__ d3 dmk(double x, double y, double z) { return d3{x, y, z}; }
__device__ __forceinline__ d3 dof(f3 v) { return d3{(double)v.x, (double)v.y, (double)v.z}; }
__device__ __forceinline__ d3 dsub(d3 a, d3 b) { return dmk(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ d3 dadd(d3 a, d3 b) { return dmk(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ d3 dscl(d3 a, double s) { return dmk(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ double ddot(d3 a, d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ d3 dcross(d3 l, d3 r) {
  return dmk(l.y * r.z - l.z * r.y, l.z * r.x - l.x * r.z, l.x * r.y - l.y * r.x);
}
__device__ __forceinline__ void dacc(d3* g, int i, d3 v) { g[i] = dadd(g[i], v); }

__device__ __forceinline__ d3 face_m(const d3* T, int f, d3& F0) {
  F0 = T[c_face[f][0]];
  return dcross(dsub(T[c_face[f][1]], F0), dsub(T[c_face[f][2]], F0));
}

// adjoint of m = (P1 - P0) x (P2 - P0) for face f of T into gT
__device__ void face_m_adj(const d3* T, int f, d3 gm, d3* gT) {
  int i0 = c_face[f][0], i1 = c_face[f][1], i2 = c_face[f][2];
  d3 u = dsub(T[i1], T[i0]), w = dsub(T[i2], T[i0]);
  d3 gu = dcross(w, gm), gw = dcross(gm, u);
  dacc(gT, i1, gu);
  dacc(gT, i2, gw);
  dacc(gT, i0, dscl(dadd(gu, gw), -1.0));
}

__device__ d3 cand_point(int c, const d3* A, const d3* B) {
  if (c < 8) return (c & 1) ? A[c >> 1] : B[c >> 1];
  int e = (c - 8) >> 3, p = ((c - 8) >> 1) & 3;
  const d3* E = (c & 1) ? A : B;
  const d3* T = (c & 1) ? B : A;
  d3 a = E[c_edge[e][0]], b = E[c_edge[e][1]], F0;
  d3 m = face_m(T, p, F0);
  double dA = fabs(ddot(m, dsub(a, F0))), dB = fabs(ddot(m, dsub(b, F0)));
  double t = dA / (dA + dB);
  return dadd(a, dscl(dsub(b, a), t));
}

__device__ void cand_adj(int c, const d3* A, const d3* B, d3 gq, d3* gA, d3* gB) {
  if (c < 8) {
    dacc((c & 1) ? gA : gB, c >> 1, gq);
    return;
  }
  int e = (c - 8) >> 3, p = ((c - 8) >> 1) & 3;
  const d3* E = (c & 1) ? A : B;
  const d3* T = (c & 1) ? B : A;
  d3* gE = (c & 1) ? gA : gB;
  d3* gT = (c & 1) ? gB : gA;
  int ia = c_edge[e][0], ib = c_edge[e][1];
  d3 a = E[ia], b = E[ib], F0;
  d3 m = face_m(T, p, F0);
  double sA = ddot(m, dsub(a, F0)), sB = ddot(m, dsub(b, F0));
  double sgA = sA < 0.0 ? -1.0 : 1.0, sgB = sB < 0.0 ? -1.0 : 1.0;
  double dA = fabs(sA), dB = fabs(sB), S = dA + dB;
  double t = dA / S;
  // q = a + (b - a) t
  dacc(gE, ia, dscl(gq, 1.0 - t));
  dacc(gE, ib, dscl(gq, t));
  double gt = ddot(gq, dsub(b, a));
  double gdA = gt * dB / (S * S), gdB = -gt * dA / (S * S);
  // dA = sgA m.(a - F0), dB = sgB m.(b - F0)
  dacc(gE, ia, dscl(m, sgA * gdA));
  dacc(gE, ib, dscl(m, sgB * gdB));
  dacc(gT, c_face[p][0], dscl(dadd(dscl(m, sgA * gdA), dscl(m, sgB * gdB)), -1.0));
  d3 gm = dadd(dscl(dsub(a, F0), sgA * gdA), dscl(dsub(b, F0), sgB * gdB));
  face_m_adj(T, p, gm, gT);
}

struct AdjointArgs {
  const uint32_t* candA;
  const uint32_t* candB;
  unsigned cand_cap;
  const uint4* __restrict__ tets;
  const int4* __restrict__ rec;
  const float* dd;
  const float* dn;
  unsigned out_cap;
  VertexSource vs;
  float* grad;
  TravCtl* ctl;
};

__global__ void __launch_bounds__(128) adjoint_kernel(AdjointArgs a) {
  unsigned n_cand = min(*(volatile unsigned*)&a.ctl->n_cand, a.cand_cap);
  for (unsigned ci = blockIdx.x * blockDim.x + threadIdx.x; ci < n_cand; ci += gridDim.x * blockDim.x) {
    int4 r = a.rec[ci];
    if (r.z <= 0 || r.x < 0) continue;
    double gd = 0.0;
    d3 gn = dmk(0.0, 0.0, 0.0);
    for (int k = 0; k < r.z; ++k) {
      unsigned row = (unsigned)r.w + (unsigned)k;
      if (row >= a.out_cap) break;
      gd += (double)a.dd[row];
      if (a.dn) gn = dadd(gn, dmk(a.dn[3 * row], a.dn[3 * row + 1], a.dn[3 * row + 2]));
    }
    uint4 qa = __ldg(a.tets + a.candA[ci]), qb = __ldg(a.tets + a.candB[ci]);
    uint32_t va[4] = {qa.x, qa.y, qa.z, qa.w}, vb[4] = {qb.x, qb.y, qb.z, qb.w};
    d3 A[4], B[4], gA[4], gB[4];
    for (int v = 0; v < 4; ++v) {
      A[v] = dof(world_vertex(a.vs, va[v]));
      B[v] = dof(world_vertex(a.vs, vb[v]));
      gA[v] = gB[v] = dmk(0.0, 0.0, 0.0);
    }
    int imin = r.y & 0xFF, imax = (r.y >> 8) & 0xFF;
    d3 F0;
    d3 m = face_m(A, r.x, F0);
    double len = sqrt(ddot(m, m));
    d3 n = dscl(m, 1.0 / len);
    d3 qmin = cand_point(imin, A, B), qmax = cand_point(imax, A, B);
    // depth = qmin . n - qmax . n
    cand_adj(imin, A, B, dscl(n, gd), gA, gB);
    cand_adj(imax, A, B, dscl(n, -gd), gA, gB);
    d3 gnt = dadd(gn, dscl(dsub(qmin, qmax), gd));
    d3 gm = dscl(dsub(gnt, dscl(n, ddot(n, gnt))), 1.0 / len);
    face_m_adj(A, r.x, gm, gA);
    for (int v = 0; v < 4; ++v) {
      atomicAdd(a.grad + 3 * (size_t)va[v], (float)gA[v].x);
      atomicAdd(a.grad + 3 * (size_t)va[v] + 1, (float)gA[v].y);
      atomicAdd(a.grad + 3 * (size_t)va[v] + 2, (float)gA[v].z);
      atomicAdd(a.grad + 3 * (size_t)vb[v], (float)gB[v].x);
      atomicAdd(a.grad + 3 * (size_t)vb[v] + 1, (float)gB[v].y);
      atomicAdd(a.grad + 3 * (size_t)vb[v] + 2, (float)gB[v].z);
    }
  }
}

static VertexSource vsrc(kdop_scene* s) {
  VertexSource vs;
  vs.rest = s->rest;
  vs.world = s->world;
  vs.quat = s->quat;
  vs.pos = s->pos;
  vs.deform.amp = s->amp;
  vs.deform.w = s->w;
  vs.deform.phase = s->phase_dev;
  vs.mode = s->refit_mode < 0 ? 0 : s->refit_mode;
  if (vs.mode != KDOP_REFIT_VERTICES) {
    // the world positions the last pose / deform refit computed (and traversed)
    vs.mode = KDOP_REFIT_VERTICES;
    vs.world = s->posed;
  }
  return vs;
}

cudaError_t launch_contacts(kdop_scene* s) {
  ContactArgs a;
  a.candA = s->cand;
  a.candB = s->cand + s->cand_cap;
  a.surv = s->cand + 3 * s->cand_cap;
  a.mid = s->cand + 4 * s->cand_cap;
  a.cand_cap = (unsigned)s->cand_cap;
  a.tets = s->tets;
  a.surf = s->surf;
  a.vs = vsrc(s);
  a.out = s->contacts;
  a.rec = s->records;
  a.out_cap = (unsigned)s->contact_cap;
  a.ctl = s->ctl;
  unsigned grid = (unsigned)s->ctx->sm_count * 8u;
  contacts_filter_kernel<<<grid, 256, 0, s->ctx->stream>>>(a);
  contacts_edge_kernel<<<grid, 256, 0, s->ctx->stream>>>(a);
  contacts_thread_kernel<<<grid * 2, 128, 0, s->ctx->stream>>>(a);
  s->ctx->launches += 3;
  return cudaGetLastError();
}

cudaError_t launch_adjoint(kdop_scene* s, const float* dd, const float* dn, float* grad) {
  AdjointArgs a;
  a.candA = s->cand;
  a.candB = s->cand + s->cand_cap;
  a.cand_cap = (unsigned)s->cand_cap;
  a.tets = s->tets;
  a.rec = s->records;
  a.dd = dd;
  a.dn = dn;
  a.out_cap = (unsigned)s->contact_cap;
  a.vs = vsrc(s);
  a.grad = grad;
  a.ctl = s->ctl;
  unsigned grid = (unsigned)s->ctx->sm_count * 8u;
  adjoint_kernel<<<grid, 128, 0, s->ctx->stream>>>(a);
  s->ctx->launches += 1;
  return cudaGetLastError();
}

}  // namespace kdop
