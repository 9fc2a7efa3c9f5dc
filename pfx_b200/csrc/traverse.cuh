// BVH traversal on the B200 layout (pfxt_types.h: WideNode, TravTri, InstRec).
//
// Closest hit restates scene() (crates/trace/src/trace.wgsl:999-1075, with
// tri_hit :780-804 and box_hit :453-468); any hit restates occluded()
// (:1096-1168, tri_blocks :1076-1095).  Both walk the reference's tree, the
// closest hit in the reference's order (left child first, right child when the
// left subtree is done).  What decides a hit is tested as the reference tests
// it: the same fp32 boxes with the same slab arithmetic (the quotients
// (lo - o)/d are correctly rounded, so they equal the reference's divisions
// bit for bit) and the same Moller-Trumbore test with the same operation order,
// so the hit slot, record and distance are bit-identical to the CPU oracle's.  Clip planes, cutouts, alpha, sprites,
// motion and analytic shapes are outside this library's scope; the scenes it
// accepts have none.
//
// Two walks.
//  * QuadWalker, the one the batch and queue kernels run: four-box nodes
//    (QuadNode) tested with quotients that are a rounding or two off and a
//    comparison widened by more than that, so it may open a box that the
//    reference skips but never skips one that the reference opens; where a
//    triangle would be accepted, its leaf's own box is tested as the reference
//    tests it, and the leaf is dropped if that fails.  Rays it cannot take are
//    marked for retry.
//  * Walker, on the two-box nodes with the reference's own box tests: the
//    work-counting kernels, the retry kernels (IEEE division throughout) and
//    queries inside shading code.
//
// The per-ray stack holds (entry, near) pairs.  `near` is the entry distance
// of the child box computed when its parent was opened; box_hit(node, hit.t)
// at pop time is exactly "geometry passes && near <= hit.t", so re-checking
// near against the current hit distance on pop reproduces the reference's
// pruning.  Walker's stack never holds more entries than the reference's
// 64-entry stack holds at the same point; scenes that would overflow that
// stack are refused when they are created.
//
// Work accounting (COUNT): the reference tests a node's box when it pops the
// node, and it pushes both children of every inner node it opens.  The
// counting variant therefore charges the left child when its parent is opened
// (the reference pops it next) and the right child when it is popped, pushing
// failed right children with near = +inf so they are charged, not visited.
#pragma once
#include "pfxt_math.h"
#include "pfxt_types.h"

namespace pfxt {

constexpr uint32_t STACK_SENTINEL = 0xfffffffeu;

struct SceneView {
  const WideNode* __restrict__ wide;
  const QuadNode* __restrict__ quad;  // by the index of the two-box node it stands for
  const TravTri* __restrict__ tris;
  const InstRec* __restrict__ insts;  // null in a scene without instances
  uint32_t root;
  uint32_t small;  // 1 when every box coordinate is 0 or in [BOUNDED_TINY, BOUNDED_COORD] in magnitude,
                   // lo <= hi, every box holds its children's, and every leaf's triangles hold its box
                   // (2: and a ray may come to hold more than QUAD_STACK entries, QuadWalker's GUARD)
};

struct TraceHit {
  float t;
  uint32_t slot;
  uint32_t record;
  uint32_t hit;
  float u, v;  // barycentrics of the closest hit (tri_fill's u, v)
};

// Box and triangle tests one query did, counted as the reference counts them.
struct TraceCounts {
  uint32_t boxes;
  uint32_t tris;
};

// The Markstein quotients of the box test below are the correctly rounded
// (lo - o)/d whenever nothing in them underflows or overflows.  That holds for
// every box of a "bounded" ray, with no check per quotient:
//  * box coordinates and ray origin components are 0 or of magnitude in
//    [2^-70, 2^79], so a numerator x = lo - o is 0 (exact) or of magnitude in
//    [2^-93, 2^80] (a nonzero difference of two such values is a multiple of
//    the smaller one's ulp, at least 2^-93);
//  * direction components are degenerate (below 1e-12, never divided by) or of
//    magnitude in [1e-12, 2^20], so a nonzero quotient lies in [2^-113, 2^120]
//    (normal, with margin), and the residual x - q d, a multiple of
//    ulp(q) ulp(d) >= 2^-141 (q d is within a few ulps of x), is exact.
// Box coordinates are checked once per scene (SceneView::small); origins and
// directions per ray, in world space and in every instance's space.
constexpr float BOUNDED_COORD = 0x1p+79f;
constexpr float BOUNDED_TINY = 0x1p-70f;
constexpr float BOUNDED_DIR = 0x1p+20f;

// A ray in the space it is being traversed in, with the per-axis reciprocal
// used by the quotients (only read on axes with |d| >= 1e-12).  The boxes of
// a ray that is not `bounded` are all tested with IEEE division.
struct TRay {
  v3 o, d, r;
  bool bounded;
};

__device__ __forceinline__ bool bounded_axis(float o, float d) {
  float ao = fabsf(o), ad = fabsf(d);
  return (ao == 0.0f || (ao >= BOUNDED_TINY && ao <= BOUNDED_COORD)) && (ad <= BOUNDED_DIR || ad < 1e-12f);
}

__device__ __forceinline__ TRay make_tray(v3 o, v3 d, uint32_t small) {
  TRay t;
  t.o = o;
  t.d = d;
  t.r = mk3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
  t.bounded = small != 0u && bounded_axis(o.x, d.x) && bounded_axis(o.y, d.y) && bounded_axis(o.z, d.z);
  return t;
}

// Slab test of one box with IEEE division throughout, for rays that are not
// bounded (see above).
__device__ __forceinline__ bool box_geometry_ieee_inline(float lx, float ly, float lz, float hx, float hy, float hz,
                                                         const TRay& ray, float& near) {
  float n = 0.0f, f = INFINITY;
  if (fabsf(ray.d.x) < 1e-12f) {
    if (ray.o.x < lx || ray.o.x > hx) return false;
  } else {
    float a = (lx - ray.o.x) / ray.d.x, b = (hx - ray.o.x) / ray.d.x;
    n = fmaxf(n, fminf(a, b));
    f = fminf(f, fmaxf(a, b));
  }
  if (fabsf(ray.d.y) < 1e-12f) {
    if (ray.o.y < ly || ray.o.y > hy) return false;
  } else {
    float a = (ly - ray.o.y) / ray.d.y, b = (hy - ray.o.y) / ray.d.y;
    n = fmaxf(n, fminf(a, b));
    f = fminf(f, fmaxf(a, b));
  }
  if (fabsf(ray.d.z) < 1e-12f) {
    if (ray.o.z < lz || ray.o.z > hz) return false;
  } else {
    float a = (lz - ray.o.z) / ray.d.z, b = (hz - ray.o.z) / ray.d.z;
    n = fmaxf(n, fminf(a, b));
    f = fminf(f, fmaxf(a, b));
  }
  near = n;
  return !(n > f);
}

// The same test out of line, for walks that take both kinds of ray (the work
// counting variant).
static __device__ __noinline__ bool box_geometry_ieee(float lx, float ly, float lz, float hx, float hy, float hz,
                                                      const TRay& ray, float& near) {
  return box_geometry_ieee_inline(lx, ly, lz, hx, hy, hz, ray, near);
}

// x / d by Markstein's correction from r = RN(1/d) (Markstein 1990; Cornea,
// Harrison and Tang, "Scientific Computing on Itanium-based Systems", 2002,
// ch. 8): with q = RN(x r) the residual fma(-q, d, x) is exact and
// RN(q + e r) is the correctly rounded quotient, provided nothing underflows
// or overflows, which a bounded ray guarantees.
__device__ __forceinline__ float quotient(float x, float d, float r) {
  float q = x * r;
  float e = fmaf(-q, d, x);
  return fmaf(e, r, q);
}

// Slab test of one box for a bounded ray: true when the ray's geometry passes
// (degenerate axes inside the slab, entry <= exit); `near` receives
// max(0, entries).  The six quotients equal IEEE division's (the reference
// divides).
__device__ __forceinline__ bool box_geometry_bounded(float lx, float ly, float lz, float hx, float hy, float hz,
                                                     const TRay& ray, float& near) {
  float n = 0.0f, f = INFINITY;
  if (fabsf(ray.d.x) < 1e-12f) {
    if (ray.o.x < lx || ray.o.x > hx) return false;
  } else {
    float a = quotient(lx - ray.o.x, ray.d.x, ray.r.x), b = quotient(hx - ray.o.x, ray.d.x, ray.r.x);
    n = fmaxf(n, fminf(a, b));
    f = fminf(f, fmaxf(a, b));
  }
  if (fabsf(ray.d.y) < 1e-12f) {
    if (ray.o.y < ly || ray.o.y > hy) return false;
  } else {
    float a = quotient(ly - ray.o.y, ray.d.y, ray.r.y), b = quotient(hy - ray.o.y, ray.d.y, ray.r.y);
    n = fmaxf(n, fminf(a, b));
    f = fminf(f, fmaxf(a, b));
  }
  if (fabsf(ray.d.z) < 1e-12f) {
    if (ray.o.z < lz || ray.o.z > hz) return false;
  } else {
    float a = quotient(lz - ray.o.z, ray.d.z, ray.r.z), b = quotient(hz - ray.o.z, ray.d.z, ray.r.z);
    n = fmaxf(n, fminf(a, b));
    f = fminf(f, fmaxf(a, b));
  }
  near = n;
  return !(n > f);
}

// Two fp32 lanes in one 64-bit register and the sm_100 paired instructions on
// them: each lane is one IEEE round-to-nearest subtraction or multiplication,
// the same operation as the scalar instruction, two per issue.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float lo, float hi) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpair(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// 1/x to within an ulp (the hardware's approximation), for the loose box test.
__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The sm_100 three-input minimum and maximum: the same value as two two-input
// ones (no NaN reaches them here; a signed zero only ever meets comparisons).
__device__ __forceinline__ float min3f(float a, float b, float c) {
  float r;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3f(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// How Walker tests boxes.
//  BOX_EITHER:  bounded rays with the Markstein quotients, other rays with the
//               out-of-line IEEE test (one walk for every ray; the call costs
//               the walk loop spills);
//  BOX_IEEE:    IEEE division throughout, inline.
// Both give the same bits for every box they test.
constexpr int BOX_EITHER = 0, BOX_IEEE = 2;

template <int BOX>
__device__ __forceinline__ bool box_test(float lx, float ly, float lz, float hx, float hy, float hz, const TRay& ray,
                                         float& near) {
  if (BOX == BOX_IEEE) return box_geometry_ieee_inline(lx, ly, lz, hx, hy, hz, ray, near);
  if (BOX == BOX_EITHER && !ray.bounded) return box_geometry_ieee(lx, ly, lz, hx, hy, hz, ray, near);
  return box_geometry_bounded(lx, ly, lz, hx, hy, hz, ray, near);
}

// to_object (trace.wgsl:449-452): (dot(lo,q), dot(hi,q), dot(rows2,q)), q=(p,w).
__device__ __forceinline__ v3 to_object(const float4& r0, const float4& r1, const float4& r2, v3 p, float w) {
  v3 o;
  o.x = ((r0.x * p.x + r0.y * p.y) + r0.z * p.z) + r0.w * w;
  o.y = ((r1.x * p.x + r1.y * p.y) + r1.z * p.z) + r1.w * w;
  o.z = ((r2.x * p.x + r2.y * p.y) + r2.z * p.z) + r2.w * w;
  return o;
}

// The traversal stack of one lane: (ref, near bits) pairs, one 8-byte store
// per push and one 8-byte load per pop (measured 1037 against 1011 Mrays/s
// with two 4-byte arrays).  With SHORT > 0 the first SHORT entries live in
// shared memory, one column per lane (entry k of lane t at word k * lanes + t,
// so a warp's accesses fall in distinct banks), and the rest in local memory;
// with SHORT == 0 all of it is local.  Only where entries are kept differs:
// the walk pushes and pops exactly the same entries.
template <int SHORT, int DEPTH>
struct LaneStack {
  static constexpr int CAPACITY = DEPTH;
  uint32_t* sh_ref;
  float* sh_near;
  uint32_t lanes;
  uint2 entry[DEPTH - SHORT];  // past the shared-memory top
  __device__ __forceinline__ void put(int k, uint32_t r, float n) {
    if (k < SHORT) {
      sh_ref[k * lanes] = r;
      sh_near[k * lanes] = n;
    } else {
      entry[k - SHORT] = make_uint2(r, __float_as_uint(n));
    }
  }
  __device__ __forceinline__ void get(int k, uint32_t& r, float& n) const {
    if (k < SHORT) {
      r = sh_ref[k * lanes];
      n = sh_near[k * lanes];
    } else {
      uint2 e = entry[k - SHORT];
      r = e.x;
      n = __uint_as_float(e.y);
    }
  }
};
template <int DEPTH>
struct LaneStack<0, DEPTH> {
  static constexpr int CAPACITY = DEPTH;
  uint2 entry[DEPTH];
  __device__ __forceinline__ void put(int k, uint32_t r, float n) { entry[k] = make_uint2(r, __float_as_uint(n)); }
  __device__ __forceinline__ void get(int k, uint32_t& r, float& n) const {
    uint2 e = entry[k];
    r = e.x;
    n = __uint_as_float(e.y);
  }
};
using RefStack = LaneStack<0, (int)REF_STACK>;
using QuadStack = LaneStack<0, (int)QUAD_STACK>;

// Resident warps per SM the traversal kernels are compiled for: it sets their
// register budget.
#ifndef TRACE_WARPS_PER_SM
#define TRACE_WARPS_PER_SM 32
#endif

// One 32-byte sector in one load (sm_100's 256-bit loads), as pairs.
__device__ __forceinline__ void load32(const void* p, f32x2 (&q)[4]) {
  asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(q[0]), "=l"(q[1]), "=l"(q[2]), "=l"(q[3]) : "l"(p));
}

// The nine numbers of a triangle that its test reads.
__device__ __forceinline__ void load_tri(const TravTri* t, v3& a, v3& e1, v3& e2) {
  f32x2 q[4];
  load32(t, q);
  unpair(q[0], a.x, a.y);
  unpair(q[1], a.z, e1.x);
  unpair(q[2], e1.y, e1.z);
  unpair(q[3], e2.x, e2.y);
  e2.z = __ldg(reinterpret_cast<const float*>(t) + 8);
}

// Lanes of each of `warps` resident warps that take rays when there are n.  A
// warp pays for the union of its lanes' walks, so few rays are spread over all
// the warps: 4097 closest rays 45.5 -> 37.7 us, a 960 x 540 adaptive render, whose
// last rounds and bounces are small, 98.9 -> 89.5 ms.
__host__ __device__ __forceinline__ uint32_t lanes_per_warp(uint32_t n, uint32_t warps) {
  const uint32_t per = (n + warps - 1u) / warps;
  return per < 1u ? 1u : (per < 32u ? per : 32u);
}

// The reference's triangle test (tri_hit, trace.wgsl:780-804): false when the
// ray misses; u, v and t otherwise.
template <bool ANY>
__device__ __forceinline__ bool tri_test(v3 o, v3 d, v3 a, v3 e1, v3 e2, float inv_det, uint32_t word, float& u,
                                         float& v, float& t) {
  v3 pv = cross3(d, e2);
  float det = dot3(e1, pv);
  float seen = det * inv_det;
  if (fabsf(seen) < 1e-9f) return false;
  if (!ANY && (word & ONE_SIDED) != 0u && seen < 0.0f) return false;
  float inv = 1.0f / det;
  v3 sv = sub3(o, a);
  u = dot3(sv, pv) * inv;
  if (u < 0.0f || u > 1.0f) return false;
  v3 qv = cross3(sv, e1);
  v = dot3(d, qv) * inv;
  if (v < 0.0f || u + v > 1.0f) return false;
  t = dot3(e2, qv) * inv;
  return true;
}

// One query's traversal state on the two-box nodes; the stack is the caller's.
template <bool ANY, bool COUNT, int BOX = BOX_EITHER>
struct Walker {
  TRay ray;     // ray in the current space (the world ray itself is the caller's: see inner_phase)
  float limit;
  uint32_t base, record, word;
  float inv_det;
  uint32_t ref;
  float near_cur;
  int top;
  bool done;
  TraceHit hit;
  TraceCounts counts;

  __device__ __forceinline__ void start(const SceneView& s, v3 wo, v3 wd, float lim) {
    ray = make_tray(wo, wd, s.small);
    limit = lim;
    base = record = word = 0u;
    inv_det = 1.0f;
    ref = s.root;
    near_cur = -INFINITY;
    top = 0;
    done = (s.root == REF_NONE);
    hit.t = lim;
    hit.slot = hit.record = hit.hit = 0u;
    hit.u = hit.v = 0.0f;
    counts.boxes = counts.tris = 0u;
  }

  template <class Stack>
  __device__ __forceinline__ void pop(const Stack& st) {
    if (top == 0) {
      done = true;
      return;
    }
    --top;
    st.get(top, ref, near_cur);
    if (COUNT && ref != STACK_SENTINEL) counts.boxes += 1u;
  }

  // Walk inner nodes until the current entry is a leaf that passes its
  // near check, or the traversal is finished.  world(o, d) gives the world
  // ray again where an instance is entered or left (the walk keeps only the
  // ray of the current space; callers read it back from where it came from).
  template <class Stack, class World>
  __device__ __forceinline__ void inner_phase(const SceneView& s, Stack& st, const World& world) {
    while (!done) {
      if (ref == STACK_SENTINEL) {
        v3 o, d;
        world(o, d);
        ray = make_tray(o, d, s.small);
        base = record = word = 0u;
        inv_det = 1.0f;
        pop(st);
        continue;
      }
      if (!(near_cur <= hit.t)) {
        pop(st);
        continue;
      }
      if ((ref & REF_LEAF) == 0u) {
        const float4* p = reinterpret_cast<const float4*>(s.wide + ref);
        uint4 q3 = __ldg(reinterpret_cast<const uint4*>(p + 3));
        float n0 = 0.0f, n1 = 0.0f;
        bool has1 = q3.y != REF_NONE;
        float4 q0 = __ldg(p + 0), q1 = __ldg(p + 1), q2 = __ldg(p + 2);
        bool ok0 = box_test<BOX>(q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, ray, n0) && n0 <= hit.t;
        bool ok1 = has1 && box_test<BOX>(q1.z, q1.w, q2.x, q2.y, q2.z, q2.w, ray, n1) && n1 <= hit.t;
        if (COUNT) counts.boxes += 1u;  // the left child, popped next by the reference
        if ((ok1 || (COUNT && has1)) && top < Stack::CAPACITY) {
          st.put(top, q3.y, ok1 ? n1 : INFINITY);
          ++top;
        }
        if (ok0) {
          ref = q3.x;
          near_cur = n0;
        } else {
          pop(st);
        }
        continue;
      }
      if ((ref & REF_INST) == REF_INST) {
        if (top >= Stack::CAPACITY) {  // refused at creation; never taken
          pop(st);
          continue;
        }
        const float4* p = reinterpret_cast<const float4*>(s.insts + (ref & 0x3fffffffu));
        float4 r0 = __ldg(p + 0), r1 = __ldg(p + 1), r2 = __ldg(p + 2);
        uint4 m = __ldg(reinterpret_cast<const uint4*>(p + 3));
        float4 m2 = __ldg(p + 4);
        st.put(top, STACK_SENTINEL, -INFINITY);
        ++top;
        base = m.y;
        record = m.z;
        word = m.w;
        inv_det = m2.x;
        if (__float_as_uint(m2.y) != 0u) {
          v3 o, d;
          world(o, d);
          ray = make_tray(to_object(r0, r1, r2, o, 1.0f), to_object(r0, r1, r2, d, 0.0f), s.small);
        }
        ref = m.x;
        near_cur = -INFINITY;
        continue;
      }
      return;  // a leaf that passed its near check
    }
  }

  // Test the triangles of the current leaf, then move to the next entry.
  template <class Stack>
  __device__ __forceinline__ void leaf_phase(const SceneView& s, Stack& st) {
    uint32_t first = ref & LEAF_FIRST_MASK;
    uint32_t n = ((ref >> LEAF_FIRST_BITS) & 15u) + 1u;
    bool skip = ANY ? ((word & CASTS_NO_SHADOW) != 0u) : ((word & SHADOW_ONLY) != 0u);
    if (COUNT && skip) counts.tris += n;
    if (!skip) {
      for (uint32_t j = 0; j < n; ++j) {
        if (COUNT) counts.tris += 1u;  // the reference stops counting at an any-hit blocker
        uint32_t i = base + first + j;
        v3 a, e1, e2;
        load_tri(s.tris + i, a, e1, e2);
        float u, v, t;
        if (!tri_test<ANY>(ray.o, ray.d, a, e1, e2, inv_det, word, u, v, t)) continue;
        if (ANY) {
          if (t <= 0.0001f || t >= limit) continue;
          hit.hit = 1u;
          hit.t = t;
          hit.slot = i;
          hit.record = record;
          done = true;
          return;
        } else if (t > 0.0001f && t < hit.t) {
          hit.t = t;
          hit.slot = i;
          hit.record = record;
          hit.hit = 1u;
          hit.u = u;
          hit.v = v;
        }
      }
    }
    pop(st);
  }

  // Run to completion (one query, no work sharing).  FLAT: leave the loop between
  // the phases, which decides where the compiler brings a warp's lanes together
  // again.  The retry kernels, on 2^21 rays of two axes: a room of 100k triangles
  // closest 767 us FLAT and 952 not, any 468 and 632; the instanced scene 5.97 ms
  // and 3.04, 2.37 and 1.63.
  template <bool FLAT = false, class Stack, class World>
  __device__ __forceinline__ void run(const SceneView& s, Stack& st, const World& world) {
    while (!done) {
      inner_phase(s, st, world);
      if (FLAT && done) break;
      if (FLAT || !done) leaf_phase(s, st);
    }
  }
};

// The walk of the batch and queue kernels, on the four-box nodes.
//
// What it may skip.  The reference tests a leaf's triangles when the leaf's box
// and every ancestor's passed, each against the hit distance at its turn.  The
// fp32 quotients are monotone in the plane, so in one space a box that passes
// implies that the boxes holding it pass, with entries no larger, and hit
// distances only shrink: the leaf's own exact test at its turn decides alone
// (and, for an instance, the instance leaf's in world space).  Every box on
// the way down may therefore be skipped or tested loosely, as long as nothing
// that holds a passing leaf is dropped.
//
// The loose test.  A plane's quotient is x * r with x = lo - o rounded as the
// reference rounds it and r within an ulp of 1/d: within 2^-21 of the
// reference's quotient x / d in relative terms for a bounded ray (no
// underflow); entry and exit are their minima and maxima as the reference takes
// them.  Entry <= exit and entry <= hit.t are compared with the right side
// scaled by 1 + 2^-18, so a box that passes exactly passes here.
//
// The exact test (box_exact) runs where it decides: before the first triangle
// of a leaf is accepted, against the hit distance from before that leaf, and
// when an instance is entered.
//
// What bounds it.  The two-box walk spent 24 instructions on each box and, at
// 10 to 13 of 32 lanes, issue slots (70 % busy).  Four boxes a visit, tested
// loosely, and votes that name every lane leave half the warp instructions at
// 18 to 20 lanes, and the L1's handling of divergent sectors (84 % busy for
// shadow rays) bounds it: hence planes stored so that one 32-byte load brings
// a whole sector of an axis, four loads a node (with six 16-byte loads of the
// planes that the ray's signs pick: 1897 and 1048 us instead of 1797 and 925).
// Start to now, one B200: room closest 2^21 rays 2646 -> 1797 us, room any
// 1.5 M rays 1100 -> 925 us (523 by the order below), instanced closest and any
// 0.5 M rays 476 -> 355 and 518 -> 403 us (359).  32 resident warps (64 registers) beat 24, 28, 36 and 40.
//
// Order.  An any-hit answer does not depend on it, and a blocker is mostly near:
// the nearest child goes first (1.5 M shadow rays in the room 925 -> 523 us,
// instanced 406 -> 359).  For a closest hit children are visited in the
// reference's left-first order (nearest first took 973 instead of 1794 us on the
// room's 2^21 rays, and the same hits on 1.26 billion rays, but 12 of 10,000 rays
// aimed to within 1e-8 rad along a triangle's plane ended elsewhere: such a
// triangle's distance is off by any amount, so its box tells nothing) and a
// popped entry is checked again against the current distance, so the leaves
// tested, their order and the distance at each are the reference's.  A lane
// that reaches a leaf while other lanes of its warp still walk inner nodes
// sets the leaf aside (`held`) and walks on, so that the warp's leaf tests run
// with more lanes at once (Aila and Laine, "Understanding the efficiency of
// ray traversal on GPUs", 2009): the held leaf is the next one in the
// reference's order and is tested before any other, and what the lane walked
// past it was decided against a distance no smaller than the reference's.  A
// held leaf is tested before the walk enters or leaves an instance, so it is
// tested in its own space.
constexpr float LOOSE = 1.0f + 0x1p-18f;
// Lanes with a leaf set aside that send the warp to its leaf tests.  Measured
// (us; room closest 2^21 rays, room any 1.5 M, instanced closest and any 0.5 M):
// only when nobody looks any more 1922, 1072, 377, 445; 12 lanes 1970, 1060,
// 341, 401; 16 lanes 1897, 1048, 343, 410; 20 lanes 1867, 1041, 358, 420; as
// many as still look 1984, 1043, 334, 392 (16-byte node loads).
constexpr int HOLDERS = 16;

// GUARD: a ray that may find no room on the stack for what a node pushes is
// handed over.  Scenes whose rays cannot (TraversalLayout::stack_need) walk
// without: checked at every node, as a branch or with the votes, their rays paid
// 1 % (room closest 2^21 rays 1216 -> 1226 us) and a 320 x 180 preview 1 to 4 %.
template <bool ANY, bool GUARD = false>
struct QuadWalker {
  // the ray of the current space: origins and approximate reciprocals in both
  // lanes of a pair (a node's planes come two children to a pair), and the
  // direction
  f32x2 ox, oy, oz, rx, ry, rz;
  v3 d;
  uint32_t inst;  // the instance the walk is in, REF_NONE in world space
  uint32_t ref;   // the entry at hand, REF_NONE when there is none
  float near_cur;
  int top;
  uint32_t held;  // the leaf set aside, REF_NONE when none
  TraceHit hit;   // any hit: t stays the limit; record: the instance until `record()` gives its record

  static constexpr uint32_t RETRY = 2u;  // hit.hit of a ray to be walked again with BOX_IEEE: not bounded, or
                                         // with a degenerate axis, in world or instance space, or (GUARD)
                                         // without room on its stack

  // A lane without a ray.
  __device__ __forceinline__ void idle() { ref = held = REF_NONE; }

  // Ends the walk (GUARD): the ray is walked again.
  __device__ __forceinline__ void hand_over() {
    hit.hit = RETRY;
    ref = held = REF_NONE;
  }

  // False when the ray cannot be taken (the walk is then over).
  __device__ __forceinline__ bool aim(const SceneView& s, v3 o, v3 dir) {
    if (!(s.small != 0u && bounded_axis(o.x, dir.x) && bounded_axis(o.y, dir.y) && bounded_axis(o.z, dir.z) &&
          fabsf(dir.x) >= 1e-12f && fabsf(dir.y) >= 1e-12f && fabsf(dir.z) >= 1e-12f)) {
      hit.hit = RETRY;
      ref = REF_NONE;
      return false;
    }
    ox = pair(o.x, o.x);
    oy = pair(o.y, o.y);
    oz = pair(o.z, o.z);
    const float r0 = rcp_approx(dir.x), r1 = rcp_approx(dir.y), r2 = rcp_approx(dir.z);
    rx = pair(r0, r0);
    ry = pair(r1, r1);
    rz = pair(r2, r2);
    d = dir;
    return true;
  }

  __device__ __forceinline__ void start(const SceneView& s, v3 wo, v3 wd, float lim) {
    inst = REF_NONE;
    ref = s.root;
    near_cur = -INFINITY;
    top = 0;
    held = REF_NONE;
    hit.t = lim;
    hit.slot = hit.hit = 0u;
    hit.record = REF_NONE;
    hit.u = hit.v = 0.0f;
    if (ref != REF_NONE) aim(s, wo, wd);
  }

  // The surface record of the hit (0: the world's, or no hit).
  __device__ __forceinline__ uint32_t record(const SceneView& s) const {
    return hit.record == REF_NONE ? 0u : __ldg(&s.insts[hit.record].record);
  }

  // The next entry that the current hit distance leaves.
  template <class Stack>
  __device__ __forceinline__ void pop(const Stack& st) {
    do {
      if (top == 0) {
        ref = REF_NONE;
        return;
      }
      --top;
      st.get(top, ref, near_cur);
    } while (!(near_cur <= hit.t * LOOSE));
  }

  __device__ __forceinline__ v3 origin() const {
    float x, y, z, spare;
    unpair(ox, x, spare);
    unpair(oy, y, spare);
    unpair(oz, z, spare);
    return mk3(x, y, z);
  }

  // The reference's test of one box (box_geometry_bounded for a ray without a
  // degenerate axis) against the hit distance `reach`.
  __device__ __forceinline__ bool box_exact(float lx, float ly, float lz, float hx, float hy, float hz,
                                            float reach) const {
    const v3 o = origin();
    float r = 1.0f / d.x;
    float a = quotient(lx - o.x, d.x, r), b = quotient(hx - o.x, d.x, r);
    float n = fmaxf(0.0f, fminf(a, b)), f = fmaxf(a, b);
    r = 1.0f / d.y;
    a = quotient(ly - o.y, d.y, r), b = quotient(hy - o.y, d.y, r);
    n = fmaxf(n, fminf(a, b)), f = fminf(f, fmaxf(a, b));
    r = 1.0f / d.z;
    a = quotient(lz - o.z, d.z, r), b = quotient(hz - o.z, d.z, r);
    n = fmaxf(n, fminf(a, b)), f = fminf(f, fmaxf(a, b));
    return !(n > f) && n <= reach;
  }

  // Opens the inner node at hand: tests its four children loosely.  Closest hit:
  // the first that passes is next, the others are pushed last first; any hit:
  // the nearest is next.  An unused child passes too (its planes are both
  // infinite), but unused children are last, so they are looked at while `next`
  // is still REF_NONE, and leave it so: nothing is pushed for them.
  template <class Stack>
  __device__ __forceinline__ void open(const SceneView& s, Stack& st) {
    if (GUARD && top > Stack::CAPACITY - 3) {  // three children may wait
      hand_over();
      return;
    }
    const char* p = reinterpret_cast<const char*>(s.quad + ref);
    const uint4 c = __ldg(reinterpret_cast<const uint4*>(p + 96));
    f32x2 x[4], y[4], z[4];  // lo of children 0-1 and 2-3, hi of 0-1 and 2-3
    load32(p, x);
    load32(p + 32, y);
    load32(p + 64, z);
    uint32_t next = REF_NONE;
    float next_near = 0.0f;
#pragma unroll
    for (int h = 1; h >= 0; --h) {
      float xl[2], yl[2], zl[2], xh[2], yh[2], zh[2];
      unpair(mul2(sub2(x[h], ox), rx), xl[0], xl[1]);
      unpair(mul2(sub2(y[h], oy), ry), yl[0], yl[1]);
      unpair(mul2(sub2(z[h], oz), rz), zl[0], zl[1]);
      unpair(mul2(sub2(x[2 + h], ox), rx), xh[0], xh[1]);
      unpair(mul2(sub2(y[2 + h], oy), ry), yh[0], yh[1]);
      unpair(mul2(sub2(z[2 + h], oz), rz), zh[0], zh[1]);
#pragma unroll
      for (int k = 1; k >= 0; --k) {
        const float entry = fmaxf(max3f(fminf(xl[k], xh[k]), fminf(yl[k], yh[k]), fminf(zl[k], zh[k])), 0.0f);
        const float exit = fminf(min3f(fmaxf(xl[k], xh[k]), fmaxf(yl[k], yh[k]), fmaxf(zl[k], zh[k])), hit.t);
        if (entry <= exit * LOOSE) {
          const uint32_t child = h ? (k ? c.w : c.z) : (k ? c.y : c.x);
          if (ANY && next != REF_NONE && entry >= next_near) {
            st.put(top++, child, entry);
          } else {
            if (next != REF_NONE) st.put(top++, next, next_near);
            next = child;
            next_near = entry;
          }
        }
      }
    }
    if (next != REF_NONE) {
      ref = next;
      near_cur = next_near;
    } else {
      pop(st);
    }
  }

  // Whether the entry at hand enters or leaves an instance.
  __device__ __forceinline__ bool at_instance() const {
    return ref != REF_NONE && (ref & REF_INST) == REF_INST;
  }
  static_assert((STACK_SENTINEL & REF_INST) == REF_INST, "the sentinel is told from leaves by the instance bits");

  // Sets the leaf at hand aside.
  template <class Stack>
  __device__ __forceinline__ void take_leaf(const Stack& st) {
    if (held == REF_NONE && (ref & REF_INST) == REF_LEAF) {
      held = ref;
      pop(st);
    }
  }

  // Enters or leaves the instance at hand.  Only without a held leaf, which is
  // tested in its own space.
  template <class Stack, class World>
  __device__ __forceinline__ void cross_instance(const SceneView& s, Stack& st, const World& world) {
    if (ref == STACK_SENTINEL) {
      v3 o, dir;
      world(o, dir);
      aim(s, o, dir);
      inst = REF_NONE;
      pop(st);
      return;
    }
    const uint32_t index = ref & 0x3fffffffu;
    const float4* p = reinterpret_cast<const float4*>(s.insts + index);
    const uint32_t root = __ldg(reinterpret_cast<const uint32_t*>(p + 3));
    const float4 m2 = __ldg(p + 4), m3 = __ldg(p + 5);
    if (!box_exact(m2.z, m2.w, m3.x, m3.y, m3.z, m3.w, hit.t)) {
      pop(st);
      return;
    }
    if (GUARD && top >= Stack::CAPACITY) {
      hand_over();
      return;
    }
    st.put(top++, STACK_SENTINEL, -INFINITY);
    inst = index;
    ref = root;
    near_cur = -INFINITY;
    if (__float_as_uint(m2.y) != 0u) {
      const float4 r0 = __ldg(p + 0), r1 = __ldg(p + 1), r2 = __ldg(p + 2);
      v3 o, dir;
      world(o, dir);
      aim(s, to_object(r0, r1, r2, o, 1.0f), to_object(r0, r1, r2, dir, 0.0f));
    }
  }

  // Walks every lane's inner nodes until enough lanes hold a leaf; called by
  // all 32 lanes.  world(o, d): as Walker::inner_phase.  The votes name every
  // lane, so the warp takes each step together: with votes among whichever
  // lanes had come together, a warp fell apart (5.4 lanes an instruction
  // against 8.6 on a small frame's rays).
  template <class Stack, class World>
  __device__ __forceinline__ void inner_phase(const SceneView& s, Stack& st, const World& world) {
    constexpr unsigned FULL = 0xffffffffu;
    for (;;) {
      take_leaf(st);
      if (__any_sync(FULL, at_instance() && held == REF_NONE)) {
        if (at_instance() && held == REF_NONE) cross_instance(s, st, world);
        continue;
      }
      const bool inner = (ref & REF_LEAF) == 0u;
      // Lanes that hold a leaf walk on while others still look for one, until
      // half the warp holds one or nobody looks any more.
      const unsigned look = __ballot_sync(FULL, inner && held == REF_NONE);
      if (look == 0u) break;
      if (__popc(__ballot_sync(FULL, held != REF_NONE)) >= HOLDERS) break;
      if (inner) open(s, st);
    }
  }

  // Is there a leaf to test?  Without one, inner_phase has ended the walk.
  __device__ __forceinline__ bool leaf_ready() const { return held != REF_NONE; }
  __device__ __forceinline__ bool finished() const { return ref == REF_NONE && held == REF_NONE; }

  // Test the triangles of the held leaf; the entry at hand stays, checked
  // again against the new distance.
  template <class Stack>
  __device__ __forceinline__ void leaf_phase(const SceneView& s, Stack& st) {
    uint32_t i = held & LEAF_FIRST_MASK, word = 0u;
    const uint32_t n = ((held >> LEAF_FIRST_BITS) & 15u) + 1u;
    float inv_det = 1.0f;
    held = REF_NONE;
    if (inst != REF_NONE) {
      const InstRec* r = s.insts + inst;
      i += __ldg(&r->base);
      word = __ldg(&r->word);
      inv_det = __ldg(&r->inv_det);
      if (ANY ? ((word & CASTS_NO_SHADOW) != 0u) : ((word & SHADOW_ONLY) != 0u)) return;
    }
    const float reach = hit.t;
    const v3 o = origin();
    bool checked = false;
    for (const uint32_t end = i + n; i < end; ++i) {
      const TravTri* tri = s.tris + i;
      v3 a, e1, e2;
      load_tri(tri, a, e1, e2);
      float u, v, t;
      if (!tri_test<ANY>(o, d, a, e1, e2, inv_det, word, u, v, t)) continue;
      if (ANY ? (t <= 0.0001f || t >= hit.t) : !(t > 0.0001f && t < hit.t)) continue;
      if (!checked) {
        const float* b = tri->lo;
        if (!box_exact(__ldg(b), __ldg(b + 1), __ldg(b + 2), __ldg(b + 3), __ldg(b + 4), __ldg(b + 5), reach)) return;
        checked = true;
      }
      hit.hit = 1u;
      if (ANY) {
        ref = REF_NONE;
        return;
      }
      hit.t = t;
      hit.slot = i;
      hit.record = inst;
      hit.u = u;
      hit.v = v;
    }
    if (ref != REF_NONE && !(near_cur <= hit.t * LOOSE)) pop(st);
  }
};

// Single-query helpers used by shading code.
template <bool ANY>
__device__ __forceinline__ TraceHit traverse(const SceneView& s, v3 o, v3 d, float limit) {
  RefStack st;
  Walker<ANY, false, BOX_EITHER> w;
  w.start(s, o, d, limit);
  w.run(s, st, [&](v3& wo, v3& wd) {
    wo = o;
    wd = d;
  });
  return w.hit;
}

}  // namespace pfxt
