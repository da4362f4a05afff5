// Per-ray traversal device code shared by the one-structure kernels
// (trace.cu) and the persistent many-structure kernel (trace_batched.cu).
#pragma once
#include <type_traits>

#include "rq_device.cuh"
#include "rq_internal.hpp"

namespace rq {

struct Ray {
  F3 o, d;
  float tmin, tmax;
};

// Rays are read once: streaming loads (evict first), which leave L1 and L2
// to the tree's nodes and primitives.
__device__ __forceinline__ Ray load_ray(const float4* __restrict__ rays, uint32_t r) {
  float4 a = __ldcs(rays + 2 * (size_t)r), b = __ldcs(rays + 2 * (size_t)r + 1);
  return {{a.x, a.y, a.z}, {b.x, b.y, b.z}, a.w, b.w};
}

struct Closest {
  float t;
  uint32_t prim;
  float u, v;
};
// Hits are written once: a streaming store.
__device__ __forceinline__ void store_hit(float4* __restrict__ hits, uint32_t r, const Closest& c) {
  __stcs(hits + r, make_float4(c.t, __uint_as_float(c.prim), c.u, c.v));
}

// Test the primitives of one leaf.  Returns true when an any-hit query is done.
// FAST closest hit (REF = false) keeps the smallest t and, among primitives
// hit at exactly that t, the smallest primitive id, so the result does not
// depend on the order in which a walk meets the primitives.  REF keeps the
// reference's first closest (strict <, castRay main.cpp:343-358).
template <int KIND, bool ANY, bool REF>
__device__ __forceinline__ bool test_leaf(const float4* __restrict__ prims,
                                          const uint32_t* __restrict__ order, uint32_t first,
                                          int count, const Ray& ray, Closest& c) {
  for (int k = 0; k < count; ++k) {
    uint32_t slot = first + (uint32_t)k;
    // closest hit: accept t <= c.t once something is hit (ties go to the smaller id)
    const float bound = (ANY || REF || c.prim == kMiss) ? c.t : nextafterf(c.t, __int_as_float(0x7F800000));
    if (KIND == kTriangles) {
      float4 p0 = __ldg(prims + 3 * (size_t)slot), p1 = __ldg(prims + 3 * (size_t)slot + 1),
             p2 = __ldg(prims + 3 * (size_t)slot + 2);
      float t, u, v;
      if (tri_mt(p0, p1, p2, ray.o, ray.d, ray.tmin, ANY ? ray.tmax : bound, t, u, v)) {
        if (ANY) return true;
        const uint32_t id = __float_as_uint(p0.w);
        if (REF || t < c.t || id < c.prim) c = {t, id, u, v};
      }
    } else {
      float4 s = __ldg(prims + slot);
      if (ANY) {
        float t0, t1, t;
        if (REF ? sphere_ref(s, ray.o, ray.d, t0, t1)
                : sphere_closest(s, ray.o, ray.d, ray.tmin, ray.tmax, false, t))
          return true;
      } else {
        float t;
        if (sphere_closest(s, ray.o, ray.d, ray.tmin, bound, REF, t)) {
          const uint32_t id = __ldg(order + slot);
          if (REF || t < c.t || id < c.prim) c = {t, id, 0.f, 0.f};
        }
      }
    }
  }
  return false;
}

// Primitive tests one leaf visit performs: every primitive for closest hit;
// up to and including the first accepted one for any hit (the oracle's count).
template <int KIND, bool ANY>
__device__ __forceinline__ uint32_t test_count(const float4* __restrict__ prims, uint32_t first, int count,
                                               const Ray& ray) {
  if (!ANY) return (uint32_t)count;
  Closest dummy = {ray.tmax, kMiss, 0.f, 0.f};
  for (int k = 0; k < count; ++k)
    if (test_leaf<KIND, true, false>(prims, nullptr, first + (uint32_t)k, 1, ray, dummy)) return (uint32_t)k + 1;
  return (uint32_t)count;
}

// One 64-byte BVH2 node as two 256-bit loads (nodes are 64-byte aligned).
__device__ __forceinline__ void load_node(const float4* nd, float4& a, float4& b, float4& z, int4& l) {
  uint32_t r[16];
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "l"(nd));
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "l"(nd + 2));
  a = make_float4(__uint_as_float(r[0]), __uint_as_float(r[1]), __uint_as_float(r[2]), __uint_as_float(r[3]));
  b = make_float4(__uint_as_float(r[4]), __uint_as_float(r[5]), __uint_as_float(r[6]), __uint_as_float(r[7]));
  z = make_float4(__uint_as_float(r[8]), __uint_as_float(r[9]), __uint_as_float(r[10]), __uint_as_float(r[11]));
  l = make_int4((int)r[12], (int)r[13], (int)r[14], (int)r[15]);
}

// FAST walk of one ray through a BVH2: near child first, far child on a
// per-thread stack of STACK entries, boxes clipped to [tmin, closest hit].
// EXACT: the exact-sign box test (rays with a zero direction component).
// Returns true when an any-hit query found a hit.
// UNIT: every leaf holds one primitive (LBVH), so a stack entry is the
// 4-byte link alone: half the local-memory footprint, which shares L1 with
// the nodes the walk fetches.
template <int KIND, bool ANY, bool COUNT, int STACK, bool EXACT, bool UNIT = false>
__device__ __forceinline__ bool walk_bvh2_form(const Bvh2View& bvh, const Ray& ray, const SlabRay& sr, Closest& c,
                                               uint32_t& visits, uint32_t& tests, uint32_t* err) {
  float tn;
  const float* rb = bvh.root;
  if (!slab_box<EXACT>(sr, ray.o, rb[0], rb[3], rb[1], rb[4], rb[2], rb[5], ray.tmin, ray.tmax, tn)) return false;
  typename std::conditional<UNIT, int, int2>::type stack[STACK];
  int sp = 0;
  int cur = bvh.n_internal ? 0 : -1;
  int cnt = bvh.n_internal ? 0 : (int)bvh.n_slots;
  // A valid walk visits every node at most once.
  const uint32_t max_steps = 2u * (bvh.n_internal + bvh.n_slots) + 8u;
  uint32_t steps = 0;
  for (;;) {
    if (++steps > max_steps) { atomicOr(err, kErrCorrupt); return false; }
    if (cur >= 0) {
      float4 a, b, z;
      int4 l;
      const float4* nd = bvh.nodes + 4 * (size_t)cur;
      if (ANY) {  // any hit measured 1% faster with four 128-bit loads, closest hit 2% slower
        a = __ldg(nd); b = __ldg(nd + 1); z = __ldg(nd + 2);
        l = __ldg(reinterpret_cast<const int4*>(nd + 3));
      } else {
        load_node(nd, a, b, z, l);
      }
      if (COUNT) ++visits;
      const float tfar = ANY ? ray.tmax : c.t;
      float tl, tr;
      bool hl = slab_box<EXACT>(sr, ray.o, a.x, a.y, a.z, a.w, z.x, z.y, ray.tmin, tfar, tl);
      bool hr = slab_box<EXACT>(sr, ray.o, b.x, b.y, b.z, b.w, z.z, z.w, ray.tmin, tfar, tr);
      if (hl && hr) {
        int2 nearE = make_int2(l.x, l.z), farE = make_int2(l.y, l.w);
        if (tr < tl) { int2 t = nearE; nearE = farE; farE = t; }
        if (sp >= STACK) { atomicOr(err, kErrStackOverflow); return false; }
        if constexpr (UNIT) stack[sp++] = farE.x;
        else stack[sp++] = farE;
        cur = nearE.x;
        cnt = nearE.y;
        continue;
      }
      if (hl) { cur = l.x; cnt = l.z; continue; }
      if (hr) { cur = l.y; cnt = l.w; continue; }
    } else {
      if (UNIT) cnt = 1;
      if (COUNT) tests += test_count<KIND, ANY>(bvh.prims, (uint32_t)(~cur), cnt, ray);
      if (test_leaf<KIND, ANY, false>(bvh.prims, bvh.order, (uint32_t)(~cur), cnt, ray, c)) return true;
    }
    if (sp == 0) return false;
    if constexpr (UNIT) {
      cur = stack[--sp];
    } else {
      const int2 e = stack[--sp];
      cur = e.x;
      cnt = e.y;
    }
  }
}

// walk_bvh2_form with the box test each ray needs.
template <int KIND, bool ANY, bool COUNT, int STACK, bool UNIT = false>
__device__ __forceinline__ bool walk_bvh2(const Bvh2View& bvh, const Ray& ray, Closest& c, uint32_t& visits,
                                          uint32_t& tests, uint32_t* err) {
  const SlabRay sr = slab_ray(ray.o, ray.d);
  return zero_dir(sr) ? walk_bvh2_form<KIND, ANY, COUNT, STACK, true, UNIT>(bvh, ray, sr, c, visits, tests, err)
                      : walk_bvh2_form<KIND, ANY, COUNT, STACK, false, UNIT>(bvh, ray, sr, c, visits, tests, err);
}

// Sum the per-thread visit / test counts of a warp into counters[0..1].
__device__ __forceinline__ void add_counts(unsigned long long* counters, uint32_t visits, uint32_t tests) {
  unsigned long long v = visits, t = tests;
  for (int o = 16; o > 0; o >>= 1) {
    v += __shfl_down_sync(0xffffffffu, v, o);
    t += __shfl_down_sync(0xffffffffu, t, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(counters, v);
    atomicAdd(counters + 1, t);
  }
}

// ---------------------------------------------------------------- 4-wide
// FAST traversal of the collapsed 4-wide BVH: one 128-byte node fetch tests
// up to four child boxes.  The hit children are ordered by a 32-bit key, the
// order-preserving bits of the entry distance with the low two bits replaced
// by the slot (unique keys, so a sorting network gives the same order as any
// sort); the nearest is visited next and the others pushed farthest first.
// Three entries per level at most: 96 stack entries cover trees 64 binary
// levels deep, like the binary walk's 64.
constexpr int kStack4 = 96;

__device__ __forceinline__ uint32_t order_key(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ void cswap(uint32_t& a, uint32_t& b) {
  uint32_t lo = min(a, b), hi = max(a, b);
  a = lo;
  b = hi;
}

__device__ __forceinline__ int pick(const int4& v, uint32_t k) {
  return k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
}

// FAST walk of one ray through the collapsed 4-wide BVH.  Returns true when
// an any-hit query found a hit.
template <int KIND, bool ANY, bool COUNT, int STACK, bool EXACT>
__device__ __forceinline__ bool walk_bvh4_form(const Bvh4View& bvh, const Ray& ray, Closest& c, uint32_t& visits,
                                               uint32_t& tests, uint32_t* err) {
  const SlabRay sr = slab_ray(ray.o, ray.d);
  float tn;
  const float* rb = bvh.root;
  if (!slab_box<EXACT>(sr, ray.o, rb[0], rb[3], rb[1], rb[4], rb[2], rb[5], ray.tmin, ray.tmax, tn)) return false;
  int2 stack[STACK];
  int sp = 0;
  int cur = bvh.n_binary ? 0 : -1;
  int cnt = bvh.n_binary ? 0 : (int)bvh.n_slots;
  // A valid walk visits every node and leaf at most once.
  const uint32_t max_steps = 2u * (bvh.n_binary + bvh.n_slots) + 8u;
  uint32_t steps = 0;
  for (;;) {
    if (++steps > max_steps) { atomicOr(err, kErrCorrupt); return false; }
    if (cur >= 0) {
      const float4* nd = bvh.nodes + 8 * (size_t)cur;
      const float4 lx = __ldg(nd), hx = __ldg(nd + 1), ly = __ldg(nd + 2), hy = __ldg(nd + 3);
      const float4 lz = __ldg(nd + 4), hz = __ldg(nd + 5);
      const int4 lk = __ldg(reinterpret_cast<const int4*>(nd + 6));
      const int4 ct = __ldg(reinterpret_cast<const int4*>(nd + 7));
      if (COUNT) ++visits;
      const float tfar = ANY ? ray.tmax : c.t;
      float t0, t1, t2, t3;
      uint32_t k0 = 0xFFFFFFFFu, k1 = 0xFFFFFFFFu, k2 = 0xFFFFFFFFu, k3 = 0xFFFFFFFFu;
      if (ct.x >= 0 && slab_box<EXACT>(sr, ray.o, lx.x, hx.x, ly.x, hy.x, lz.x, hz.x, ray.tmin, tfar, t0))
        k0 = (order_key(t0) & ~3u) | 0u;
      if (ct.y >= 0 && slab_box<EXACT>(sr, ray.o, lx.y, hx.y, ly.y, hy.y, lz.y, hz.y, ray.tmin, tfar, t1))
        k1 = (order_key(t1) & ~3u) | 1u;
      if (ct.z >= 0 && slab_box<EXACT>(sr, ray.o, lx.z, hx.z, ly.z, hy.z, lz.z, hz.z, ray.tmin, tfar, t2))
        k2 = (order_key(t2) & ~3u) | 2u;
      if (ct.w >= 0 && slab_box<EXACT>(sr, ray.o, lx.w, hx.w, ly.w, hy.w, lz.w, hz.w, ray.tmin, tfar, t3))
        k3 = (order_key(t3) & ~3u) | 3u;
      // A hit key is at most order_key(+inf) | 3 < 0xFFFFFFFF, so misses sort last.
      const int m = (k0 != 0xFFFFFFFFu) + (k1 != 0xFFFFFFFFu) + (k2 != 0xFFFFFFFFu) + (k3 != 0xFFFFFFFFu);
      if (m > 0) {
        cswap(k0, k1);
        cswap(k2, k3);
        cswap(k0, k2);
        cswap(k1, k3);
        cswap(k1, k2);
        if (sp + m - 1 > STACK) { atomicOr(err, kErrStackOverflow); return false; }
        if (m >= 4) stack[sp++] = make_int2(pick(lk, k3 & 3u), pick(ct, k3 & 3u));
        if (m >= 3) stack[sp++] = make_int2(pick(lk, k2 & 3u), pick(ct, k2 & 3u));
        if (m >= 2) stack[sp++] = make_int2(pick(lk, k1 & 3u), pick(ct, k1 & 3u));
        cur = pick(lk, k0 & 3u);
        cnt = pick(ct, k0 & 3u);
        continue;
      }
    } else {
      if (COUNT) tests += test_count<KIND, ANY>(bvh.prims, (uint32_t)(~cur), cnt, ray);
      if (test_leaf<KIND, ANY, false>(bvh.prims, bvh.order, (uint32_t)(~cur), cnt, ray, c)) return true;
    }
    if (sp == 0) return false;
    int2 e = stack[--sp];
    cur = e.x;
    cnt = e.y;
  }
}

template <int KIND, bool ANY, bool COUNT, int STACK>
__device__ __forceinline__ bool walk_bvh4(const Bvh4View& bvh, const Ray& ray, Closest& c, uint32_t& visits,
                                          uint32_t& tests, uint32_t* err) {
  return zero_dir(slab_ray(ray.o, ray.d)) ? walk_bvh4_form<KIND, ANY, COUNT, STACK, true>(bvh, ray, c, visits, tests, err)
                         : walk_bvh4_form<KIND, ANY, COUNT, STACK, false>(bvh, ray, c, visits, tests, err);
}

// ---------------------------------------------------------------- 8-wide
// FAST traversal of the compressed 8-wide BVH (layout in bvh8.cu).  A node
// visit decodes and tests its (up to) eight child boxes and keeps the hit
// ones as a bit mask in the ray's visiting order (bit k = slot k ^ oct); the
// walk takes children from the mask lowest bit first, and when it descends
// it pushes the node with its remaining mask (one stack entry per level, at
// most 22 for a tree 64 binary levels deep).
constexpr int kStack8 = 32;

// One child plane: fma(S, F(q), pm), F(q) = 1 + q * 2^-15 built by one byte
// permute from byte k of `word` (the builder decodes with these operations).
__device__ __forceinline__ float q8(uint32_t word, int k, float S, float pm) {
  return __fmaf_rn(S, __uint_as_float(__byte_perm(word, 0x3F800000u, 0x7604u | (k << 4))), pm);
}

template <bool EXACT>
__device__ __forceinline__ uint32_t node8_hits(const float4* nd, const SlabRay& sr, F3 o, float tmin, float tfar,
                                               uint32_t oct) {
  uint32_t r[16];
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "l"(nd));
  asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "l"(nd + 2));
  const float pmx = __uint_as_float(r[0]), pmy = __uint_as_float(r[1]), pmz = __uint_as_float(r[2]);
  const uint32_t hb = r[3];
  const float Sx = __uint_as_float((hb & 0xFFu) << 23), Sy = __uint_as_float((hb & 0xFF00u) << 15),
              Sz = __uint_as_float((hb & 0xFF0000u) << 7);
  const uint32_t valid = hb >> 24;
  uint32_t mask = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int k = i & 3, h = i >> 2;
    const float lx = q8(r[4 + h], k, Sx, pmx), hx = q8(r[6 + h], k, Sx, pmx);
    const float ly = q8(r[8 + h], k, Sy, pmy), hy = q8(r[10 + h], k, Sy, pmy);
    const float lz = q8(r[12 + h], k, Sz, pmz), hz = q8(r[14 + h], k, Sz, pmz);
    float tn;
    const bool hit = slab_box<EXACT>(sr, o, lx, hx, ly, hy, lz, hz, tmin, tfar, tn);
    mask |= (hit && (valid >> i & 1u)) ? 1u << (i ^ oct) : 0u;
  }
  return mask;
}

template <int KIND, bool ANY, bool COUNT, int STACK, bool EXACT>
__device__ __forceinline__ bool walk_bvh8_form(const Bvh8View& bvh, const Ray& ray, Closest& c, uint32_t& visits,
                                               uint32_t& tests, uint32_t* err) {
  const SlabRay sr = slab_ray(ray.o, ray.d);
  float tn;
  const float* rb = bvh.root;
  if (!slab_box<EXACT>(sr, ray.o, rb[0], rb[3], rb[1], rb[4], rb[2], rb[5], ray.tmin, ray.tmax, tn)) return false;
  if (bvh.n_binary == 0) {  // the root is one leaf
    if (COUNT) tests += test_count<KIND, ANY>(bvh.prims, 0u, (int)bvh.n_slots, ray);
    return test_leaf<KIND, ANY, false>(bvh.prims, bvh.order, 0u, (int)bvh.n_slots, ray, c);
  }
  const uint32_t oct = (ray.d.x < 0.f ? 1u : 0u) | (ray.d.y < 0.f ? 2u : 0u) | (ray.d.z < 0.f ? 4u : 0u);
  uint2 stack[STACK];
  int sp = 0;
  uint32_t node = 0;
  if (COUNT) ++visits;
  uint32_t mask = node8_hits<EXACT>(bvh.nodes, sr, ray.o, ray.tmin, ANY ? ray.tmax : c.t, oct);
  // A valid walk takes every child (node or leaf) at most once.
  const uint32_t max_steps = 2u * (bvh.n_binary + bvh.n_slots) + 8u;
  uint32_t steps = 0;
  for (;;) {
    if (mask == 0u) {
      if (sp == 0) return false;
      const uint2 e = stack[--sp];
      node = e.x;
      mask = e.y;
    }
    if (++steps > max_steps) { atomicOr(err, kErrCorrupt); return false; }
    const uint32_t k = (uint32_t)__ffs(mask) - 1u;
    mask &= mask - 1u;
    const int2 lc = __ldg(reinterpret_cast<const int2*>(bvh.nodes + 8 * (size_t)node + 4) + (k ^ oct));
    if (lc.y == 0) {
      if (mask) {
        if (sp >= STACK) { atomicOr(err, kErrStackOverflow); return false; }
        stack[sp++] = make_uint2(node, mask);
      }
      node = (uint32_t)lc.x;
      if (COUNT) ++visits;
      mask = node8_hits<EXACT>(bvh.nodes + 8 * (size_t)node, sr, ray.o, ray.tmin, ANY ? ray.tmax : c.t, oct);
    } else {
      if (COUNT) tests += test_count<KIND, ANY>(bvh.prims, (uint32_t)lc.x, lc.y, ray);
      if (test_leaf<KIND, ANY, false>(bvh.prims, bvh.order, (uint32_t)lc.x, lc.y, ray, c)) return true;
    }
  }
}

template <int KIND, bool ANY, bool COUNT, int STACK>
__device__ __forceinline__ bool walk_bvh8(const Bvh8View& bvh, const Ray& ray, Closest& c, uint32_t& visits,
                                          uint32_t& tests, uint32_t* err) {
  return zero_dir(slab_ray(ray.o, ray.d)) ? walk_bvh8_form<KIND, ANY, COUNT, STACK, true>(bvh, ray, c, visits, tests, err)
                                          : walk_bvh8_form<KIND, ANY, COUNT, STACK, false>(bvh, ray, c, visits, tests, err);
}

// ------------------------------------------------- shared lanes of a warp
// One warp's rays walked by all of its lanes.  Every lane starts with its own
// ray; a round is at most kWalkChunk node steps a lane, then one leaf test
// for the lanes that reached a leaf, then a meeting of the warp: lanes whose
// ray is finished take over the oldest (largest) stacked subtree of lanes
// that still have some, with a copy of the ray.
//
// A ray's result is that of the one-lane walk, whichever lanes walk it and
// when.  An any-hit walk culls by the ray's own interval alone, so no order
// matters.  A closest hit is the smallest (t, id) of the primitives tested, so
// what could differ is which boxes are culled.  Call a hit early when its box
// would be culled with that very hit as the bound: a triangle's t is off by
// about |e1||e2||o - v0| 2^-24 / det, and for a long triangle seen edge-on (det
// is 1e-6 or more) that can be far outside the slab test's widening.  Where no
// hit is early no bound that is itself a hit culls the answer, and every order
// gives it; an early hit is the one-lane walk's answer or not by what was found
// before.  So, once lanes are shared,
//  * pieces carry their place in the one-lane order (as in the KD walk), and a
//    lane's bound comes only from hits that the one-lane walk comes to before:
//    its own, those it got with its piece, and the ray's best one if that is
//    from an earlier piece;
//  * an early hit is no bound and no answer, it is noted (the smallest t a
//    ray), and a ray whose noted t is not behind its answer is walked again by
//    its own lane alone.  A ray's first piece needs no such care: what it has
//    found is what the one-lane walk has found by then.
// Every box that the one-lane walk visits is visited then: what culls it here
// is a hit from before it whose box the one-lane walk visited too, or culled by
// a nearer hit.  So an early hit that the one-lane walk may have taken is noted.
// Boxes have to hold what is below them, as those of every build do; an imported
// tree is checked, and without that its closest hits keep their lanes (alone).
// Long edge-on triangles among ordinary ones: one ray in eight had another hit
// in another batch without this.  It costs 1% on 1M random rays, 2% on 8.3M
// bounce rays, 4% on a median BVH (test beside the vote on hits; inside the
// leaf test 7, 10 and 7%).
//
// Closest hits on spheres stay with their lane: a small distant sphere's t
// cancels, so early hits are common there.
//
// What it is for: with one lane a ray the warp waits for its longest ray
// (8.5 of 32 lanes busy on bounce rays), and a ray is one chain of dependent
// fetches (a launch of few rays lasts as long as its longest chain).  With
// shared lanes 17 of 32 are busy and the walk is bound by L1 wavefronts (85%
// of peak; the one-lane walk 48%).  Testing leaves once a round instead of
// at every step matters as much: a tenth of the visits are leaves, so nearly
// every step of a full warp paid for a leaf test of one or two lanes.
// Measured on a GB300 against the one-lane walk (us): 8.3M bounce rays
// 4371 -> 2590 (in octant order 3332 -> 2673), 1M random rays 620 -> 374
// (any hit 417 -> 319), 2M bounce rays on a median BVH 1421 -> 721, 115k
// scanner rays 250 -> 91, 1k random rays 82 -> 31; coherent rays gain
// nothing: 8.3M camera rays 997 -> 1020, shadow rays 999 -> 1009.
//
// kWalkChunk: 2 / 3 / 4 / 6 / 8 node steps a round give 2915 / 2838 / 2853 /
// 2922 / 3016 us on the ordered bounce rays, and camera rays want 4 or more
// (1181 / 1087 / 1071 / 1065 / 1067).  kWalkIdle(Any): lanes idle before
// subtrees move (a move is some 40 instructions of the whole warp, and a far
// subtree taken early may be one that the nearer hit would have culled):
// closest hit 1 / 8 / 12 / 16 / 24 give 417 / 397 / 387 / 385 / 397 us on the
// random rays and 2853 / 2826 / 2833 / 2875 / 3076 on the bounce rays; any
// hit, where every taken subtree of a ray that is hit is wasted, 452 / 432 /
// 419 / 403 / 374.  Rays kept in shared memory, a sentinel entry instead of
// the two stack bounds and a forced convergence at every step were all
// slower (up to 1.4x).
constexpr int kWalkChunk = 4;
constexpr int kWalkIdle = 12;
constexpr int kWalkIdleAny = 20;
// Blocks of 128 an SM: 4-byte stack entries 8 / 9 / 10: 2920 / 2817 / 2738 us
// (bounce rays in octant order), 8-byte ones 747 / 721 / 798 (2M bounce rays on
// a median BVH; 10 spill).
constexpr int kWalkBlocks = 10, kWalkBlocksWide = 9;

// Stack entries of a closest-hit walk that sit in shared memory, the deeper
// ones in local memory: the lanes' stack heights differ, so a push or pop of
// the warp touches as many lines of local memory as there are heights, but
// one line of banks here.  0 / 8 / 12 entries: 383 / 370 / 368 us on the
// random rays, 2627 / 2547 / 2535 bounce, 745 / 696 / 696 on the median BVH
// (8-byte entries), 1028 / 1042 / 1042 camera.  Any hit keeps its stack local:
// 0 / 8 entries 1009 / 1024 us on the coherent shadow rays, 319 / 311 random.
template <bool ANY>
constexpr int kWalkTop = ANY ? 0 : 12;

template <bool ANY, bool MANY, bool UNIT>
struct WarpShare {
  typename std::conditional<UNIT, int, int2>::type stack[kWalkTop<ANY> ? kWalkTop<ANY> : 1][32];
  uint32_t give[32];           // a meeting's donors, by rank
  const float4* prims[MANY ? 32 : 1];    // MANY: the structure of each ray
  const uint32_t* order[MANY ? 32 : 1];
  unsigned long long key[ANY ? 1 : 32];  // best hit per ray: (order-preserving bits of t + 0, prim)
  float t[ANY ? 1 : 32];
  float2 uv[ANY ? 1 : 32];
  uint32_t place[ANY ? 1 : 32];  // the best hit's place in the one-lane order
  uint32_t doubt[ANY ? 1 : 32];  // smallest t of an early hit, order-preserving bits
  uint32_t piece[ANY || MANY ? 1 : 32];  // what a lane walks: places lo .. lo + 2^k - 1 of its ray's order, as lo << 5 | k
};
constexpr uint32_t kWholeRay = 27u;  // a piece's size in places is halved at each give; lo has 27 bits

__device__ __forceinline__ float from_order_key(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}
__device__ __forceinline__ unsigned long long hit_key(const Closest& c) {
  return ((unsigned long long)order_key(__fadd_rn(c.t, 0.f)) << 32) | c.prim;  // -0 and +0 tie
}

// slab_box<false> with each axis' two plane distances from one packed
// multiply-add (camera rays 1073 -> 1034 us, bounce rays 2769 -> 2738).
__device__ __forceinline__ void plane_pair(float lo, float hi, float inv, float noi, float& t0, float& t1) {
  asm("{\n\t.reg .b64 p, i, n, r;\n\t"
      "mov.b64 p, {%2, %3};\n\tmov.b64 i, {%4, %4};\n\tmov.b64 n, {%5, %5};\n\t"
      "fma.rn.f32x2 r, p, i, n;\n\tmov.b64 {%0, %1}, r;\n\t}"
      : "=f"(t0), "=f"(t1)
      : "f"(lo), "f"(hi), "f"(inv), "f"(noi));
}
__device__ __forceinline__ bool slab_pairs(const SlabRay& r, float lx, float hx, float ly, float hy, float lz, float hz,
                                           float tmin, float tfar, float& tnear) {
  float tx0, tx1, ty0, ty1, tz0, tz1;
  plane_pair(lx, hx, r.inv.x, r.noi.x, tx0, tx1);
  plane_pair(ly, hy, r.inv.y, r.noi.y, ty0, ty1);
  plane_pair(lz, hz, r.inv.z, r.noi.z, tz0, tz1);
  tnear = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fmaxf(fminf(tz0, tz1), tmin));
  const float tf = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fminf(fmaxf(tz0, tz1), tfar));
  return tnear <= __fmaf_rn(tf, kWiden, r.eps);
}

// Whether a triangle's hit at t is early: its box, entered with the hit as the
// bound, may fail the slab test.  The box is the triangle's own from its
// payload (v0, v1 - v0, v2 - v0), each entry plane moved inwards by more than
// what the two roundings of a vertex can have moved it; any larger box is
// entered no later, and its exit has passed the test already.  A NaN is early.
__device__ __forceinline__ bool early_hit(const float4* __restrict__ tri, const SlabRay& r, float tmin, float t) {
  const float4 v = __ldg(tri), e1 = __ldg(tri + 1), e2 = __ldg(tri + 2);
  const float far = __fmaf_rn(t, kWiden, r.eps);
  auto entered = [&](float p0, float d1, float d2, float inv, float noi) {
    const float p1 = __fadd_rn(p0, d1), p2 = __fadd_rn(p0, d2);
    const float p = inv > 0.f ? fminf(fminf(p0, p1), p2) : fmaxf(fmaxf(p0, p1), p2);
    const float pad = __fmul_rn(__fadd_rn(fabsf(p), fmaxf(fabsf(d1), fabsf(d2))), 0x3p-24f);
    return __fmaf_rn(__fadd_rn(p, inv > 0.f ? pad : -pad), inv, noi) <= far;
  };
  return !(tmin <= far && entered(v.x, e1.x, e2.x, r.inv.x, r.noi.x) && entered(v.y, e1.y, e2.y, r.inv.y, r.noi.y) &&
           entered(v.z, e1.z, e2.z, r.inv.z, r.noi.z));
}

// The warp's 32 lanes call it together, each with its ray (walk: it has one,
// and not one for the exact box test).  c starts as the ray's (tmax, miss)
// and returns its closest hit; any hit returns whether the lane's ray is
// occluded, closest hit whether it is in doubt: the caller walks it again with
// alone, where no lane takes over another's work.  eager: lanes start without a
// ray (fewer than 32 rays), so subtrees move as soon as a lane is idle.  MANY:
// the lanes' rays may belong to different structures (bvh is the lane's own).
// KEEP: a lane's piece is in a register, not in shared memory: 1-3% faster where
// registers do not bound the kernel, 1-2% slower where they do (k_trace_warps).
template <int KIND, bool ANY, bool UNIT, int STACK, bool MANY, bool KEEP>
__device__ __forceinline__ bool walk_warp(const Bvh2View& bvh, Ray ray, SlabRay sr, bool walk, bool eager, bool alone,
                                          Closest& c, WarpShare<ANY, MANY, UNIT>& sh, uint32_t* err) {
  constexpr bool kShare = ANY || KIND == kTriangles;
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  using Entry = typename std::conditional<UNIT, int, int2>::type;
  constexpr int kTop = kWalkTop<ANY>;
  Entry deep[STACK];
  auto get = [&](int i) -> Entry {
    if constexpr (kTop > 0)
      if (i < kTop) return sh.stack[i][lane];
    return deep[i];
  };
  int sp = 0, bot = 0;  // entries [bot, sp): lanes that take over work take the entry at bot
  int cur = bvh.n_internal ? 0 : -1;
  int cnt = bvh.n_internal ? 0 : (int)bvh.n_slots;
  const float4* nodes = bvh.nodes;
  uint32_t home = lane;  // the lane whose ray this lane works on
  uint32_t found = 0;    // any hit: the rays that are done (one bit each)
  bool shared = false;   // some lane has taken over another's subtree (warp-uniform)
  // A ray's walk visits every node and leaf at most once, and a lane that
  // takes over a subtree continues its donor's walk: whatever lane is busy at
  // a meeting, at least one node or leaf of its ray lies behind it for every
  // meeting so far.
  uint32_t meetings = 2u * (bvh.n_internal + bvh.n_slots) + 8u;  // that are left
  uint32_t piece_reg = kWholeRay;  // KEEP: sh.piece of this lane
  auto piece = [&]() -> uint32_t& {
    if constexpr (KEEP) return piece_reg;
    else return sh.piece[lane];
  };
  if constexpr (!ANY && kShare) piece() = kWholeRay;
  if (MANY) {
    meetings = __reduce_max_sync(0xffffffffu, walk ? meetings : 0u);
    sh.prims[MANY ? lane : 0] = bvh.prims;
    sh.order[MANY ? lane : 0] = bvh.order;
    __syncwarp();
  }
  if (walk) {
    float tn;
    const float* rb = bvh.root;
    walk = slab_box<false>(sr, ray.o, rb[0], rb[3], rb[1], rb[4], rb[2], rb[5], ray.tmin, ray.tmax, tn);
  }
  auto pop = [&]() {
    if (sp == bot) {
      walk = false;
    } else if constexpr (UNIT) {
      cur = get(--sp);
    } else {
      const int2 e = get(--sp);
      cur = e.x;
      cnt = e.y;
    }
  };
  for (;;) {
#pragma unroll 1
    for (int k = 0; k < kWalkChunk && walk && cur >= 0; ++k) {
      float4 a, b, z;
      int4 l;
      load_node(nodes + 4 * (size_t)cur, a, b, z, l);
      const float tfar = ANY ? ray.tmax : c.t;
      float tl, tr;
      const bool hl = slab_pairs(sr, a.x, a.y, a.z, a.w, z.x, z.y, ray.tmin, tfar, tl);
      const bool hr = slab_pairs(sr, b.x, b.y, b.z, b.w, z.z, z.w, ray.tmin, tfar, tr);
      if (hl || hr) {
        const bool left = hl && !(hr && tr < tl);
        cur = left ? l.x : l.y;
        if (!UNIT) cnt = left ? l.z : l.w;
        if (hl && hr) {
          Entry e;
          if constexpr (UNIT) e = left ? l.y : l.x;
          else e = left ? make_int2(l.y, l.w) : make_int2(l.x, l.z);
          if (kTop > 0 && sp < kTop) {
            sh.stack[sp][lane] = e;
          } else if (sp < STACK) {
            deep[sp] = e;
          } else {
            atomicOr(err, kErrStackOverflow);
            walk = false;
            break;
          }
          ++sp;
        }
      } else {
        pop();
      }
    }
    bool hit = false;  // any hit: the ray is occluded; closest hit: c is a new one
    const uint32_t had = c.prim;  // a leaf is tested once: a new hit is another primitive
    const float had_t = c.t;
    const int leaf = cur;
    if (walk && cur < 0) {
      if (UNIT) cnt = 1;
      hit = test_leaf<KIND, ANY, false>(MANY ? sh.prims[MANY ? home : 0] : bvh.prims,
                                        MANY ? sh.order[MANY ? home : 0] : bvh.order, (uint32_t)(~cur), cnt, ray, c);
      if (!ANY) hit = c.prim != had;
      pop();
    }
    __syncwarp();
    if (__any_sync(0xffffffffu, hit)) {
      if constexpr (ANY) {
        found |= __reduce_or_sync(0xffffffffu, hit ? 1u << home : 0u);
        if ((found >> home) & 1u) walk = false;
      } else if (shared) {
        if (hit && piece() >= 32u) {  // not the ray's first piece
          const float4* tri = (MANY ? sh.prims[MANY ? home : 0] : bvh.prims) + 3 * (size_t)(uint32_t)(~leaf);
          if (!UNIT)
            while (__float_as_uint(__ldg(&tri->w)) != c.prim) tri += 3;  // the hit is one of this leaf's
          if (early_hit(tri, sr, ray.tmin, c.t)) {
            atomicMin(&sh.doubt[home], order_key(__fadd_rn(c.t, 0.f)));
            c.t = had_t;
            c.prim = had;
            hit = false;
          }
        }
        const unsigned long long mine = hit_key(c);
        if (hit) atomicMin(&sh.key[home], mine);
        __syncwarp();
        const unsigned long long best = sh.key[home];
        if (hit && best == mine) {  // equal keys: the same primitive, so the same t, u, v
          sh.t[home] = c.t;
          sh.uv[home] = make_float2(c.u, c.v);
          sh.place[home] = piece() >> 5;
        }
        __syncwarp();
        if (sh.place[home] <= piece() >> 5) {
          c.t = from_order_key((uint32_t)(best >> 32));
          c.prim = (uint32_t)best;
        }
      }
    }
    const uint32_t busy = __ballot_sync(0xffffffffu, walk);
    if (busy == 0u) break;
    if (meetings-- == 0u) {
      if (lane == 0) atomicOr(err, kErrCorrupt);
      break;
    }
    if (!kShare || (!ANY && alone) || 32 - __popc(busy) < (eager ? 1 : ANY ? kWalkIdleAny : kWalkIdle)) continue;
    const bool can = walk && sp > bot && (ANY || !kShare || (piece() & 31u));
    const uint32_t donors = __ballot_sync(0xffffffffu, can);
    if (donors == 0u) continue;
    if constexpr (!ANY) {
      if (!shared) {  // every lane still holds its own ray
        sh.key[lane] = hit_key(c);
        sh.t[lane] = c.t;
        sh.uv[lane] = make_float2(c.u, c.v);
        sh.place[lane] = 0u;
        sh.doubt[lane] = 0xFFFFFFFFu;
      }
    }
    shared = true;
    const int pairs = min(__popc(donors), 32 - __popc(busy));
    const int rank = __popc((walk ? donors : ~busy) & below);
    int give = 0, give_cnt = 0;
    if (can && rank < pairs) {
      if constexpr (!ANY) --piece();  // the lower half stays here
      if constexpr (UNIT) {
        give = get(bot++);
      } else {
        const int2 e = get(bot++);
        give = e.x;
        give_cnt = e.y;
      }
      sh.give[rank] = lane;
    }
    __syncwarp();
    const bool take = !walk && rank < pairs;
    const int src = take ? (int)sh.give[rank] : (int)lane;
    auto from = [&](float& x) { x = __shfl_sync(0xffffffffu, x, src); };
    from(ray.o.x); from(ray.o.y); from(ray.o.z);
    from(ray.d.x); from(ray.d.y); from(ray.d.z);
    from(ray.tmin);
    from(sr.inv.x); from(sr.inv.y); from(sr.inv.z);
    from(sr.noi.x); from(sr.noi.y); from(sr.noi.z);
    from(sr.eps);
    home = __shfl_sync(0xffffffffu, home, src);
    if (ANY) {
      from(ray.tmax);
    } else {
      from(c.t);
      c.prim = __shfl_sync(0xffffffffu, c.prim, src);
    }
    if (MANY)
      nodes = reinterpret_cast<const float4*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(nodes), src));
    give = __shfl_sync(0xffffffffu, give, src);
    uint32_t half = 0;
    if constexpr (!ANY) half = KEEP ? __shfl_sync(0xffffffffu, piece_reg, src) : sh.piece[src];
    if (!UNIT) give_cnt = __shfl_sync(0xffffffffu, give_cnt, src);
    if (take) {
      if constexpr (!ANY) piece() = half + (32u << (half & 31u));  // the upper half of what the donor had
      walk = true;
      cur = give;
      cnt = give_cnt;
      sp = bot = 0;
    }
    __syncwarp();
  }
  if constexpr (!ANY) {
    if (shared) {
      __syncwarp();  // the last round's stores; a ballot does not order memory
      const float2 uv = sh.uv[lane];
      const unsigned long long best = sh.key[lane];
      const uint32_t doubt = sh.doubt[lane];
      c = {sh.t[lane], (uint32_t)best, uv.x, uv.y};
      found = doubt != 0xFFFFFFFFu && doubt <= (uint32_t)(best >> 32) ? 1u << lane : 0u;
      __syncwarp();
    }
  }
  return (found >> lane) & 1u;
}

}  // namespace rq
