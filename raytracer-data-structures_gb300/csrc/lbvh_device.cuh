// Device helpers shared by the single-scene LBVH kernels (morton.cu,
// lbvh.cu) and the batched ones (batch.cu), so that a batched build performs
// exactly the operations of a single build.
#pragma once
#include "rq_device.cuh"
#include "rq_internal.hpp"

namespace rq {

// Scene box from the ordered-int accumulators: lo and extent per axis.
__device__ __forceinline__ void bounds_from(const int32_t* lohi, float* lo, float* ext) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    lo[k] = ordered_to_float(lohi[k]);
    float hi = ordered_to_float(lohi[3 + k]);
    ext[k] = __fsub_rn(hi, lo[k]);
  }
}

// Cube normalisation (RQ_MORTON_SCENE_CUBE): every axis scaled by the
// largest extent of the scene box, so the curve splits space evenly on flat
// or elongated scenes.
__device__ __forceinline__ void cube_extent(float* ext) {
  const float e = fmaxf(fmaxf(ext[0], ext[1]), ext[2]);
  ext[0] = ext[1] = ext[2] = e;
}

// (c - lo) / ext per axis, 0 where the extent is 0.
__device__ __forceinline__ uint32_t code_scene(F3 c, const float* lo, const float* ext) {
  float q0 = ext[0] > 0.f ? __fdiv_rn(__fsub_rn(c.x, lo[0]), ext[0]) : 0.f;
  float q1 = ext[1] > 0.f ? __fdiv_rn(__fsub_rn(c.y, lo[1]), ext[1]) : 0.f;
  float q2 = ext[2] > 0.f ? __fdiv_rn(__fsub_rn(c.z, lo[2]), ext[2]) : 0.f;
  return morton3d(q0, q1, q2);
}

// Triangle centroid ((v0 + v1) + v2) / 3 per axis, from the packed copies (one 16-byte load per triangle and per
// vertex instead of twelve scattered 4-byte loads).
__device__ __forceinline__ F3 tri_centroid(const float4* __restrict__ verts4, const uint4* __restrict__ idx4,
                                           uint32_t i) {
  const uint4 t = __ldg(idx4 + i);
  const float4 a = __ldg(verts4 + t.x), b = __ldg(verts4 + t.y), c = __ldg(verts4 + t.z);
  F3 cen;
  cen.x = __fdiv_rn(__fadd_rn(__fadd_rn(a.x, b.x), c.x), 3.0f);
  cen.y = __fdiv_rn(__fadd_rn(__fadd_rn(a.y, b.y), c.y), 3.0f);
  cen.z = __fdiv_rn(__fadd_rn(__fadd_rn(a.z, b.z), c.z), 3.0f);
  return cen;
}

// Treelets of an LBVH: the maximal subtrees of at most kTreeletSpan leaves
// (each a contiguous slot range); the nodes above them are the top nodes
// (about 2n / kTreeletSpan), of which kRefitTopCap are listed.
constexpr uint32_t kTreeletSpan = 2048;
constexpr uint32_t kRefitTopCap = 2048;
constexpr uint32_t kTopMark = 0x80000000u;
constexpr uint32_t kSlotMask = 0x7FFFFFFFu;
constexpr uint32_t kTreeletRight = 0x80000000u;  // treelet record: the subtree is a right child

// Atomic exchange with acquire-release semantics at device scope: the
// thread's earlier stores are visible to a thread whose own exchange returns
// this value, and that thread's later loads see them.
__device__ __forceinline__ uint32_t atomic_exch_acq_rel(uint32_t* p, uint32_t v) {
  uint32_t old;
  asm volatile("atom.acq_rel.gpu.global.exch.b32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
  return old;
}

struct Box6 {
  float lo[3], hi[3];
};

// Payload of triangle p in slot `slot` (3 float4: (v0, id), (v1 - v0, 0),
// (v2 - v0, 0)) and its box.
__device__ __forceinline__ Box6 emit_tri(F3 a, F3 c1, F3 c2, uint32_t p, float4* __restrict__ prims,
                                         uint32_t slot) {
  Box6 b;
  F3 e1 = sub_rn(c1, a), e2 = sub_rn(c2, a);
  float4* q = prims + 3 * (size_t)slot;
  q[0] = make_float4(a.x, a.y, a.z, __uint_as_float(p));
  q[1] = make_float4(e1.x, e1.y, e1.z, 0.f);
  q[2] = make_float4(e2.x, e2.y, e2.z, 0.f);
  b.lo[0] = fminf(fminf(a.x, c1.x), c2.x); b.hi[0] = fmaxf(fmaxf(a.x, c1.x), c2.x);
  b.lo[1] = fminf(fminf(a.y, c1.y), c2.y); b.hi[1] = fmaxf(fmaxf(a.y, c1.y), c2.y);
  b.lo[2] = fminf(fminf(a.z, c1.z), c2.z); b.hi[2] = fmaxf(fmaxf(a.z, c1.z), c2.z);
  return b;
}

// Sphere p into slot `slot` (1 float4) and its box: centre -/+ radius
// (main.cpp:686-688).
__device__ __forceinline__ Box6 emit_sphere(const float4* __restrict__ sph, uint32_t p, float4* __restrict__ prims,
                                            uint32_t slot) {
  Box6 b;
  float4 s = __ldg(sph + p);
  prims[slot] = s;
  b.lo[0] = __fsub_rn(s.x, s.w); b.lo[1] = __fsub_rn(s.y, s.w); b.lo[2] = __fsub_rn(s.z, s.w);
  b.hi[0] = __fadd_rn(s.x, s.w); b.hi[1] = __fadd_rn(s.y, s.w); b.hi[2] = __fadd_rn(s.z, s.w);
  return b;
}

// Gather primitive `p` into payload slot `slot` and return its box.
__device__ __forceinline__ Box6 emit_prim(int kind, const float* __restrict__ verts,
                                          const uint32_t* __restrict__ idx,
                                          const float4* __restrict__ sph, uint32_t p,
                                          float4* __restrict__ prims, uint32_t slot) {
  if (kind != kTriangles) return emit_sphere(sph, p, prims, slot);
  uint32_t i0 = __ldg(idx + 3 * (size_t)p), i1 = __ldg(idx + 3 * (size_t)p + 1), i2 = __ldg(idx + 3 * (size_t)p + 2);
  F3 a = {__ldg(verts + 3 * (size_t)i0), __ldg(verts + 3 * (size_t)i0 + 1), __ldg(verts + 3 * (size_t)i0 + 2)};
  F3 c1 = {__ldg(verts + 3 * (size_t)i1), __ldg(verts + 3 * (size_t)i1 + 1), __ldg(verts + 3 * (size_t)i1 + 2)};
  F3 c2 = {__ldg(verts + 3 * (size_t)i2), __ldg(verts + 3 * (size_t)i2 + 1), __ldg(verts + 3 * (size_t)i2 + 2)};
  return emit_tri(a, c1, c2, p, prims, slot);
}

}  // namespace rq
