// LBVH topology, payload and boxes.
//
// The reference cites Karras' construction (accelerators.h:371,568) but its
// findSplit (accelerators.h:397-449) is discarded and no refit exists.  The
// tree here is Karras' radix tree over the sorted codes (2012, "Maximizing
// Parallelism in the Construction of BVHs, Octrees, and k-d Trees"; ties
// broken by the index), in his numbering: a left child's index is its last
// leaf, a right child's its first, the root's 0.  It is built from the leaves
// up (Apetrei 2014, "Fast and Simple Agglomerative LBVH Construction"): a
// subtree over the leaves l .. r joins the neighbour with which it shares the
// longer prefix, so its parent's split is r | r + 1 or l - 1 | l, and the
// second of two siblings to arrive at their split makes the node.  Topology
// and boxes come out of one pass, with no searches and no parent links.
//
// BVH2 node (64 B, 4 x float4):
//   [0] left  child box (lo.x, hi.x, lo.y, hi.y)
//   [1] right child box (lo.x, hi.x, lo.y, hi.y)
//   [2] (left lo.z, left hi.z, right lo.z, right hi.z)
//   [3] int (left, right, left count, right count); child >= 0 internal,
//       child < 0 leaf holding slots [~child, ~child + count)
#include "lbvh_device.cuh"
#include "rq_build.hpp"

namespace rq {
namespace {

constexpr int kThreads = 256;

// Triangle p's payload (3 float4: (v0, id), (v1 - v0, 0), (v2 - v0, 0)) in
// q and its box, from the packed copies.
__device__ __forceinline__ Box6 tri_payload(const float4* __restrict__ verts4, const uint4* __restrict__ idx4,
                                            uint32_t p, float4 q[3]) {
  const uint4 t = __ldg(idx4 + p);
  const float4 a = __ldg(verts4 + t.x), c1 = __ldg(verts4 + t.y), c2 = __ldg(verts4 + t.z);
  const F3 e1 = sub_rn({c1.x, c1.y, c1.z}, {a.x, a.y, a.z}), e2 = sub_rn({c2.x, c2.y, c2.z}, {a.x, a.y, a.z});
  q[0] = make_float4(a.x, a.y, a.z, __uint_as_float(p));
  q[1] = make_float4(e1.x, e1.y, e1.z, 0.f);
  q[2] = make_float4(e2.x, e2.y, e2.z, 0.f);
  Box6 b;
  b.lo[0] = fminf(fminf(a.x, c1.x), c2.x); b.hi[0] = fmaxf(fmaxf(a.x, c1.x), c2.x);
  b.lo[1] = fminf(fminf(a.y, c1.y), c2.y); b.hi[1] = fmaxf(fmaxf(a.y, c1.y), c2.y);
  b.lo[2] = fminf(fminf(a.z, c1.z), c2.z); b.hi[2] = fmaxf(fmaxf(a.z, c1.z), c2.z);
  return b;
}

// The warp's payloads (lane l: slot base + l, for l < nvalid) stored as 96
// consecutive float4s: store k writes float4s 32k .. 32k + 31, each lane one
// (slot m / 3, part m % 3, fetched from its lane), so every store is one
// contiguous 512-byte run.  All 32 lanes take part.
__device__ __forceinline__ void store_payload_warp(float4* __restrict__ out, int nvalid, uint32_t lane,
                                                   const float4 q[3]) {
  for (int k = 0; k < 3; ++k) {
    const int m = 32 * k + (int)lane, src = m / 3, part = m - 3 * src;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int c = 0; c < 3; ++c) {  // every lane shuffles every part and keeps its own
      const float x = __shfl_sync(0xffffffffu, q[c].x, src), y = __shfl_sync(0xffffffffu, q[c].y, src);
      const float z = __shfl_sync(0xffffffffu, q[c].z, src), w = __shfl_sync(0xffffffffu, q[c].w, src);
      if (part == c) v = make_float4(x, y, z, w);
    }
    if (src < nvalid) out[m] = v;
  }
}

// The tree over a window of kTreeWindow leaves is made in shared memory, one
// block a window and one thread a leaf; the subtrees left over (those whose
// parent reaches into another window: at most one on each step of the paths
// from the root to the two leaves at a boundary, so at most 2 x 64 a window)
// climb on with device-scope arrivals, one thread each.
//
// Bound by latency: the leaf's three dependent gathers, about ten shared
// steps, then about log2(windows) device-scope exchanges of a microsecond;
// whole rebuilds of 36k spheres, 125k, 998k and 2.7M triangles took 124, 144,
// 265 and 518 us with one search a node, parent links and a second kernel for
// the boxes, and take 79, 91, 191 and 348 us.  Windows of 1024 leaves: 87,
// 92, 201, 367 us; 512: 83, 93, 198, 358; 128: 79, 90, 190, 342, with twice
// the records.
constexpr uint32_t kTreeBlocks = 6;  // an SM; 5 and 8 blocks: within 3%
static_assert(kTreeWindow >= kTreeMaxLeft, "one thread a subtree left over");
static_assert(kTreeWindow <= kTreeletSpan, "a top node is made by the slow climb");
static_assert(kTreeWindow < (1u << 16), "a far end and a height share a word");

struct TreeShared {
  float box[6][kTreeWindow];        // a finished subtree's box, at its index (its last leaf as a left child, else its first)
  uint32_t arrived[kTreeWindow];    // split w | w + 1: 0, or the one child here: (far end + 1) | height << 16 | left << 31
  int8_t delta[kTreeWindow + 1];    // prefix shared by leaves w - 1 and w; -1 at the ends of a scene
  uint32_t left_lr[kTreeMaxLeft];   // the subtrees left over: first leaf | last leaf << 16
  uint8_t left_h[kTreeMaxLeft];     // their heights
  uint32_t n_left;
};

// The node over leaves l .. r split after g (scene-local slots): links and
// both child boxes, two 32-byte stores.
__device__ __forceinline__ void store_node(float4* node, uint32_t l, uint32_t g, uint32_t r, const Box6& L,
                                           const Box6& R) {
  const int lc = g == l ? ~(int)g : (int)g, rc = g + 1 == r ? ~(int)(g + 1) : (int)(g + 1);
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(node), "f"(L.lo[0]), "f"(L.hi[0]),
               "f"(L.lo[1]), "f"(L.hi[1]), "f"(R.lo[0]), "f"(R.hi[0]), "f"(R.lo[1]), "f"(R.hi[1])
               : "memory");
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(node + 2), "r"(__float_as_int(L.lo[2])),
               "r"(__float_as_int(L.hi[2])), "r"(__float_as_int(R.lo[2])), "r"(__float_as_int(R.hi[2])), "r"(lc), "r"(rc),
               "r"(lc < 0 ? 1 : 0), "r"(rc < 0 ? 1 : 0)
               : "memory");
}

__device__ __forceinline__ Box6 join(const Box6& L, const Box6& R) {
  Box6 b;
  for (int k = 0; k < 3; ++k) { b.lo[k] = fminf(L.lo[k], R.lo[k]); b.hi[k] = fmaxf(L.hi[k], R.hi[k]); }
  return b;
}

__device__ __forceinline__ void store_root(float* root, const Box6& b) {
  for (int k = 0; k < 3; ++k) { root[k] = b.lo[k]; root[3 + k] = b.hi[k]; }
}

// What the treelet pass needs of node i over leaves l .. r split after g: a
// node of more than kTreeletSpan leaves is a top node (mark[i] = kTopMark |
// slot, top[slot] = i for slots below kRefitTopCap, count[0] = their number,
// possibly above the cap; its children get their parent words) and lists its
// children of at most kTreeletSpan leaves as treelets ({first slot, leaf
// count | kTreeletRight for a right child}, count[1] = their number); a root
// of at most kTreeletSpan leaves is the one treelet.
__device__ __forceinline__ void list_node(const TreeArgs& a, uint32_t i, uint32_t l, uint32_t g, uint32_t r, bool root) {
  uint2* tl = reinterpret_cast<uint2*>(a.top.treelets);
  if (r - l + 1 <= kTreeletSpan) {
    if (root) tl[atomicAdd(a.top.count + 1, 1u)] = make_uint2(0u, (r - l + 1) | kTreeletRight);
    return;
  }
  const uint32_t slot = atomicAdd(a.top.count, 1u);
  if (slot < kRefitTopCap) a.top.top[slot] = i;
  a.top.mark[i] = kTopMark | (slot & kSlotMask);
  const uint32_t ls = g - l + 1, rs = r - g;
  if (ls > 1) a.parent[g] = i << 1;
  if (rs > 1) a.parent[g + 1] = i << 1 | 1u;
  if (ls <= kTreeletSpan) {
    if (ls > 1) a.top.mark[g] = 0u;
    tl[atomicAdd(a.top.count + 1, 1u)] = make_uint2(l, ls);
  }
  if (rs <= kTreeletSpan) {
    if (rs > 1) a.top.mark[g + 1] = 0u;
    tl[atomicAdd(a.top.count + 1, 1u)] = make_uint2(g + 1, rs | kTreeletRight);
  }
}

// MANY: the slots of several scenes back to back (poff), each with its own
// codes, nodes, root and indices, sorted by (scene << 30) | code; otherwise
// one scene.  LIST: also what the treelet pass reads (node heights, top nodes,
// treelets).
template <bool MANY, bool LIST>
__global__ void __launch_bounds__(kTreeWindow, kTreeBlocks) k_tree(TreeArgs a) {
  __shared__ TreeShared sh;
  constexpr uint32_t kCodeMask = (1u << 30) - 1u;
  const uint32_t base = blockIdx.x * kTreeWindow;
  const uint32_t cnt = min(kTreeWindow, a.n - base);
  const uint32_t w = threadIdx.x, lane = w & 31u, g0 = base + w;
  const bool live = w < cnt;
  // Scene of slot g (its number and first slot) and the prefix length of the
  // leaves g - 1 and g.
  auto scene_of = [&](uint32_t g, uint32_t& s, uint32_t& p0) {
    s = p0 = 0u;
    if constexpr (MANY) {
      s = (uint32_t)(__ldg(a.keys + g) >> 30);
      if (s >= a.n_scenes || g < __ldg(a.poff + s) || g >= __ldg(a.poff + s + 1)) {
        atomicOr(a.err, kErrCorrupt);  // the sort keeps scenes contiguous
        s = segment_of(a.poff, a.n_scenes, g);
      }
      p0 = __ldg(a.poff + s);
    }
  };
  auto code_of = [&](uint32_t g) { return MANY ? (uint32_t)__ldg(a.keys + g) & kCodeMask : __ldg(a.codes + g); };
  auto delta_at = [&](uint32_t g, uint32_t p0) {
    if (g == p0 || g >= a.n) return -1;
    const uint32_t x = code_of(g - 1), y = code_of(g), i = g - 1 - p0;
    return x != y ? __clz(x ^ y) : 32 + __clz(i ^ (i + 1u));
  };
  auto leave = [&](uint32_t l, uint32_t r, uint32_t h) {
    const uint32_t at = atomicAdd(&sh.n_left, 1u);
    if (at >= kTreeMaxLeft) { atomicOr(a.err, kErrCorrupt); return; }
    sh.left_lr[at] = l | r << 16;
    sh.left_h[at] = (uint8_t)h;
  };
  if (w == 0) {
    sh.n_left = 0u;
    uint32_t s = 0u, p0 = 0u;
    if (base + cnt < a.n) scene_of(base + cnt, s, p0);
    sh.delta[cnt] = (int8_t)delta_at(base + cnt, p0);
  }
  uint32_t s = 0u, p0 = 0u;
  Box6 b = {};
  float4 q[3] = {};
  if (live) {
    scene_of(g0, s, p0);
    uint32_t p;
    if constexpr (MANY) {
      p = __ldg(a.vals + g0) - p0;
      if (p >= __ldg(a.poff + s + 1) - p0) {
        atomicOr(a.err, kErrCorrupt);
        p = 0u;
      }
      a.codes_out[g0] = code_of(g0);
      a.order_out[g0] = p;
    } else {
      p = __ldg(a.order + g0);
    }
    sh.arrived[w] = 0u;
    sh.delta[w] = (int8_t)delta_at(g0, p0);
    if (a.kind == kTriangles)
      b = tri_payload(MANY ? a.desc[s].verts4 : a.verts, MANY ? a.desc[s].idx4 : a.idx, p, q);
    else
      b = emit_sphere(MANY ? a.desc[s].sph : a.sph, p, a.prims, g0);
  }
  if (a.kind == kTriangles) {  // warp-wide stores
    const int nvalid = (int)cnt - (int)(w - lane);
    if (nvalid > 0) store_payload_warp(a.prims + 3 * (size_t)(g0 - lane), nvalid < 32 ? nvalid : 32, lane, q);
  }
  __syncthreads();
  if (live) {
    float4* const nodes = a.nodes + 4 * (size_t)(p0 - s);  // scene s's nodes start at its first slot - s
    const uint32_t off = base - p0;                        // window slot -> scene slot (modulo 2^32)
    uint32_t l = w, r = w, h = 0;
    for (int step = 0;; ++step) {
      if (step >= 128) { atomicOr(a.err, kErrCorrupt); break; }  // the tree is at most 64 deep
      const int dl = sh.delta[l], dr = sh.delta[r + 1];
      if ((dl & dr) < 0) {  // the whole scene
        store_root(a.roots + 8 * (size_t)s, b);
        break;
      }
      const bool left = dr > dl;  // a left child: the parent's split is r | r + 1
      if (left ? r + 1 == cnt : l == 0) {
        leave(l, r, h);
        for (int c = 0; c < 3; ++c) { sh.box[c][left ? r : l] = b.lo[c]; sh.box[3 + c][left ? r : l] = b.hi[c]; }
        break;
      }
      const uint32_t g = left ? r : l - 1, mine = left ? r : l, other = left ? r + 1 : l - 1;
      for (int c = 0; c < 3; ++c) { sh.box[c][mine] = b.lo[c]; sh.box[3 + c][mine] = b.hi[c]; }
      __threadfence_block();
      const uint32_t old = atomicExch(&sh.arrived[g], ((left ? l : r) + 1u) | h << 16 | (left ? 1u << 31 : 0u));
      if (old == 0u) break;  // the sibling's thread makes the node
      __threadfence_block();
      sh.arrived[g] = 0u;
      Box6 o;
      for (int c = 0; c < 3; ++c) { o.lo[c] = sh.box[c][other]; o.hi[c] = sh.box[3 + c][other]; }
      const uint32_t far = (old & 0xFFFFu) - 1u;
      if (left) r = far; else l = far;
      if (l > r || r >= cnt) { atomicOr(a.err, kErrCorrupt); break; }
      h = 1u + max(h, (old >> 16) & 0x7FFFu);
      const int nl = sh.delta[l], nr = sh.delta[r + 1];
      const uint32_t i = (nl & nr) < 0 ? 0u : (nr > nl ? r : l) + off;
      store_node(nodes + 4 * (size_t)i, l + off, g + off, r + off, left ? b : o, left ? o : b);
      b = left ? join(b, o) : join(o, b);
      if constexpr (LIST) {
        a.heights[i] = (uint8_t)min(h, 255u);
        if ((nl & nr) < 0) list_node(a, 0u, l, g, r, true);
      }
    }
  }
  __syncthreads();
  // A child whose sibling reaches into another window is left over too.
  if (live) {
    const uint32_t v = sh.arrived[w], far = (v & 0xFFFFu) - 1u;
    if (v) leave(v >> 31 ? far : w + 1u, v >> 31 ? w : far, (v >> 16) & 0x7FFFu);
  }
  __syncthreads();
  if (w >= min(sh.n_left, kTreeMaxLeft)) return;
  // The subtrees left over, over scene slots; their boxes go to the sibling's
  // thread in records of this window.
  const uint32_t wl = sh.left_lr[w] & 0xFFFFu, wr = sh.left_lr[w] >> 16;
  scene_of(base + wl, s, p0);
  const uint32_t count = (MANY ? __ldg(a.poff + s + 1) : a.n) - p0;
  float4* const nodes = a.nodes + 4 * (size_t)(p0 - s);
  uint32_t l = base + wl - p0, r = base + wr - p0, h = sh.left_h[w];
  int dl = sh.delta[wl], dr = sh.delta[wr + 1];
  const uint32_t at = dr > dl ? wr : wl;
  for (int c = 0; c < 3; ++c) { b.lo[c] = sh.box[c][at]; b.hi[c] = sh.box[3 + c][at]; }
  const uint32_t rec = blockIdx.x * kTreeMaxLeft + w;
  for (int step = 0;; ++step) {
    if (step >= 128) { atomicOr(a.err, kErrCorrupt); break; }
    const bool left = dr > dl;
    const uint32_t g = left ? r : l - 1;
    if (left ? r + 1 >= count : l == 0) { atomicOr(a.err, kErrCorrupt); break; }
    a.pool[2 * (size_t)rec] = make_float4(b.lo[0], b.lo[1], b.lo[2], __uint_as_float(left ? l : r));
    a.pool[2 * (size_t)rec + 1] =
        make_float4(b.hi[0], b.hi[1], b.hi[2], __uint_as_float((uint32_t)((left ? dl : dr) + 1) | h << 8));
    const uint32_t old = atomic_exch_acq_rel(a.flags + p0 + g, rec + 1u);
    if (old == 0u) break;
    const float4 x = __ldcg(a.pool + 2 * (size_t)(old - 1u)), y = __ldcg(a.pool + 2 * (size_t)(old - 1u) + 1);
    const Box6 o = {{x.x, x.y, x.z}, {y.x, y.y, y.z}};
    const uint32_t far = __float_as_uint(x.w), dh = __float_as_uint(y.w);
    const int dfar = (int)(dh & 0xFFu) - 1;
    if (left) { r = far; dr = dfar; } else { l = far; dl = dfar; }
    if (l > r || r >= count) { atomicOr(a.err, kErrCorrupt); break; }
    h = 1u + max(h, dh >> 8);
    const bool root = (dl & dr) < 0;
    const uint32_t i = root ? 0u : dr > dl ? r : l;
    store_node(nodes + 4 * (size_t)i, l, g, r, left ? b : o, left ? o : b);
    b = left ? join(b, o) : join(o, b);
    if constexpr (LIST) {
      a.heights[i] = (uint8_t)min(h, 255u);
      list_node(a, i, l, g, r, root);
    }
    if (root) {
      store_root(a.roots + 8 * (size_t)s, b);
      break;
    }
  }
}

__global__ void __launch_bounds__(kThreads) k_prims_by_id(int kind, const float* __restrict__ verts,
                                                          const uint32_t* __restrict__ idx,
                                                          const float4* __restrict__ sph, uint32_t n,
                                                          float4* __restrict__ prims,
                                                          float* __restrict__ aabb6) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  Box6 b = emit_prim(kind, verts, idx, sph, p, prims, p);
  if (aabb6)
    for (int k = 0; k < 3; ++k) { aabb6[6 * (size_t)p + k] = b.lo[k]; aabb6[6 * (size_t)p + 3 + k] = b.hi[k]; }
}

}  // namespace

cudaError_t launch_tree(const TreeArgs& a, bool list, cudaStream_t s) {
  if (a.n == 0) return cudaSuccess;
  count_launch();
  const uint32_t blocks = tree_windows(a.n);
  const auto k = a.poff ? k_tree<true, false> : list ? k_tree<false, true> : k_tree<false, false>;
  k<<<blocks, kTreeWindow, 0, s>>>(a);
  return cudaGetLastError();
}

void launch_prims_by_id(int kind, const float* verts, const uint32_t* idx, const float4* sph,
                        uint32_t n, float4* prims, float* aabb6, cudaStream_t s) {
  if (n == 0) return;
  count_launch();
  k_prims_by_id<<<(n + kThreads - 1) / kThreads, kThreads, 0, s>>>(kind, verts, idx, sph, n, prims,
                                                                   aabb6);
}

}  // namespace rq

namespace rq {
namespace {

__global__ void __launch_bounds__(kThreads) k_prims_gather(int kind, const float* __restrict__ verts,
                                                           const uint32_t* __restrict__ idx,
                                                           const float4* __restrict__ sph,
                                                           const uint32_t* __restrict__ order, uint32_t n,
                                                           float4* __restrict__ prims) {
  uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  emit_prim(kind, verts, idx, sph, __ldg(order + j), prims, j);
}

}  // namespace

void launch_prims_gather(int kind, const float* verts, const uint32_t* idx, const float4* sph,
                         const uint32_t* order, uint32_t n, float4* prims, cudaStream_t s) {
  if (n == 0) return;
  count_launch();
  k_prims_gather<<<(n + kThreads - 1) / kThreads, kThreads, 0, s>>>(kind, verts, idx, sph, order, n, prims);
}

}  // namespace rq
