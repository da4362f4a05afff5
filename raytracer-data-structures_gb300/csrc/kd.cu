// SAH KD tree on the GPU: constructKDTreeNew / buildTree (accelerators.h:815-988)
// built breadth first, then laid out depth first exactly as the reference lays
// it out (below child = node + 1, above child = next free node after the below
// subtree, accelerators.h:940-947), plus its traversal (kdtreeIntersect,
// accelerators.h:997-1086).
//
// Parameters are the reference's effective ones: maxPrims = 5, isectCost = 80,
// traversalCost = 1, emptyBonus = 0 (the global `char emptyBonus = 0.5f`
// truncates, accelerators.h:767-770); maxDepth = round(8 + 1.3 log2 N).
//
// Edges are sorted once: at the root, one list per axis, ordered by (t,
// start before end, primitive id), the order of buildTree's edge sort
// (:872-879) with ties in id order.  A node's edges are a contiguous segment
// of each list, and a stable partition hands every child its segments still
// sorted.  Per level, for every node still splitting:
//  * the SAH cost of every edge on every axis, with the reference's float
//    operations (no fused multiply-add); nBelow is carried with each edge;
//  * per node and axis, a 64-bit atomicMin of (cost, edge offset) takes the
//    first cheapest edge (buildTree's strict <); the axis is the first from
//    the longest on with a candidate edge, as the retries (:915-919) choose;
//  * the leaf rules (maxPrims, depth, 4x old cost under 16 primitives, three
//    bad refines, :843, :920-925) decide; primitives whose start edge precedes
//    the split go below, those whose end edge follows it go above (:928-934).
// Leaves list their primitives by id (the reference's order inside a leaf
// comes from an unstable sort).
//
// A level is five launches: costs; decisions with the numbering of interior
// nodes and leaf refs; sides of the refs with their ranks (both one-pass
// prefix sums); side counts of the edges, while the host reads the level's
// totals; children (nodes, refs) ; and the partition of the edges.  Small
// trees are bound by launches and the one wait a level, large ones by the
// partition's and cost pass's edge traffic.  GB300 rebuild, against some
// twenty launches a level, edges as four arrays and side flags and ranks as
// four more: 36k spheres 4552 -> 1656 us, 82k triangles 5522 -> 2316, 330k
// 9164 -> 5401, 998k 13824 -> 9880.
#include <algorithm>
#include <atomic>
#include <vector>

#include "rq_build.hpp"
#include "trace_device.cuh"

namespace rq {
namespace {

constexpr int kThreads = 256;
constexpr int kMaxPrims = 5;
constexpr float kIsect = 80.f, kTrav = 1.f, kEmptyBonus = 0.f;
constexpr unsigned long long kNone = ~0ull;

inline unsigned grid(uint64_t n) { return n ? (unsigned)((n + kThreads - 1) / kThreads) : 1u; }

__device__ __forceinline__ uint32_t float_key(float f) {
  uint32_t b = __float_as_uint(__fadd_rn(f, 0.0f));
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

// Level-local node state.
struct LevelNodes {
  float4* lo;         // box minimum, 1 / surface area
  float4* hi;         // box maximum, first ref (bits)
  uint32_t* open;     // ref count of a node still undecided, else 0
  uint32_t* rs;       // first ref
  uint32_t* rc;       // ref count
  int32_t* depth;
  int32_t* bad;       // badRefines
  unsigned long long* best;  // 3 per node, one per axis: (cost key << 32) | edge offset in the node
  int32_t* axis;      // interior nodes: the split axis; leaves: 3
  uint2* split;       // the split edge: ordered t key and (ref << 1 | end)
  uint32_t* irank;    // interior nodes before it
  uint32_t* lofs;     // leaf refs before it
  uint4* plan;        // interior nodes: (sA[rs], sB[rs], sB[rs + rc], first child) for the partition
};

// Edge lists: one per axis, each holding 2 edges per ref of the level (the
// node's refs' edges at [2 rs, 2 rs + 2 rc)), sorted inside every node by
// (t, start before end, ref), the order buildTree's edge sort gives
// (:872-879) with ties in primitive-id order.  An edge is 16 bytes: x the
// ordered float key of t, y ref << 1 | end, z its node, w the number of start
// edges before it in its node (the nBelow of the cost, carried through the
// partitions).  A child's lists come from its parent's by a stable partition,
// so the edges are sorted once, at the root.
struct EdgeLists {
  uint4* base;
  size_t cap;  // edges per list
  __host__ __device__ uint4* list(int a) const { return base + (size_t)a * cap; }
};

// ------------------------------------------------------- one-pass prefix sums
// A tile's exclusive prefix by decoupled look-back: two sums of at most 31
// bits each in one word (high and low half), with the state in the top two
// bits.  The first warp reads 32 earlier tiles a round trip; waits are
// bounded, and a tile that gives up marks itself so later tiles do too.
constexpr unsigned long long kTileAgg = 1ull << 62, kTilePrefix = 2ull << 62, kTileAbort = 3ull << 62;
constexpr unsigned long long kTileValue = (1ull << 62) - 1;
constexpr uint32_t kTilePolls = 1u << 20;  // polls of the same 32 tiles before giving up

__device__ __forceinline__ unsigned long long tile_load(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void tile_store(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long pair31(uint32_t hi, uint32_t lo) {
  return ((unsigned long long)hi << 31) | lo;
}

// The exclusive prefix of thread v over the grid's tiles in tile order; the
// whole block (256 threads) calls it.  tmp: 34 words of shared memory.  The
// total up to and including the block in tmp[33].
__device__ __forceinline__ unsigned long long grid_prefix(unsigned long long v, uint32_t tile,
                                                          unsigned long long* status, unsigned long long* tmp,
                                                          uint32_t* err) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  constexpr uint32_t kW = kThreads / 32;
  unsigned long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) tmp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    unsigned long long total = 0;
#pragma unroll
    for (uint32_t w = 0; w < kW; ++w) total += tmp[w];
    unsigned long long excl = 0;
    if (tile == 0) {
      if (lane == 0) tile_store(status, kTilePrefix | total);
    } else {
      if (lane == 0) tile_store(status + tile, kTileAgg | total);
      uint32_t polls = 0;
      for (int64_t j = (int64_t)tile - 1;;) {
        const int64_t at = j - lane;
        const unsigned long long s = at >= 0 ? tile_load(status + at) : kTilePrefix;
        const uint32_t flag = (uint32_t)(s >> 62);
        const uint32_t prefix = __ballot_sync(0xffffffffu, flag >= 2u);  // prefix or abort
        const uint32_t empty = __ballot_sync(0xffffffffu, flag == 0u);
        const uint32_t use = prefix ? (prefix & (0u - prefix)) * 2u - 1u : 0xffffffffu;  // up to the nearest prefix
        const bool aborted = __any_sync(0xffffffffu, flag == 3u && ((use >> lane) & 1u));
        if (aborted || polls > kTilePolls) {
          if (lane == 0) {
            atomicOr(err, kErrTimeout);
            tile_store(status + tile, kTileAbort);
          }
          excl = 0;
          total = 0;
          break;
        }
        if (empty & use) {
          if (++polls > 64u) __nanosleep(100);
          continue;
        }
        unsigned long long part = ((use >> lane) & 1u) ? s & kTileValue : 0ull;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        excl += part;
        if (prefix) {
          if (lane == 0) tile_store(status + tile, kTilePrefix | ((excl + total) & kTileValue));
          break;
        }
        j -= 32;
        polls = 0;  // the limit is for the same 32 tiles
      }
    }
    if (lane == 0) {
      tmp[32] = excl;
      tmp[33] = excl + total;
    }
  }
  __syncthreads();
  unsigned long long before = tmp[32];
#pragma unroll
  for (uint32_t w = 0; w < kW; ++w) before += w < warp ? tmp[w] : 0ull;
  return before + x - v;
}

// Node k's first state: a leaf by the pre-leaf test (:843), or undecided with
// its box's surface (:855-857).
__device__ __forceinline__ void init_node(const LevelNodes& L, uint32_t k, F3 lo, F3 hi, uint32_t rs, uint32_t rc,
                                          int depth, int bad) {
  const float ax = __fsub_rn(hi.x, lo.x), ay = __fsub_rn(hi.y, lo.y), az = __fsub_rn(hi.z, lo.z);
  const float totalSA = __fmul_rn(2.f, __fadd_rn(__fadd_rn(__fmul_rn(ax, ay), __fmul_rn(ax, az)), __fmul_rn(ay, az)));
  L.lo[k] = make_float4(lo.x, lo.y, lo.z, __fdiv_rn(1.f, totalSA));
  L.hi[k] = make_float4(hi.x, hi.y, hi.z, __uint_as_float(rs));
  L.open[k] = ((int)rc <= kMaxPrims || depth == 0) ? 0u : rc;
  L.rs[k] = rs;
  L.rc[k] = rc;
  L.depth[k] = depth;
  L.bad[k] = bad;
  for (int a = 0; a < 3; ++a) L.best[3 * (size_t)k + a] = kNone;
}

__global__ void k_root_node(LevelNodes L, const int32_t* lohi, float* root, uint32_t n, int depth) {
  if (threadIdx.x != 0) return;
  float b[6];
  for (int q = 0; q < 6; ++q) root[q] = b[q] = ordered_to_float(lohi[q]);
  init_node(L, 0, {b[0], b[1], b[2]}, {b[3], b[4], b[5]}, 0, n, depth, 0);
}

// Root edge lists before the sort: starts of refs 0..n-1, then their ends,
// so a stable sort by t alone orders equal t start-first and by ref.  Also
// the root's refs.
__global__ void k_root_edges(const float* __restrict__ aabb, uint32_t n, uint32_t* __restrict__ t,
                             uint32_t* __restrict__ v, uint32_t* __restrict__ ref_prim, uint32_t* __restrict__ ref_node) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  ref_prim[p] = p;
  ref_node[p] = 0u;
  const float* q = aabb + 6 * (size_t)p;
  for (int a = 0; a < 3; ++a) {
    const size_t at = (size_t)a * 2 * n;
    t[at + p] = float_key(__ldg(q + a));
    v[at + p] = p << 1;
    t[at + n + p] = float_key(__ldg(q + 3 + a));
    v[at + n + p] = (p << 1) | 1u;
  }
}

// The sorted root lists as edges (blockIdx.y: the axis): the start ranks are
// a prefix sum of the start flags.
constexpr int kRootItems = 8;
__global__ void __launch_bounds__(kThreads) k_root_lists(const uint32_t* __restrict__ t, const uint32_t* __restrict__ v,
                                                         uint32_t E, EdgeLists el, unsigned long long* status,
                                                         uint32_t* ticket, uint32_t tiles, uint32_t* err) {
  __shared__ unsigned long long tmp[34];
  __shared__ uint32_t s_tile;
  const int a = blockIdx.y;
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket + a, 1u);
  __syncthreads();
  const uint32_t tile = s_tile, e0 = (tile * kThreads + threadIdx.x) * kRootItems;
  uint32_t vv[kRootItems], starts = 0;
#pragma unroll
  for (int j = 0; j < kRootItems; ++j) {
    vv[j] = e0 + j < E ? __ldg(v + (size_t)a * E + e0 + j) : 1u;
    starts += (vv[j] & 1u) ^ 1u;
  }
  uint32_t rank = (uint32_t)grid_prefix(starts, tile, status + (size_t)a * tiles, tmp, err);
#pragma unroll
  for (int j = 0; j < kRootItems; ++j)
    if (e0 + j < E) {
      el.list(a)[e0 + j] = make_uint4(__ldg(t + (size_t)a * E + e0 + j), vv[j], 0u, rank);
      rank += (vv[j] & 1u) ^ 1u;
    }
}

constexpr int kEdgeItems = 8;
constexpr uint32_t kEdgeRun = 32 * kEdgeItems;               // edges per warp: lane l takes 32 j + l in round j
constexpr uint32_t kEdgeTile = kEdgeRun * (kThreads / 32);  // edges per block of the partition passes
constexpr int kCostItems = 4;
constexpr uint32_t kCostRun = 32 * kCostItems;               // edges per warp of the cost pass

// SAH cost of splitting at every edge of every undecided node, on all three
// axes at once (buildTree :883-912, same float operations).  buildTree tries
// the longest axis and moves to the next only when it has no candidate edge
// (:915-919); every axis's minimum is kept and k_decide takes the first axis
// in that order that has a candidate, which is the same choice.
//
// One warp per run of 128 consecutive edges of one list, lane l taking edge
// 32 j + l in round j.  A round whose lanes share a node takes its minimum by
// one warp reduction; otherwise a segmented shuffle reduction finds every
// node's.  The run that reaches lane 31 is carried into the next round, and
// only runs that end issue an atomicMin (near the root a level has a few
// nodes of millions of edges, and one atomic per edge on one address
// serialises in L2).  The first blocks also clear the level's look-back words.
__device__ __forceinline__ void flush_best(LevelNodes L, uint32_t k, int a, unsigned long long ck) {
  if (ck != kNone) atomicMin(L.best + 3 * (size_t)k + a, ck);
}

__global__ void __launch_bounds__(kThreads) k_cost(EdgeLists el, uint32_t E2, uint32_t runs_per_list, uint32_t M,
                                                   LevelNodes L, unsigned long long* clear, uint32_t clear_words,
                                                   uint32_t* err) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < clear_words; i += gridDim.x * blockDim.x) clear[i] = 0ull;
  const uint32_t gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (gw >= 3 * runs_per_list) return;  // whole warps
  const int lane = threadIdx.x & 31;
  const int a = (int)(gw / runs_per_list);
  const uint32_t run0 = (gw - (uint32_t)a * runs_per_list) * kCostRun;
  const uint4* __restrict__ list = el.list(a);
  uint32_t carry_k = 0xFFFFFFFFu;  // the open run from the previous round (warp-uniform)
  unsigned long long carry = kNone;
  uint4 edge[kCostItems];
  uint32_t open[kCostItems];
#pragma unroll
  for (int j = 0; j < kCostItems; ++j) {
    const uint32_t e = run0 + 32 * j + lane;
    edge[j] = e < E2 ? __ldg(list + e) : make_uint4(0u, 0u, 0xFFFFFFFFu, 0u);
  }
#pragma unroll
  for (int j = 0; j < kCostItems; ++j) {
    if (edge[j].z != 0xFFFFFFFFu && edge[j].z >= M) { atomicOr(err, kErrCorrupt); edge[j].z = 0xFFFFFFFFu; }
    open[j] = edge[j].z != 0xFFFFFFFFu ? __ldg(L.open + edge[j].z) : 0u;
  }
#pragma unroll
  for (int j = 0; j < kCostItems; ++j) {
    const uint32_t e = run0 + 32 * j + lane, k = edge[j].z;
    unsigned long long ck = kNone;
    uint32_t key = 0xFFFFFFFFu, off = 0;
    bool have = false;
    if (open[j]) {
      const float t = key_float(edge[j].x);
      const float4 bl = __ldg(L.lo + k), bh = __ldg(L.hi + k);
      const float lo = a == 0 ? bl.x : a == 1 ? bl.y : bl.z, hi = a == 0 ? bh.x : a == 1 ? bh.y : bh.z;
      if (t > lo && t < hi) {
        const uint32_t rs = __float_as_uint(bh.w), n = open[j];
        const uint32_t nBelow = edge[j].w;
        off = e - 2 * rs;
        const uint32_t nEndIncl = off - nBelow + (edge[j].y & 1u);
        const uint32_t nAbove = n - nEndIncl;
        const float invTotalSA = bl.w;
        const float ex = __fsub_rn(bh.x, bl.x), ey = __fsub_rn(bh.y, bl.y), ez = __fsub_rn(bh.z, bl.z);
        const float d0 = a == 0 ? ey : a == 1 ? ez : ex;  // the other two axes, (a + 1) % 3 and (a + 2) % 3
        const float d1 = a == 0 ? ez : a == 1 ? ex : ey;
        float dd = __fmul_rn(d0, d1), ds = __fadd_rn(d0, d1);
        float belowSA = __fmul_rn(2.f, __fadd_rn(dd, __fmul_rn(__fsub_rn(t, lo), ds)));
        float aboveSA = __fmul_rn(2.f, __fadd_rn(dd, __fmul_rn(__fsub_rn(hi, t), ds)));
        float pB = __fmul_rn(belowSA, invTotalSA), pA = __fmul_rn(aboveSA, invTotalSA);
        float eb = (nAbove == 0 || nBelow == 0) ? kEmptyBonus : 0.f;
        float cost = __fadd_rn(kTrav, __fmul_rn(__fmul_rn(kIsect, __fsub_rn(1.f, eb)),
                                                __fadd_rn(__fmul_rn(pB, (float)nBelow),
                                                          __fmul_rn(pA, (float)nAbove))));
        key = float_key(cost);
        ck = ((unsigned long long)key << 32) | (unsigned long long)off;
        have = true;
      }
    }
    const uint32_t k0 = __shfl_sync(0xffffffffu, k, 0);
    if (__all_sync(0xffffffffu, k == k0)) {  // one node: offsets grow with the lane, so the first lane of the minimum
      const uint32_t m = __reduce_min_sync(0xffffffffu, key);
      const uint32_t at = __ballot_sync(0xffffffffu, have && key == m);
      unsigned long long best = kNone;
      if (at) best = ((unsigned long long)m << 32) | __shfl_sync(0xffffffffu, off, __ffs(at) - 1);
      if (carry_k == k0) {
        if (best < carry) carry = best;
      } else {
        if (lane == 0 && carry_k != 0xFFFFFFFFu) flush_best(L, carry_k, a, carry);
        carry_k = k0;
        carry = best;
      }
      continue;
    }
    // Minimum over the lane's run of equal nodes from this lane on.
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long x = __shfl_down_sync(0xffffffffu, ck, o);
      const uint32_t kk = __shfl_down_sync(0xffffffffu, k, o);
      if (lane + o < 32 && kk == k && x < ck) ck = x;
    }
    const uint32_t kprev = __shfl_up_sync(0xffffffffu, k, 1);
    const bool head = lane == 0 || kprev != k;
    const uint32_t heads = __ballot_sync(0xffffffffu, head);
    const int last = 31 - __clz(heads);  // head of the run that reaches lane 31
    // the carried run continues into lane 0's run or ends here
    if (lane == 0) {
      if (carry_k == k0) { if (carry < ck) ck = carry; }
      else if (carry_k != 0xFFFFFFFFu) flush_best(L, carry_k, a, carry);
    }
    if (head && lane != last && k != 0xFFFFFFFFu) flush_best(L, k, a, ck);
    carry_k = __shfl_sync(0xffffffffu, k, last);
    carry = __shfl_sync(0xffffffffu, ck, last);
  }
  if (lane == 0 && carry_k != 0xFFFFFFFFu) flush_best(L, carry_k, a, carry);
}

// Split decision (:915-925) of an undecided node: the first axis from the
// longest on with a candidate edge; none -> leaf.  Returns whether it is an
// interior node.
__device__ __forceinline__ bool decide_node(EdgeLists el, LevelNodes L, uint32_t k, uint32_t rc, uint32_t E2, uint32_t* err) {
  const float4 lo = L.lo[k], hi = L.hi[k];
  const float ax = __fsub_rn(hi.x, lo.x), ay = __fsub_rn(hi.y, lo.y), az = __fsub_rn(hi.z, lo.z);
  const int axis0 = (ax > ay && ax > az) ? 0 : (ay > az ? 1 : 2);
  unsigned long long bs[3];
  for (int a = 0; a < 3; ++a) bs[a] = L.best[3 * (size_t)k + a];
  for (int q = 0; q < 3; ++q) {
    const int a = (axis0 + q) % 3;
    const unsigned long long b = a == 0 ? bs[0] : a == 1 ? bs[1] : bs[2];
    if (b == kNone) continue;
    const float bestCost = key_float((uint32_t)(b >> 32));
    const float oldCost = __fmul_rn(kIsect, (float)rc);
    const int bad = L.bad[k] + (bestCost > oldCost ? 1 : 0);
    L.bad[k] = bad;
    const bool leaf = (bestCost > __fmul_rn(4.f, oldCost) && rc < 16) || bad == 3;
    if (leaf) return false;
    const uint32_t e = 2 * L.rs[k] + (uint32_t)(b & 0xFFFFFFFFull);
    if (e >= E2) { atomicOr(err, kErrCorrupt); return false; }
    const uint4 edge = el.list(a)[e];
    L.split[k] = make_uint2(edge.x, edge.y);
    L.axis[k] = a;
    return true;
  }
  return false;  // no split found on any axis
}

// Decides every undecided node and numbers the level's interior nodes and
// leaf refs (totals: [0] interiors, [1] leaf refs).
__global__ void __launch_bounds__(kThreads) k_decide(EdgeLists el, LevelNodes L, uint32_t M, uint32_t E2,
                                                     unsigned long long* status, uint32_t* ticket,
                                                     uint32_t* __restrict__ totals, uint32_t* err) {
  __shared__ unsigned long long tmp[34];
  __shared__ uint32_t s_tile;
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
  __syncthreads();
  const uint32_t tile = s_tile, k = tile * kThreads + threadIdx.x;
  uint32_t interior = 0, leaf_refs = 0;
  if (k < M) {
    const uint32_t rc = L.rc[k], open = L.open[k];
    if (open && decide_node(el, L, k, open, E2, err)) {
      interior = 1u;
    } else {
      L.axis[k] = 3;
      leaf_refs = rc;
    }
  }
  const unsigned long long at = grid_prefix(pair31(interior, leaf_refs), tile, status, tmp, err);
  if (k < M) {
    L.irank[k] = (uint32_t)(at >> 31);
    L.lofs[k] = (uint32_t)(at & 0x7FFFFFFFull);
  }
  if (tile == gridDim.x - 1 && threadIdx.x == 0) {
    totals[0] = (uint32_t)((tmp[33] & kTileValue) >> 31);
    totals[1] = (uint32_t)(tmp[33] & 0x7FFFFFFFull);
  }
}

// Below/above sides (:928-934): a ref whose start edge precedes the split
// edge in the chosen axis's sorted order goes below, one whose end edge
// follows it goes above.  The order is (t key, start before end, ref), so
// the comparison needs only the ref's box and the split edge, not the list.
// sides[r] = (below refs before r | below flag << 31, the same for above),
// r = 0 .. R; totals: [2] below refs, [3] above refs.
constexpr uint32_t kSideFlag = 0x80000000u, kSideRank = 0x7FFFFFFFu;
constexpr int kSideItems = 4;
__global__ void __launch_bounds__(kThreads) k_sides(const uint32_t* __restrict__ ref_prim,
                                                    const uint32_t* __restrict__ ref_node, uint32_t R, uint32_t M,
                                                    const float* __restrict__ aabb, LevelNodes L,
                                                    uint2* __restrict__ sides, unsigned long long* status,
                                                    uint32_t* ticket, uint32_t* __restrict__ totals, uint32_t* err) {
  __shared__ unsigned long long tmp[34];
  __shared__ uint32_t s_tile;
  if (threadIdx.x == 0) s_tile = atomicAdd(ticket, 1u);
  __syncthreads();
  const uint32_t tile = s_tile, r0 = (tile * kThreads + threadIdx.x) * kSideItems;
  uint32_t b = 0, ab = 0;  // flags of the thread's refs
  uint32_t node[kSideItems], axis[kSideItems], prim[kSideItems];
#pragma unroll
  for (int j = 0; j < kSideItems; ++j) {
    node[j] = r0 + j < R ? __ldg(ref_node + r0 + j) : 0xFFFFFFFFu;
    prim[j] = r0 + j < R ? __ldg(ref_prim + r0 + j) : 0u;
    if (node[j] != 0xFFFFFFFFu && node[j] >= M) { atomicOr(err, kErrCorrupt); node[j] = 0xFFFFFFFFu; }
  }
#pragma unroll
  for (int j = 0; j < kSideItems; ++j) axis[j] = node[j] != 0xFFFFFFFFu ? (uint32_t)L.axis[node[j]] : 3u;
#pragma unroll
  for (int j = 0; j < kSideItems; ++j) {
    if (axis[j] == 3u) continue;
    const uint2 sp = L.split[node[j]];
    const uint32_t sk = sp.x, sv = sp.y, sr = sv >> 1, r = r0 + j;
    const float* q = aabb + 6 * (size_t)prim[j] + axis[j];
    const uint32_t lo = float_key(__ldg(q)), hi = float_key(__ldg(q + 3));
    if (lo < sk || (lo == sk && ((sv & 1u) || r < sr))) b |= 1u << j;    // (lo, start, r) < split
    if (hi > sk || (hi == sk && (!(sv & 1u) || r > sr))) ab |= 1u << j;  // (hi, end, r) > split
  }
  const unsigned long long at = grid_prefix(pair31(__popc(b), __popc(ab)), tile, status, tmp, err);
  uint32_t sb = (uint32_t)(at >> 31), sa = (uint32_t)(at & 0x7FFFFFFFull);
#pragma unroll
  for (int j = 0; j < kSideItems; ++j) {
    const uint32_t fb = (b >> j) & 1u, fa = (ab >> j) & 1u;
    if (r0 + j <= R) sides[r0 + j] = make_uint2(sb | (fb ? kSideFlag : 0u), sa | (fa ? kSideFlag : 0u));
    sb += fb;
    sa += fa;
  }
  if (tile == gridDim.x - 1 && threadIdx.x == 0) {
    totals[2] = (uint32_t)((tmp[33] & kTileValue) >> 31);
    totals[3] = (uint32_t)(tmp[33] & 0x7FFFFFFFull);
  }
}

// Children's edge lists: a stable partition of every interior node's edges,
// on each axis, into its below child (refs with the below flag) and above
// child (refs with the above flag); straddling refs go to both.  With sB / sA
// the below / above refs before a ref (sides), and BS, BE, AS, AE the
// list-wide counts of below-start, below-end, above-start and above-end
// edges before e:
//   below child: position BS + BE + 2 sA[rs], ref sA[rs] + sB[r],
//                start rank BS - sB[rs]
//   above child: position AS + AE + 2 sB[re], ref sB[re] + sA[r],
//                start rank AS - sA[rs]
// (re = rs + rc; children are laid out node by node, below before above,
// and leaf refs count in neither), matching k_spawn_emit's numbering of
// the refs.  Per node the bases come from plan[k] = (sA[rs], sB[rs], sB[re],
// first child), written by k_spawn_emit.
//
// Passes, none waiting on another block: k_part_count counts each tile's
// (BS, BE) and (AS, AE), packed 31 bits apiece in two 64-bit words (lists
// hold fewer than 2^31 edges, so the fields never carry), and keeps the side
// flags as one ballot word per 32 edges; k_partition adds up the earlier
// tiles' counts (k_part_scan does when there are more than kPartSelf) and the
// warp offsets inside the tile, and scatters.
constexpr uint32_t kPartSelf = 1024;

__global__ void __launch_bounds__(kThreads) k_part_count(EdgeLists el, uint32_t E2, uint32_t tiles_per_list,
                                                         uint32_t R, const uint2* __restrict__ sides,
                                                         uint32_t* __restrict__ sideB, uint32_t* __restrict__ sideA,
                                                         unsigned long long* __restrict__ tile_cnt, uint32_t* err) {
  __shared__ unsigned long long wsum[2][kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t tile = blockIdx.x, a = tile / tiles_per_list;
  const uint32_t run0 = (tile - a * tiles_per_list) * kEdgeTile + (uint32_t)warp * kEdgeRun;
  const size_t words = (size_t)(E2 + 31) / 32;  // ballot words per list
  uint32_t v[kEdgeItems];
  uint2 sd[kEdgeItems];
#pragma unroll
  for (int j = 0; j < kEdgeItems; ++j) {
    const uint32_t e = run0 + 32 * j + lane;
    v[j] = e < E2 ? __ldg(&el.list(a)[e].y) : 0xFFFFFFFFu;
  }
#pragma unroll
  for (int j = 0; j < kEdgeItems; ++j) {
    sd[j] = make_uint2(0u, 0u);
    if (v[j] != 0xFFFFFFFFu) {
      if ((v[j] >> 1) < R) sd[j] = __ldg(sides + (v[j] >> 1));
      else atomicOr(err, kErrCorrupt);
    }
  }
  unsigned long long t0 = 0, t1 = 0;
#pragma unroll
  for (int j = 0; j < kEdgeItems; ++j) {
    const uint32_t kb = __ballot_sync(0xffffffffu, (sd[j].x & kSideFlag) != 0u);
    const uint32_t ka = __ballot_sync(0xffffffffu, (sd[j].y & kSideFlag) != 0u);
    const uint32_t em = __ballot_sync(0xffffffffu, (v[j] & 1u) != 0u);
    const uint32_t w = (run0 >> 5) + (uint32_t)j;
    if (lane == 0 && w < words) {
      sideB[(size_t)a * words + w] = kb;
      sideA[(size_t)a * words + w] = ka;
    }
    t0 += pair31(__popc(kb & em), __popc(kb & ~em));
    t1 += pair31(__popc(ka & em), __popc(ka & ~em));
  }
  if (lane == 0) {
    wsum[0][warp] = t0;
    wsum[1][warp] = t1;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    unsigned long long x = 0;
    for (int w = 0; w < kThreads / 32; ++w) x += wsum[threadIdx.x][w];
    tile_cnt[2 * (size_t)tile + threadIdx.x] = x;
  }
}

// Exclusive prefix of the tile counts of list blockIdx.x, both words, in
// place (one block per list; each thread sums a contiguous chunk).
__global__ void __launch_bounds__(1024) k_part_scan(unsigned long long* tile_cnt, uint32_t tiles_per_list) {
  __shared__ unsigned long long part[2][1024];
  const uint32_t t = threadIdx.x, per = (tiles_per_list + 1023) / 1024;
  unsigned long long* c = tile_cnt + 2 * (size_t)blockIdx.x * tiles_per_list;
  const uint32_t lo = t * per, hi = min(lo + per, tiles_per_list);
  unsigned long long s0 = 0, s1 = 0;
  for (uint32_t i = lo; i < hi; ++i) {
    s0 += c[2 * (size_t)i];
    s1 += c[2 * (size_t)i + 1];
  }
  part[0][t] = s0;
  part[1][t] = s1;
  __syncthreads();
  for (uint32_t o = 1; o < 1024; o <<= 1) {  // inclusive Hillis-Steele scan of the chunk sums
    const unsigned long long x0 = t >= o ? part[0][t - o] : 0ull, x1 = t >= o ? part[1][t - o] : 0ull;
    __syncthreads();
    part[0][t] += x0;
    part[1][t] += x1;
    __syncthreads();
  }
  unsigned long long r0 = part[0][t] - s0, r1 = part[1][t] - s1;
  for (uint32_t i = lo; i < hi; ++i) {
    const unsigned long long v0 = c[2 * (size_t)i], v1 = c[2 * (size_t)i + 1];
    c[2 * (size_t)i] = r0;
    c[2 * (size_t)i + 1] = r1;
    r0 += v0;
    r1 += v1;
  }
}

template <bool SCANNED>
__global__ void __launch_bounds__(kThreads) k_partition(EdgeLists el, uint32_t E2, uint32_t tiles_per_list,
                                                        LevelNodes L, const uint32_t* __restrict__ sideB,
                                                        const uint32_t* __restrict__ sideA,
                                                        const unsigned long long* __restrict__ tile_cnt,
                                                        const uint2* __restrict__ sides, EdgeLists out,
                                                        uint32_t E2next, uint32_t* err) {
  __shared__ unsigned long long wpre[2][kThreads / 32], wsum[2][kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t tile = blockIdx.x, a = tile / tiles_per_list;
  const uint32_t run0 = (tile - a * tiles_per_list) * kEdgeTile + (uint32_t)warp * kEdgeRun;
  const size_t words = (size_t)(E2 + 31) / 32;
  uint4 edge[kEdgeItems];
  uint32_t kb[kEdgeItems], ka[kEdgeItems];
#pragma unroll
  for (int j = 0; j < kEdgeItems; ++j) {
    const uint32_t e = run0 + 32 * j + lane, w = (run0 >> 5) + (uint32_t)j;
    kb[j] = w < words ? __ldg(sideB + (size_t)a * words + w) : 0u;
    ka[j] = w < words ? __ldg(sideA + (size_t)a * words + w) : 0u;
    edge[j] = e < E2 ? __ldg(el.list(a) + e) : make_uint4(0u, 0u, 0u, 0u);
  }
  unsigned long long p0 = 0, p1 = 0;
  if (SCANNED) {
    p0 = __ldg(tile_cnt + 2 * (size_t)tile);
    p1 = __ldg(tile_cnt + 2 * (size_t)tile + 1);
  } else {
    for (uint32_t t = a * tiles_per_list + threadIdx.x; t < tile; t += kThreads) {
      p0 += __ldg(tile_cnt + 2 * (size_t)t);
      p1 += __ldg(tile_cnt + 2 * (size_t)t + 1);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      p0 += __shfl_xor_sync(0xffffffffu, p0, o);
      p1 += __shfl_xor_sync(0xffffffffu, p1, o);
    }
  }
  unsigned long long t0 = 0, t1 = 0;
#pragma unroll
  for (int j = 0; j < kEdgeItems; ++j) {
    const uint32_t em = __ballot_sync(0xffffffffu, (edge[j].y & 1u) != 0u);
    t0 += pair31(__popc(kb[j] & em), __popc(kb[j] & ~em));
    t1 += pair31(__popc(ka[j] & em), __popc(ka[j] & ~em));
  }
  if (lane == 0) {
    wpre[0][warp] = t0;
    wpre[1][warp] = t1;
    wsum[0][warp] = p0;
    wsum[1][warp] = p1;
  }
  __syncthreads();
  if (!SCANNED) {
    p0 = p1 = 0;
    for (int w = 0; w < kThreads / 32; ++w) {
      p0 += wsum[0][w];
      p1 += wsum[1][w];
    }
  }
  for (int w = 0; w < warp; ++w) {
    p0 += wpre[0][w];
    p1 += wpre[1][w];
  }
  uint32_t cbs = (uint32_t)(p0 & 0x7FFFFFFFull), cbe = (uint32_t)(p0 >> 31);
  uint32_t cas = (uint32_t)(p1 & 0x7FFFFFFFull), cae = (uint32_t)(p1 >> 31);
  const uint32_t lt = (1u << lane) - 1u, me = 1u << lane;
#pragma unroll
  for (int j = 0; j < kEdgeItems; ++j) {
    const uint32_t em = __ballot_sync(0xffffffffu, (edge[j].y & 1u) != 0u);
    const uint32_t bs = kb[j] & ~em, be = kb[j] & em, as = ka[j] & ~em, ae = ka[j] & em;
    const bool b = (kb[j] & me) != 0u, ab = (ka[j] & me) != 0u;
    if (b || ab) {
      const uint32_t r = edge[j].y >> 1, end = edge[j].y & 1u;
      const uint4 pl = __ldg(L.plan + edge[j].z);  // (sA[rs], sB[rs], sB[re], first child)
      const uint2 sd = __ldg(sides + r);
      if (b) {
        const uint32_t nbs = cbs + __popc(bs & lt), nbe = cbe + __popc(be & lt);
        const uint32_t pos = nbs + nbe + 2 * pl.x;
        if (pos >= E2next) atomicOr(err, kErrCorrupt);
        else out.list(a)[pos] = make_uint4(edge[j].x, ((pl.x + (sd.x & kSideRank)) << 1) | end, pl.w, nbs - pl.y);
      }
      if (ab) {
        const uint32_t nas = cas + __popc(as & lt), nae = cae + __popc(ae & lt);
        const uint32_t pos = nas + nae + 2 * pl.z;
        if (pos >= E2next) atomicOr(err, kErrCorrupt);
        else out.list(a)[pos] = make_uint4(edge[j].x, ((pl.z + (sd.y & kSideRank)) << 1) | end, pl.w + 1, nas - pl.x);
      }
    }
    cbs += __popc(bs);
    cbe += __popc(be);
    cas += __popc(as);
    cae += __popc(ae);
  }
}

// Global node table (breadth-first ids).
struct Table {
  int32_t* leaf;        // 1 leaf, 0 interior
  int32_t* axis;
  float* split;
  uint32_t* child0;
  uint32_t* child1;
  uint32_t* count;      // leaf primitive count
  uint32_t* pool_off;   // leaf primitives in the pool
};

// Threads up to M: interior nodes spawn their two children (whose refs'
// places follow from the sides, see the partition), every node fills its
// table entry.  Threads up to R: stable filter of every interior node's refs
// into its children; leaf refs to the pool.
__global__ void __launch_bounds__(kThreads) k_spawn_emit(LevelNodes L, uint32_t M, const uint2* __restrict__ sides,
                                                         uint32_t pool_base, uint32_t level_base, uint32_t next_base,
                                                         Table T, LevelNodes N, uint32_t M2,
                                                         const uint32_t* __restrict__ ref_prim,
                                                         const uint32_t* __restrict__ ref_node, uint32_t R,
                                                         uint32_t* __restrict__ out_prim, uint32_t* __restrict__ out_node,
                                                         uint32_t* __restrict__ pool, uint32_t R2, uint32_t pool_cap,
                                                         uint32_t* err) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < R) {
    const uint32_t r = i, k = __ldg(ref_node + r), p = __ldg(ref_prim + r);
    const uint2 s = __ldg(sides + r);
    const uint32_t rs = L.rs[k];
    if (L.axis[k] == 3) {
      const uint32_t q = pool_base + L.lofs[k] + (r - rs);
      if (q >= pool_cap) atomicOr(err, kErrCorrupt);
      else pool[q] = p;
    } else {
      const uint32_t c = 2 * L.irank[k];
      if (s.x & kSideFlag) {
        const uint32_t o = (__ldg(&sides[rs].y) & kSideRank) + (s.x & kSideRank);
        if (o >= R2) atomicOr(err, kErrCorrupt);
        else { out_prim[o] = p; out_node[o] = c; }
      }
      if (s.y & kSideFlag) {
        const uint32_t o = (__ldg(&sides[rs + L.rc[k]].x) & kSideRank) + (s.y & kSideRank);
        if (o >= R2) atomicOr(err, kErrCorrupt);
        else { out_prim[o] = p; out_node[o] = c + 1; }
      }
    }
  }
  if (i >= M) return;
  const uint32_t k = i, g = level_base + k, rs = L.rs[k], rc = L.rc[k];
  const int axis = L.axis[k];
  if (axis == 3) {
    T.leaf[g] = 1;
    T.count[g] = rc;
    T.pool_off[g] = pool_base + L.lofs[k];
    return;
  }
  const uint32_t c = 2 * L.irank[k];
  if (c + 1 >= M2) { atomicOr(err, kErrCorrupt); return; }
  const float ts = key_float(L.split[k].x);
  T.leaf[g] = 0;
  T.axis[g] = axis;
  T.split[g] = ts;
  T.child0[g] = next_base + c;
  T.child1[g] = next_base + c + 1;
  const uint2 s0 = __ldg(sides + rs), s1 = __ldg(sides + rs + rc);
  const uint32_t b0 = s0.x & kSideRank, a0 = s0.y & kSideRank, b1 = s1.x & kSideRank, a1 = s1.y & kSideRank;
  const float4 lo = L.lo[k], hi = L.hi[k];
  const int depth = L.depth[k] - 1, bad = L.bad[k];
  F3 cut_hi = {hi.x, hi.y, hi.z}, cut_lo = {lo.x, lo.y, lo.z};
  if (axis == 0) cut_hi.x = cut_lo.x = ts;  // bounds0.max[axis] = bounds1.min[axis] = tSplit
  else if (axis == 1) cut_hi.y = cut_lo.y = ts;
  else cut_hi.z = cut_lo.z = ts;
  init_node(N, c, {lo.x, lo.y, lo.z}, cut_hi, a0 + b0, b1 - b0, depth, bad);
  init_node(N, c + 1, cut_lo, {hi.x, hi.y, hi.z}, b1 + a0, a1 - a0, depth, bad);
  L.plan[k] = make_uint4(a0, b0, b1, c);
}

// Depth-first layout: subtree sizes bottom-up, positions top-down, three
// levels a launch (a level's node lies below one node of the level two up, so
// that node's thread serves it: 30 levels took 60 launches one by one).
constexpr int kLayoutLevels = 3;
template <int D>
__device__ uint32_t subtree_size(const Table& T, uint32_t g, uint32_t* __restrict__ size, uint32_t total, uint32_t* err) {
  uint32_t s = 1;
  if (!T.leaf[g]) {
    const uint32_t c0 = T.child0[g], c1 = T.child1[g];
    if (c0 >= total || c1 >= total) {
      atomicOr(err, kErrCorrupt);
    } else if constexpr (D > 1) {
      s += subtree_size<D - 1>(T, c0, size, total, err) + subtree_size<D - 1>(T, c1, size, total, err);
    } else {
      s += size[c0] + size[c1];
    }
  }
  size[g] = s;
  return s;
}
template <int D>
__global__ void k_sizes(Table T, uint32_t lo, uint32_t hi, uint32_t* __restrict__ size, uint32_t total, uint32_t* err) {
  const uint32_t g = lo + blockIdx.x * blockDim.x + threadIdx.x;
  if (g < hi) subtree_size<D>(T, g, size, total, err);
}

template <int D>
__device__ void place_children(const Table& T, uint32_t g, uint32_t p, const uint32_t* __restrict__ size,
                               uint32_t* __restrict__ pos, uint32_t total) {
  if (T.leaf[g]) return;
  const uint32_t c0 = T.child0[g], c1 = T.child1[g];
  if (c0 >= total || c1 >= total) return;
  const uint32_t p1 = p + 1 + size[c0];
  pos[c0] = p + 1;
  pos[c1] = p1;
  if constexpr (D > 1) {
    place_children<D - 1>(T, c0, p + 1, size, pos, total);
    place_children<D - 1>(T, c1, p1, size, pos, total);
  }
}
__global__ void k_positions(Table T, uint32_t lo, uint32_t hi, const uint32_t* __restrict__ size,
                            uint32_t* __restrict__ pos, uint32_t total) {
  const uint32_t g = lo + blockIdx.x * blockDim.x + threadIdx.x;
  if (g < hi) place_children<kLayoutLevels>(T, g, pos[g], size, pos, total);
}

__global__ void k_leaf_counts(Table T, uint32_t total, const uint32_t* __restrict__ pos, uint32_t* __restrict__ cnt) {
  uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g > total) return;
  if (g == total) { cnt[total] = 0; return; }
  if (pos[g] >= total) return;
  cnt[pos[g]] = (T.leaf[g] && T.count[g] >= 2) ? T.count[g] : 0u;
}

// Final KdAccelNode words (accelerators.h:718-761) and leaf primitive indices.
__global__ void k_write_nodes(Table T, uint32_t total, const uint32_t* __restrict__ pos,
                              const uint32_t* __restrict__ off, const uint32_t* __restrict__ pool,
                              int4* __restrict__ nodes, int32_t* __restrict__ prim_idx, uint32_t n_idx,
                              uint32_t pool_cap, uint32_t* err) {
  uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= total) return;
  const uint32_t p = pos[g];
  if (p >= total) { atomicOr(err, kErrCorrupt); return; }
  if (T.leaf[g] && (T.pool_off[g] + T.count[g] > pool_cap ||
                    (T.count[g] >= 2 && off[p] + T.count[g] > n_idx))) {
    atomicOr(err, kErrCorrupt);
    return;
  }
  if (!T.leaf[g] && T.child1[g] >= total) { atomicOr(err, kErrCorrupt); return; }
  if (T.leaf[g]) {
    const uint32_t np = T.count[g];
    int w0 = 0;
    if (np == 1) w0 = (int)pool[T.pool_off[g]];
    else if (np >= 2) {
      w0 = (int)off[p];
      for (uint32_t i = 0; i < np; ++i) prim_idx[off[p] + i] = (int)pool[T.pool_off[g] + i];
    }
    nodes[p] = make_int4(w0, 3 | (int)(np << 2), (int)np, 0);
  } else {
    nodes[p] = make_int4(__float_as_int(T.split[g]), T.axis[g] | (int)(pos[T.child1[g]] << 2), 0, 0);
  }
}

// ------------------------------------------------------------- traversal

struct Todo {
  int node;
  float tMin, tMax;
};

// The walk of ray r; returns whether an any-hit query found a hit (closest-hit
// queries store their hit).
template <int KIND, bool ANY, bool REF>
__device__ __forceinline__ bool kd_walk_ray(const KdView& kd, uint32_t n_nodes, const float4* __restrict__ rays,
                                            uint32_t r, float4* __restrict__ hits, uint32_t* err) {
  bool occluded = false;
  {
    float4 ra = __ldg(rays + 2 * (size_t)r), rb = __ldg(rays + 2 * (size_t)r + 1);
    F3 o = {ra.x, ra.y, ra.z}, d = {rb.x, rb.y, rb.z};
    const float rtmin = ra.w, rtmax = rb.w;
    float best = rtmax, bu = 0.f, bv = 0.f;
    uint32_t bprim = kMiss;
    F3 inv = {__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z)};
    const float* R = kd.root;
    float tMin, tMax;
    bool in;
    if (REF) {
      in = box_ref(o, d, R[0], R[3], R[1], R[4], R[2], R[5], tMin, tMax);
    } else {
      float tn;
      const SlabRay sr = slab_ray(o, d);
      if (zero_dir(sr)) {  // the exact box test (rq_device.cuh)
        in = slab_box<true>(sr, o, R[0], R[3], R[1], R[4], R[2], R[5], rtmin, best, tn);
        tMax = __fmaf_rn(slab_exit<true>(sr, o, R[0], R[3], R[1], R[4], R[2], R[5], best), kWidenExact, sr.eps);
      } else {
        in = slab_box<false>(sr, o, R[0], R[3], R[1], R[4], R[2], R[5], rtmin, best, tn);
        tMax = __fmaf_rn(slab_exit<false>(sr, o, R[0], R[3], R[1], R[4], R[2], R[5], best), kWiden, sr.eps);
      }
      tMin = tn;
    }
    if (in) {
      Todo todo[kStackSize];
      int tp = 0, node = 0;
      const float oo[3] = {o.x, o.y, o.z}, dv[3] = {d.x, d.y, d.z}, iv[3] = {inv.x, inv.y, inv.z};
      uint32_t steps = 0;
      // While-while: descend interior nodes to a leaf, then test the leaf, so
      // the lanes of a warp test their leaves together (one loop over node
      // kinds left lanes of both kinds waiting on each other at every step).
      // The per-ray order of visits is unchanged.
      const uint32_t limit = 2u * n_nodes + 8u;
      bool bad = false;
      for (;;) {
        if (++steps > limit) { atomicOr(err, kErrCorrupt); break; }
        if (!REF && best < tMin) break;
        int4 w = __ldg(kd.nodes + node);
        while ((w.y & 3) != 3) {
          const int axis = w.y & 3;
          const float split = __int_as_float(w.x);
          const float tPlane = __fmul_rn(__fsub_rn(split, oo[axis]), iv[axis]);
          const bool belowFirst = (oo[axis] < split) || (oo[axis] == split && dv[axis] <= 0.f);
          const int above = w.y >> 2;
          const int first = belowFirst ? node + 1 : above, second = belowFirst ? above : node + 1;
          if (tPlane > tMax || tPlane <= 0.f) {
            node = first;
          } else if (tPlane < tMin) {
            node = second;
          } else {
            if (tp >= kStackSize) { atomicOr(err, kErrStackOverflow); bad = true; break; }
            todo[tp++] = {second, tPlane, tMax};
            node = first;
            tMax = tPlane;
          }
          if (++steps > limit) { atomicOr(err, kErrCorrupt); bad = true; break; }
          w = __ldg(kd.nodes + node);
        }
        if (bad) break;
        const int np = w.z;
        bool done = false;
        for (int i = 0; i < np; ++i) {
          const uint32_t id = (uint32_t)(np == 1 ? w.x : __ldg(kd.prim_idx + w.x + i));
          if (KIND == kTriangles) {
            const float4* q = kd.prims + 3 * (size_t)id;
            float t, u, v;
            if (tri_mt(__ldg(q), __ldg(q + 1), __ldg(q + 2), o, d, rtmin, ANY ? rtmax : best, t, u, v)) {
              if (ANY) { done = true; break; }
              best = t; bprim = id; bu = u; bv = v;
            }
          } else {
            const float4 s = __ldg(kd.prims + id);
            if (ANY || REF) {
              float t0, t1, t;
              if (REF ? sphere_ref(s, o, d, t0, t1) : sphere_closest(s, o, d, rtmin, rtmax, false, t)) {
                if (ANY) { done = true; break; }
              }
            }
            if (!ANY) {
              float t;
              if (sphere_closest(s, o, d, rtmin, best, REF, t)) { best = t; bprim = id; bu = bv = 0.f; }
            }
          }
        }
        if (done) { occluded = true; break; }
        if (tp > 0) {
          --tp;
          node = todo[tp].node;
          tMin = todo[tp].tMin;
          tMax = todo[tp].tMax;
        } else {
          break;
        }
      }
    }
    if (!ANY) hits[r] = make_float4(best, __uint_as_float(bprim), bu, bv);
  }
  return occluded;
}

template <int KIND, bool ANY, bool REF>
__global__ void __launch_bounds__(128) k_trace_kd(KdView kd, uint32_t n_nodes, const float4* __restrict__ rays,
                                                  uint32_t n, float4* __restrict__ hits,
                                                  uint32_t* __restrict__ occ, uint32_t* err) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  const bool occluded = r < n && kd_walk_ray<KIND, ANY, REF>(kd, n_nodes, rays, r, hits, err);
  if (ANY) {
    uint32_t bits = __ballot_sync(0xffffffffu, occluded);
    uint32_t w0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u);
    if ((threadIdx.x & 31) == 0 && w0 < n) occ[w0 >> 5] = bits;
  }
}

// The REFERENCE walk as persistent warps: a grid the GPU holds at once, each
// warp taking the next 32 rays from a counter (work, zeroed) until none are
// left.
template <int KIND, bool ANY>
__global__ void __launch_bounds__(128) k_trace_kd_warps(KdView kd, uint32_t n_nodes, const float4* __restrict__ rays,
                                                        uint32_t n, float4* __restrict__ hits,
                                                        uint32_t* __restrict__ occ, uint32_t* err, uint32_t* work) {
  const uint32_t lane = threadIdx.x & 31;
  for (;;) {
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(work, 32u);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= n) break;
    const uint32_t r = base + lane;
    const bool occluded = r < n && kd_walk_ray<KIND, ANY, true>(kd, n_nodes, rays, r, hits, err);
    if (ANY) {
      const uint32_t bits = __ballot_sync(0xffffffffu, occluded);
      if (lane == 0) occ[base >> 5] = bits;
    }
  }
}

// The FAST walk as persistent warps whose rays share the warp's lanes, as
// walk_warp (trace_device.cuh) does for the BVH: a round is at most kKdChunk
// interior nodes a lane, then the leaves that lanes reached, then a meeting
// where idle lanes take over the last todo entry (the farthest subtree) of
// busy ones.
//
// kdtreeIntersect's answer depends on its order (the first closest hit wins,
// and the walk ends at the first entry that begins behind the best hit), so
// the shared walk keeps track of it:
//  * every piece of a ray's walk carries its place in that order: a piece
//    owns [lo, hi] of the numbers, what is taken from it gets the upper half
//    (it comes later, but before what was taken earlier), and equal t go to
//    the smaller lo (sh.key = (t, lo));
//  * a hit found before its leaf's interval begins (t < tMin: a primitive
//    that reaches into nearer leaves) belongs to an earlier leaf.  The
//    one-lane walk finds it there, or ends before it gets here, unless
//    rounding made it skip the earlier leaf.  The shared walk only notes the
//    smallest such t (sh.doubt), and a ray whose noted t is smaller than its
//    best hit is walked again by its own lane alone.
// Every other hit lies in its own interval, so the one-lane walk reaches it
// whenever it is the answer, and what a best hit prunes here begins behind
// it in the one-lane walk's order too.
//
// Rays sit in shared memory (a piece moves without its ray; the split axis
// indexes them), todo entries are 8 bytes (an entry ends where the one below
// it begins, the last one at t_end).  The node loop converges at every step:
// left to itself (a loop a lane leaves at its leaf) it was up to 1.6 times
// slower.  Leaves hold from one to some dozens of primitives, so each lane
// testing its own left the warp waiting for the longest: the lists of the
// leaves reached are tested as one, a primitive a lane, and a leaf's answer
// is the smallest (t, place in the list), which is what testing them in turn
// finds.
// us, one lane a ray / lanes shared, own leaves / leaves spread: 1023 random
// rays 194 / 60 / 42, 300k random rays 377 / 279 / 237 (any hit 347 / 209 /
// 162), 307k camera rays 260 / 215 / 174, their shadow rays 348 / 257 / 212, 2M
// bounce rays 2020 / 1950 / 1400, 2M coherent shadow rays 697 / 778 / 674.
// Coherent rays by the million lose on small trees, the more the smaller: 3M
// parallel rays 86 -> 166 on 12 triangles, 180 -> 210 on 3,468, 966 -> 1028 on
// 998k (one lane a ray / now); random rays on the same trees gain from 48
// triangles on (296 -> 241, 701 -> 510, 1958 -> 1358), and no size tells the two
// apart.
constexpr int kKdChunk = 4;  // 2 / 3 / 4 / 5 / 8 / 16, 2M bounce rays: 1681 / 1569 / 1527 / 1518 / 1565 / 1733 us; 300k shadow rays: 176 / 174 / 172 / 175 / 186 / 212
constexpr uint32_t kKdLeafMax = 1u << 26;  // primitives of a leaf tested at one meeting (32 lanes' fit 32 bits)
constexpr int kKdIdle = 8;   // lanes idle before pieces move; 5 / 8 / 12: within 1%

__device__ __forceinline__ int2 load_kd(const int4* __restrict__ nodes, int node) {
  return __ldg(reinterpret_cast<const int2*>(nodes + node));
}

template <bool ANY>
struct KdShare {
  float o[3][32], inv[3][32], d[3][32], tmin[32], tmax[32];
  uint32_t give[32];
  unsigned long long leaf[ANY ? 1 : 32]; // a lane's leaf: (t, its place among the leaves' primitives) of the best hit
  unsigned long long key[ANY ? 1 : 32];  // best hit per ray: (order-preserving bits of t + 0, place)
  uint32_t doubt[ANY ? 1 : 32];          // smallest t found before its leaf, order-preserving bits
  uint32_t prim[ANY ? 1 : 32];
  float t[ANY ? 1 : 32];
  float2 uv[ANY ? 1 : 32];
};

// Blocks an SM: closest hit 6 / 7 / 8: 1641 / 1452 / 1527 us on the bounce
// rays (8 spill), any hit 8 / 9 / 10: 701 / 674 / 744 on the 2M shadow rays.
// PLACED: every warp has its rays by its place, far apart (k_trace_once,
// trace.cu; 100k shadow rays 130 -> 95 us), instead of taking them from a
// counter (one kernel for both: 1517 us on the bounce rays, 1400 apart).
template <int KIND, bool ANY, bool PLACED>
__global__ void __launch_bounds__(128, ANY ? 9 : 7) k_trace_kd_shared(KdView kd, uint32_t n_nodes,
                                                                   const float4* __restrict__ rays, uint32_t n,
                                                                   float4* __restrict__ hits,
                                                                   uint32_t* __restrict__ occ, uint32_t* err,
                                                                   uint32_t* work, uint32_t grab) {
  __shared__ KdShare<ANY> share[4];
  KdShare<ANY>& sh = share[threadIdx.x >> 5];
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  const uint32_t limit = 2u * n_nodes + 8u;  // meetings: a piece has a node of its ray behind it for every one
  int2 todo[kStackSize];                     // (node, bits of tMin)
  for (;;) {
    uint32_t base = 0, r;
    if constexpr (!PLACED) {
      if (lane == 0) base = atomicAdd(work, grab);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base >= n) break;
      r = base + lane;
    } else if constexpr (ANY) {
      r = ((lane >> 3) * gridDim.x + blockIdx.x) * 32u + ((lane & 7u) << 2 | threadIdx.x >> 5);
    } else {
      r = (lane * gridDim.x + blockIdx.x) * 4u + (threadIdx.x >> 5);
    }
    const bool own = lane < grab && r < n;
    float first = 0.f, last = 0.f;  // the ray's interval in the root box
    bool start = false;
    __syncwarp();
    if (own) {
      const float4 ra = __ldcs(rays + 2 * (size_t)r), rb = __ldcs(rays + 2 * (size_t)r + 1);
      const F3 o = {ra.x, ra.y, ra.z}, d = {rb.x, rb.y, rb.z};
      const SlabRay sr = slab_ray(o, d);
      const float* R = kd.root;
      if (zero_dir(sr)) {  // the exact box test (rq_device.cuh)
        start = slab_box<true>(sr, o, R[0], R[3], R[1], R[4], R[2], R[5], ra.w, rb.w, first);
        last = __fmaf_rn(slab_exit<true>(sr, o, R[0], R[3], R[1], R[4], R[2], R[5], rb.w), kWidenExact, sr.eps);
      } else {
        start = slab_box<false>(sr, o, R[0], R[3], R[1], R[4], R[2], R[5], ra.w, rb.w, first);
        last = __fmaf_rn(slab_exit<false>(sr, o, R[0], R[3], R[1], R[4], R[2], R[5], rb.w), kWiden, sr.eps);
      }
      sh.o[0][lane] = o.x; sh.o[1][lane] = o.y; sh.o[2][lane] = o.z;
      sh.inv[0][lane] = sr.inv.x; sh.inv[1][lane] = sr.inv.y; sh.inv[2][lane] = sr.inv.z;
      sh.d[0][lane] = d.x; sh.d[1][lane] = d.y; sh.d[2][lane] = d.z;
      sh.tmin[lane] = ra.w;
      sh.tmax[lane] = rb.w;
    }
    __syncwarp();
    uint32_t found = 0;
    bool open = own;  // the ray's answer is not stored yet
    for (int pass = 0; pass < 2; ++pass) {  // second pass: rays in doubt, one lane each
      uint32_t home = lane, lo = 1u, hi = 0xFFFFFFFFu, place = 0u;  // place: the best hit's
      int node = 0, tp = 0, bot = 0;
      int2 w = load_kd(kd.nodes, 0);  // the node's first two words
      float tMin = first, tMax = last, t_end = last;
      bool walk = start, shared = false;
      uint32_t meetings = 0;
      float best = own ? sh.tmax[lane] : 0.f, bu = 0.f, bv = 0.f;  // any hit: best stays the ray's end
      uint32_t bprim = kMiss;
      if (best < tMin) walk = false;
      for (;;) {
#pragma unroll 1
        for (int k = 0; k < kKdChunk; ++k) {
          if (walk && (w.y & 3) != 3) {
          const int axis = w.y & 3;
          const float split = __int_as_float(w.x), oa = sh.o[axis][home];
          const float tPlane = __fmul_rn(__fsub_rn(split, oa), sh.inv[axis][home]);
          const bool belowFirst = (oa < split) || (oa == split && sh.d[axis][home] <= 0.f);
          const int above = w.y >> 2;
          const int near = belowFirst ? node + 1 : above, far = belowFirst ? above : node + 1;
          const bool skip_far = tPlane > tMax || tPlane <= 0.f, skip_near = !skip_far && tPlane < tMin;
          node = skip_near ? far : near;
          if (!skip_far && !skip_near) {
            if (tp >= kStackSize) {
              atomicOr(err, kErrStackOverflow);
              walk = false;
            } else {
              todo[tp++] = make_int2(far, __float_as_int(tPlane));
              tMax = tPlane;
            }
          }
          w = load_kd(kd.nodes, node);
          }
          __syncwarp();
        }
        // The leaves' primitives, spread over the warp: the leaves' lists laid
        // end to end in lane order, one primitive a lane at a time.
        bool hit = false;
        const uint32_t whole = walk && (w.y & 3) == 3 ? (uint32_t)w.y >> 2 : 0u;
        const uint32_t leaf_n = whole > kKdLeafMax + 1u ? kKdLeafMax : whole;
        uint32_t end = leaf_n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t x = __shfl_up_sync(0xffffffffu, end, o);
          if ((int)lane >= o) end += x;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, end, 31), from = end - leaf_n;
        const uint32_t owners = __ballot_sync(0xffffffffu, leaf_n != 0u);
        if (leaf_n) sh.give[__popc(owners & below)] = lane;
        if constexpr (!ANY) sh.leaf[lane] = ~0ull;
        // equal t: only over a hit from later in the order
        const float bound = !ANY && place > lo ? nextafterf(best, __int_as_float(0x7F800000)) : best;
        unsigned long long mine_leaf = ~0ull;
        uint32_t begun = 0;  // leaves that begin before this batch
        __syncwarp();
#pragma unroll 1
        for (uint32_t batch = 0; batch < total; batch += 32) {
          const uint32_t p = batch + lane, at = from - batch;
          const uint32_t starts = __reduce_or_sync(0xffffffffu, leaf_n && at < 32u ? 1u << at : 0u);
          const bool live = p < total;
          const int src = live ? (int)sh.give[begun + __popc(starts & (below | 1u << lane)) - 1u] : (int)lane;
          begun += __popc(starts);
          const int list = __shfl_sync(0xffffffffu, w.x, src);
          const uint32_t list_n = __shfl_sync(0xffffffffu, leaf_n, src), list_from = __shfl_sync(0xffffffffu, from, src);
          const uint32_t h = __shfl_sync(0xffffffffu, home, src);
          const float bnd = __shfl_sync(0xffffffffu, bound, src);
          float t = 0.f, u = 0.f, v = 0.f;
          uint32_t id = 0;
          bool ok = false;
          if (live) {
            id = (uint32_t)(list_n == 1u ? list : __ldg(kd.prim_idx + list + (p - list_from)));
            const F3 o = {sh.o[0][h], sh.o[1][h], sh.o[2][h]}, d = {sh.d[0][h], sh.d[1][h], sh.d[2][h]};
            if (KIND == kTriangles) {
              const float4* q = kd.prims + 3 * (size_t)id;
              ok = tri_mt(__ldg(q), __ldg(q + 1), __ldg(q + 2), o, d, sh.tmin[h], bnd, t, u, v);
            } else {
              ok = sphere_closest(__ldg(kd.prims + id), o, d, sh.tmin[h], bnd, false, t);
            }
          }
          __syncwarp();
          if (!__any_sync(0xffffffffu, ok)) continue;
          if constexpr (ANY) {
            found |= __reduce_or_sync(0xffffffffu, ok ? 1u << h : 0u);
          } else {
            const float begin = __shfl_sync(0xffffffffu, tMin, src);
            const bool early = ok && shared && t < begin;  // an earlier leaf's
            if (early) atomicMin(&sh.doubt[h], order_key(t));
            // the first of the smallest: list order is p's order, p's lane p & 31
            if (ok && !early) atomicMin(&sh.leaf[src], (unsigned long long)order_key(__fadd_rn(t, 0.f)) << 32 | p);
            __syncwarp();
            const unsigned long long now = sh.leaf[lane];
            const int win = (int)((uint32_t)now & 31u);
            const float nt = __shfl_sync(0xffffffffu, t, win), nu = __shfl_sync(0xffffffffu, u, win);
            const float nv = __shfl_sync(0xffffffffu, v, win);
            const uint32_t nid = __shfl_sync(0xffffffffu, id, win);
            if (now != mine_leaf) {
              mine_leaf = now;
              best = nt; bprim = nid; bu = nu; bv = nv;
              place = shared ? lo : 0u;
              hit = true;
            }
          }
        }
        if (leaf_n != whole) {
          w.x += (int)leaf_n;
          w.y -= (int)(leaf_n << 2);
        } else if (walk && (w.y & 3) == 3) {
          if (tp > bot) {
            const int2 e = todo[--tp];
            node = e.x;
            w = load_kd(kd.nodes, node);
            tMin = __int_as_float(e.y);
            tMax = tp > bot ? __int_as_float(todo[tp - 1].y) : t_end;
            if (best < tMin) walk = false;  // this entry and those below it begin behind the best hit
          } else {
            walk = false;
          }
        }
        __syncwarp();
        if constexpr (ANY) {
          if ((found >> home) & 1u) walk = false;
        } else if (shared && __any_sync(0xffffffffu, hit)) {
          const unsigned long long mine = ((unsigned long long)order_key(__fadd_rn(best, 0.f)) << 32) | place;
          if (hit) atomicMin(&sh.key[home], mine);
          __syncwarp();
          const unsigned long long now = sh.key[home];
          if (hit && now == mine) {  // one piece, one t: one lane
            sh.t[home] = best;
            sh.prim[home] = bprim;
            sh.uv[home] = make_float2(bu, bv);
          }
          best = from_order_key((uint32_t)(now >> 32));
          place = (uint32_t)now;
        }
        const uint32_t busy = __ballot_sync(0xffffffffu, walk);
        if (busy == 0u) break;
        if (++meetings > limit) {
          if (lane == 0) atomicOr(err, kErrCorrupt);
          break;
        }
        if (pass || 32 - __popc(busy) < (grab < 32u ? 1 : kKdIdle)) continue;
        const bool can = walk && tp > bot && hi - lo >= 2u;
        const uint32_t donors = __ballot_sync(0xffffffffu, can);
        if (donors == 0u) continue;
        if constexpr (!ANY) {
          if (!shared) {  // every lane still holds its own ray
            sh.key[lane] = (unsigned long long)order_key(__fadd_rn(best, 0.f)) << 32;  // place 0: before every piece
            sh.doubt[lane] = 0xFFFFFFFFu;
            sh.t[lane] = best;
            sh.prim[lane] = bprim;
            sh.uv[lane] = make_float2(bu, bv);
          }
        }
        shared = true;
        const int pairs = min(__popc(donors), 32 - __popc(busy));
        const int rank = __popc((walk ? donors : ~busy) & below);
        int2 give = make_int2(0, 0);
        float give_end = 0.f;
        uint32_t give_lo = 0, give_hi = 0;
        if (can && rank < pairs) {
          give = todo[bot++];
          give_end = t_end;
          t_end = __int_as_float(give.y);
          give_lo = lo + (hi - lo) / 2 + 1u;
          give_hi = hi;
          hi = give_lo - 1u;
          sh.give[rank] = lane;
        }
        __syncwarp();
        const bool take = !walk && rank < pairs;
        const int src = take ? (int)sh.give[rank] : (int)lane;
        const uint32_t new_home = __shfl_sync(0xffffffffu, home, src);
        give.x = __shfl_sync(0xffffffffu, give.x, src);
        give.y = __shfl_sync(0xffffffffu, give.y, src);
        give_end = __shfl_sync(0xffffffffu, give_end, src);
        give_lo = __shfl_sync(0xffffffffu, give_lo, src);
        give_hi = __shfl_sync(0xffffffffu, give_hi, src);
        const float new_best = __shfl_sync(0xffffffffu, best, src);
        const uint32_t new_place = __shfl_sync(0xffffffffu, place, src);
        if (take) {
          home = new_home;
          best = new_best;
          place = new_place;
          lo = give_lo;
          hi = give_hi;
          node = give.x;
          tMin = __int_as_float(give.y);
          tMax = t_end = give_end;
          tp = bot = 0;
          w = load_kd(kd.nodes, node);
          walk = !(best < tMin);
        }
        __syncwarp();
      }
      if constexpr (!ANY) {
        bool again = false;
        if (shared) {
          __syncwarp();  // the last round's stores; a ballot does not order memory
          const float2 uv = sh.uv[lane];
          best = sh.t[lane];
          bprim = sh.prim[lane];
          bu = uv.x;
          bv = uv.y;
          again = open && sh.doubt[lane] < (uint32_t)(sh.key[lane] >> 32);
        }
        if (open && !again) __stcs(hits + r, make_float4(best, __uint_as_float(bprim), bu, bv));
        open = start = again;
      }
      if (ANY || !__any_sync(0xffffffffu, open)) break;
    }
    if constexpr (ANY) {
      if constexpr (!PLACED) {
        if (lane == 0) occ[base >> 5] = found;
      } else {  // the block's warps put their bits together (grab is 8 or more)
        __shared__ uint32_t bits[4];
        if (lane == 0) bits[threadIdx.x >> 5] = found;
        __syncthreads();
        const uint32_t word = threadIdx.x * gridDim.x + blockIdx.x;
        if (threadIdx.x < grab / 8u && word < (n + 31) / 32) {
          uint32_t w = 0;
          for (uint32_t q = 0; q < 4; ++q)
            for (uint32_t l = 0; l < 8; ++l) w |= ((bits[q] >> (threadIdx.x * 8 + l)) & 1u) << (l << 2 | q);
          occ[word] = w;
        }
      }
    }
    if constexpr (PLACED) break;
  }
}

// Blocks of K (128 threads) resident on the current device at once (asked for
// once per device).
template <auto K>
uint32_t kd_resident_blocks() {
  static std::atomic<uint32_t> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 1;
  uint32_t v = cache[dev & 63].load();
  if (v == 0) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, K, 128, 0) != cudaSuccess || per_sm < 1) per_sm = 1;
    v = (uint32_t)(per_sm * device_sm_count());
    cache[dev & 63].store(v);
  }
  return v;
}

template <int KIND, bool ANY>
void dispatch_kd(int traversal, const KdView& v, uint32_t n_nodes, const float4* rays, uint32_t n, float4* hits,
                 uint32_t* occ, uint32_t* err, uint32_t* work, cudaStream_t s) {
  const unsigned g = (n + 127) / 128;
  if (work) {
    if (traversal == RQ_TRAVERSAL_REFERENCE) {
      cudaMemsetAsync(work, 0, 4, s);
      const uint32_t blocks = kd_resident_blocks<k_trace_kd_warps<KIND, ANY>>();
      k_trace_kd_warps<KIND, ANY><<<std::min(g, blocks), 128, 0, s>>>(v, n_nodes, rays, n, hits, occ, err, work);
      return;
    }
    // fewer rays a warp when there are fewer rays than resident lanes, and no
    // counter when every warp's rays follow from its place, as for the BVH (trace.cu)
    const uint32_t blocks = kd_resident_blocks<k_trace_kd_shared<KIND, ANY, false>>();
    uint32_t grab = 32u;
    while (grab > (ANY ? 8u : 1u) && (uint64_t)blocks * 4 * (grab / 2) >= n) grab /= 2;
    const uint32_t need = (n + 4 * grab - 1) / (4 * grab);
    if (need <= blocks) {
      k_trace_kd_shared<KIND, ANY, true><<<need, 128, 0, s>>>(v, n_nodes, rays, n, hits, occ, err, nullptr, grab);
    } else {
      cudaMemsetAsync(work, 0, 4, s);
      k_trace_kd_shared<KIND, ANY, false><<<blocks, 128, 0, s>>>(v, n_nodes, rays, n, hits, occ, err, work, grab);
    }
  } else if (traversal == RQ_TRAVERSAL_REFERENCE) {
    k_trace_kd<KIND, ANY, true><<<g, 128, 0, s>>>(v, n_nodes, rays, n, hits, occ, err);
  } else {
    k_trace_kd<KIND, ANY, false><<<g, 128, 0, s>>>(v, n_nodes, rays, n, hits, occ, err);
  }
}

__global__ void k_box_union(const float* __restrict__ aabb, uint32_t n, int32_t* lohi) {
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
    for (int a = 0; a < 3; ++a) {
      lo[a] = fminf(lo[a], aabb[6 * (size_t)p + a]);
      hi[a] = fmaxf(hi[a], aabb[6 * (size_t)p + 3 + a]);
    }
  for (int a = 0; a < 3; ++a)
    for (int o = 16; o > 0; o >>= 1) {
      lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
      hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
    }
  if ((threadIdx.x & 31) == 0)
    for (int a = 0; a < 3; ++a) {
      atomicMin(lohi + a, float_to_ordered(lo[a]));
      atomicMax(lohi + 3 + a, float_to_ordered(hi[a]));
    }
}

// Grow a buffer keeping its first `used` bytes.
cudaError_t grow_keep(DevBuf& b, size_t bytes, size_t used, cudaStream_t st) {
  if (bytes <= b.cap && b.p) return cudaSuccess;
  void* p = nullptr;
  size_t want = bytes + bytes / 2 + 256;
  cudaError_t e = cudaMalloc(&p, want);
  if (e != cudaSuccess) return e;
  if (used && b.p) {
    e = cudaMemcpyAsync(p, b.p, used, cudaMemcpyDeviceToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
      cudaFree(p);
      return e;
    }
  }
  if (b.p) cudaFree(b.p);
  b.p = p;
  b.cap = want;
  return cudaSuccess;
}

// Grow a scratch buffer that queued kernels may still read: wait for them
// first (the level loop does not otherwise wait at the end of a level).
cudaError_t ensure_after(DevBuf& b, size_t bytes, cudaStream_t st) {
  if (bytes <= b.cap && b.p) return cudaSuccess;
  const cudaError_t e = cudaStreamSynchronize(st);
  return e != cudaSuccess ? e : b.ensure(bytes);
}

#define KD_TRY(call, what)                                           \
  do {                                                               \
    cudaError_t e_ = (call);                                         \
    if (e_ != cudaSuccess) return BuildResult::cuda_error(e_, what); \
  } while (0)

// Level node arrays carved from one buffer.
LevelNodes carve(char* base, uint32_t cap) {
  LevelNodes L;
  size_t o = 0;
  auto take = [&](size_t bytes) { char* p = base + o; o += (bytes + 255) & ~size_t(255); return p; };
  L.lo = (float4*)take((size_t)cap * 16);
  L.hi = (float4*)take((size_t)cap * 16);
  L.plan = (uint4*)take((size_t)cap * 16);
  L.best = (unsigned long long*)take((size_t)cap * 24);
  L.split = (uint2*)take((size_t)cap * 8);
  L.open = (uint32_t*)take((size_t)cap * 4);
  L.rs = (uint32_t*)take((size_t)cap * 4);
  L.rc = (uint32_t*)take((size_t)cap * 4);
  L.depth = (int32_t*)take((size_t)cap * 4);
  L.bad = (int32_t*)take((size_t)cap * 4);
  L.axis = (int32_t*)take((size_t)cap * 4);
  L.irank = (uint32_t*)take((size_t)cap * 4);
  L.lofs = (uint32_t*)take((size_t)cap * 4);
  return L;
}
size_t level_bytes(uint32_t cap) { return (size_t)cap * 112 + 13 * 256; }

Table table_at(char* base, uint32_t cap) {
  Table T;
  size_t o = 0;
  auto take = [&](size_t bytes) { char* p = base + o; o += (bytes + 255) & ~size_t(255); return p; };
  T.leaf = (int32_t*)take((size_t)cap * 4);
  T.axis = (int32_t*)take((size_t)cap * 4);
  T.split = (float*)take((size_t)cap * 4);
  T.child0 = (uint32_t*)take((size_t)cap * 4);
  T.child1 = (uint32_t*)take((size_t)cap * 4);
  T.count = (uint32_t*)take((size_t)cap * 4);
  T.pool_off = (uint32_t*)take((size_t)cap * 4);
  return T;
}
size_t table_bytes(uint32_t cap) { return (size_t)cap * 28 + 8 * 256; }
uint32_t table_fits(size_t bytes) {  // largest capacity whose table fits
  return bytes < 8 * 256 ? 0u : (uint32_t)std::min<size_t>((bytes - 8 * 256) / 28, 0xFFFFFFF0u);
}

}  // namespace

void launch_trace_kd(int kind, int traversal, bool any, const KdView& v, const float4* rays, uint32_t n,
                     float4* hits, uint32_t* occ, uint32_t* err, cudaStream_t s, uint32_t* work) {
  if (n == 0) return;
  count_launch();
  const uint32_t nn = v.n_nodes;
  if (kind == kTriangles) {
    if (any) dispatch_kd<kTriangles, true>(traversal, v, nn, rays, n, hits, occ, err, work, s);
    else dispatch_kd<kTriangles, false>(traversal, v, nn, rays, n, hits, occ, err, work, s);
  } else {
    if (any) dispatch_kd<kSpheres, true>(traversal, v, nn, rays, n, hits, occ, err, work, s);
    else dispatch_kd<kSpheres, false>(traversal, v, nn, rays, n, hits, occ, err, work, s);
  }
}

BuildResult build_kd_tree(const SceneView& s, int max_depth_cfg, AccelBuffers& a, BuildScratch& sc, uint32_t* err,
                          cudaStream_t st) {
  const uint32_t n = s.n;
  int l2 = 0;
  for (uint32_t v = n; v > 1; v >>= 1) ++l2;
  // maxDepth = round(8 + 1.3 * Log2Int(N)) (accelerators.h:957-958)
  const int depth0 = max_depth_cfg > 0 ? max_depth_cfg : (int)std::round(8 + 1.3f * l2);
  const size_t payload = s.kind == kTriangles ? 48 : 16;
  KD_TRY(a.prims.ensure((size_t)n * payload), "KD payload");
  KD_TRY(a.root.ensure(32), "KD root");
  // primitive boxes (and payload by id)
  KD_TRY(sc.m0.ensure((size_t)n * 24), "KD scratch");
  float* aabb = sc.m0.as<float>();
  launch_prims_by_id(s.kind, s.verts, s.idx, s.sph, n, a.prims.as<float4>(), aabb, st);
  KD_TRY(cudaGetLastError(), "KD prims");
  // root bounds: union of every primitive box
  KD_TRY(sc.lohi.ensure(64), "KD scratch");
  int32_t* lohi = sc.lohi.as<int32_t>();
  launch_init_bounds(lohi, st);
  count_launch();
  k_box_union<<<std::min<uint32_t>(grid(n), 1024u), kThreads, 0, st>>>(aabb, n, lohi);

  // refs of the current level, double buffered: prim, node
  uint32_t R = n, M = 1;
  if (2ull * n >= (1ull << 31)) return BuildResult::error(RQ_ERROR_INVALID_ARGUMENT, "KD tree over 2^30 primitives");
  KD_TRY(sc.m1.ensure((size_t)n * 8 * 2), "KD scratch");
  uint32_t* ref_prim = sc.m1.as<uint32_t>();
  uint32_t* ref_node = ref_prim + (size_t)n;
  // root edge lists, one per axis, each sorted once by t (stable: equal t
  // start-first, then by primitive id), in one set of launches
  const uint32_t E0 = 2 * n;
  KD_TRY(sc.keys.ensure((size_t)E0 * 3 * 16 + 64), "KD edges");
  KD_TRY(sc.vals.ensure((size_t)E0 * 12 * 4 + 64), "KD edges");
  EdgeLists el{sc.keys.as<uint4>(), (size_t)E0};
  {
    const size_t head = 3 * (kSortHistWords + kSortCounterWords), zwords = (head + 3 * sort_status_words(E0, 4) + 1) & ~(size_t)1;
    const uint32_t rtiles = (E0 + kThreads * kRootItems - 1) / (kThreads * kRootItems);
    KD_TRY(sc.m4.ensure(zwords * 4 + (3 * (size_t)rtiles + 2) * 8 + 64), "KD sort");
    uint32_t* zero = sc.m4.as<uint32_t>();
    unsigned long long* rstatus = reinterpret_cast<unsigned long long*>(zero + zwords);
    uint32_t* tk = sc.vals.as<uint32_t>();  // t, v of the three lists, and the sort's other buffers
    uint32_t* tv = tk + 3 * (size_t)E0;
    uint32_t* alt = tv + 3 * (size_t)E0;
    SortScratch ss{alt, alt + 3 * (size_t)E0, zero, zero + head, zero + 3 * kSortHistWords};
    KD_TRY(cudaMemsetAsync(zero, 0, zwords * 4 + (3 * (size_t)rtiles + 2) * 8, st), "KD sort");
    count_launch(2);
    k_root_edges<<<grid(n), kThreads, 0, st>>>(aabb, n, tk, tv, ref_prim, ref_node);
    launch_histogram(tk, E0, 4, zero, st, 3, E0);
    launch_onesweep(tk, tv, E0, 4, ss, err, st, 3, E0);
    k_root_lists<<<dim3(rtiles, 3), kThreads, 0, st>>>(tk, tv, E0, el, rstatus,
                                                       reinterpret_cast<uint32_t*>(rstatus + 3 * (size_t)rtiles), rtiles, err);
    KD_TRY(cudaGetLastError(), "KD root edges");
  }
  // level 0 node
  KD_TRY(sc.m3.ensure(level_bytes(1)), "KD scratch");
  LevelNodes L = carve(sc.m3.as<char>(), 1);
  count_launch();
  k_root_node<<<1, 32, 0, st>>>(L, lohi, a.root.as<float>(), n, depth0);
  KD_TRY(sc.host_words(), "KD scratch");
  uint32_t* h_tot = sc.pinned;
  DevBuf& tabbuf = sc.m5;
  DevBuf& poolbuf = sc.m6;
  uint32_t table_cap = tabbuf.p ? table_fits(tabbuf.cap) : 0, total = 0, pool_used = 0;
  std::vector<uint32_t> level_lo;
  for (int level = 0; M > 0; ++level) {
    if (level > 200) return BuildResult::error(RQ_ERROR_INVALID_ARGUMENT, "KD tree deeper than 200 levels");
    level_lo.push_back(total);
    // table capacity
    if (total + M > table_cap) {
      uint32_t ncap = (total + M) * 2 + 1024;
      DevBuf nb;
      KD_TRY(nb.ensure(table_bytes(ncap)), "KD table");
      if (total) {
        Table Told = table_at(tabbuf.as<char>(), table_cap), Tnew = table_at(nb.as<char>(), ncap);
        const size_t bytes = (size_t)total * 4;
        const void* from[] = {Told.leaf, Told.axis, Told.split, Told.child0, Told.child1, Told.count, Told.pool_off};
        void* to[] = {Tnew.leaf, Tnew.axis, Tnew.split, Tnew.child0, Tnew.child1, Tnew.count, Tnew.pool_off};
        for (int q = 0; q < 7; ++q) {
          const cudaError_t ce = cudaMemcpyAsync(to[q], from[q], bytes, cudaMemcpyDeviceToDevice, st);
          if (ce != cudaSuccess) {
            nb.release();
            return BuildResult::cuda_error(ce, "KD table");
          }
        }
      }
      const cudaError_t ce = cudaStreamSynchronize(st);
      if (ce != cudaSuccess) {
        nb.release();
        return BuildResult::cuda_error(ce, "KD table");
      }
      tabbuf.release();
      tabbuf = nb;
      table_cap = ncap;
    }
    Table T = table_at(tabbuf.as<char>(), table_cap);
    // per-ref sides (R + 1)
    KD_TRY(ensure_after(sc.m2, ((size_t)R + 1) * 8 + 64, st), "KD scratch");
    uint2* sides = sc.m2.as<uint2>();
    // partition scratch: tile counts and the side flags as ballot words
    const uint32_t E2 = 2 * R;
    const uint32_t runs = (E2 + kCostRun - 1) / kCostRun, tiles = (E2 + kEdgeTile - 1) / kEdgeTile;
    const size_t words = ((size_t)E2 + 31) / 32;
    KD_TRY(ensure_after(sc.m4, (size_t)tiles * 3 * 16 + words * 3 * 8 + 64, st), "KD edges");
    unsigned long long* tile_cnt = sc.m4.as<unsigned long long>();
    uint32_t* sideB = reinterpret_cast<uint32_t*>(tile_cnt + (size_t)tiles * 3 * 2);
    uint32_t* sideA = sideB + words * 3;
    // look-back words of the level's two prefix sums and their tickets (cleared by k_cost), totals
    const uint32_t dtiles = (M + kThreads - 1) / kThreads;
    const uint32_t stiles = (R + 1 + kThreads * kSideItems - 1) / (kThreads * kSideItems);
    const uint32_t clear_words = dtiles + stiles + 1;
    KD_TRY(ensure_after(sc.m7, ((size_t)clear_words + 2) * 8 + 64, st), "KD scratch");
    unsigned long long* status = sc.m7.as<unsigned long long>();
    uint32_t* ticket = reinterpret_cast<uint32_t*>(status + dtiles + stiles);
    uint32_t* totals = ticket + 2;
    count_launch(3);
    k_cost<<<grid(std::max<uint64_t>(3ull * runs * 32, 1)), kThreads, 0, st>>>(el, E2, runs, M, L, status, clear_words, err);
    k_decide<<<dtiles, kThreads, 0, st>>>(el, L, M, E2, status, ticket, totals, err);
    k_sides<<<stiles, kThreads, 0, st>>>(ref_prim, ref_node, R, M, aabb, L, sides, status + dtiles, ticket + 1, totals, err);
    KD_TRY(cudaGetLastError(), "KD split");
    KD_TRY(cudaMemcpyAsync(h_tot, totals, 16, cudaMemcpyDeviceToHost, st), "KD level");
    KD_TRY(cudaEventRecord(sc.host_ready, st), "KD level");
    if (E2) {  // needs no totals: runs while the host reads them
      count_launch();
      k_part_count<<<3 * tiles, kThreads, 0, st>>>(el, E2, tiles, R, sides, sideB, sideA, tile_cnt, err);
      if (tiles > kPartSelf) {
        count_launch();
        k_part_scan<<<3, 1024, 0, st>>>(tile_cnt, tiles);
      }
    }
    KD_TRY(cudaEventSynchronize(sc.host_ready), "KD level");
    const uint32_t interiors = h_tot[0], leaf_refs = h_tot[1];
    const uint64_t R2l = (uint64_t)h_tot[2] + h_tot[3];
    if (2 * R2l >= (1ull << 31)) return BuildResult::error(RQ_ERROR_INVALID_ARGUMENT, "KD tree over 2^30 references");
    const uint32_t R2 = (uint32_t)R2l;
    // next level nodes
    const uint32_t M2 = 2 * interiors;
    DevBuf& nextbuf = (level & 1) ? sc.m3 : sc.keys_alt;  // alternate level buffers
    KD_TRY(ensure_after(nextbuf, level_bytes(M2 ? M2 : 1), st), "KD scratch");
    LevelNodes N = carve(nextbuf.as<char>(), M2 ? M2 : 1);
    // leaf pool growth
    KD_TRY(grow_keep(poolbuf, ((size_t)pool_used + leaf_refs + 1) * 4, (size_t)pool_used * 4, st), "KD pool");
    // the next level's nodes and refs (separate buffer), leaf refs to the pool
    KD_TRY(ensure_after(sc.kd_refs, ((size_t)R2 + 1) * 8, st), "KD refs");
    uint32_t* out_prim = sc.kd_refs.as<uint32_t>();
    uint32_t* out_node = out_prim + (R2 + 1);
    count_launch();
    k_spawn_emit<<<grid(std::max(R, M)), kThreads, 0, st>>>(L, M, sides, pool_used, total, total + M, T, N, M2, ref_prim,
                                                            ref_node, R, out_prim, out_node, poolbuf.as<uint32_t>(), R2,
                                                            (uint32_t)(poolbuf.cap / 4), err);
    KD_TRY(cudaGetLastError(), "KD spawn");
    // the children's edge lists
    KD_TRY(ensure_after(sc.vals, (size_t)R2 * 2 * 3 * 16 + 64, st), "KD edges");
    EdgeLists eln{sc.vals.as<uint4>(), (size_t)R2 * 2};
    if (E2 && R2) {
      count_launch();
      const auto part = tiles > kPartSelf ? k_partition<true> : k_partition<false>;
      part<<<3 * tiles, kThreads, 0, st>>>(el, E2, tiles, L, sideB, sideA, tile_cnt, sides, eln, 2 * R2, err);
      KD_TRY(cudaGetLastError(), "KD partition");
    }
    pool_used += leaf_refs;
    total += M;
    std::swap(sc.m1, sc.kd_refs);  // the children's refs become the current refs
    std::swap(sc.keys, sc.vals);   // and their edge lists
    el = EdgeLists{sc.keys.as<uint4>(), (size_t)R2 * 2};
    ref_prim = sc.m1.as<uint32_t>();
    ref_node = ref_prim + (R2 + 1);
    R = R2;
    M = M2;
    L = N;
  }
  // depth-first layout
  level_lo.push_back(total);
  Table T = table_at(tabbuf.as<char>(), table_cap);
  // size, pos, cnt, off: four arrays of total + 2 words
  KD_TRY(ensure_after(sc.m7, ((size_t)total + 2) * 16 + scan_tmp_words((uint64_t)total + 2) * 4 + 64, st), "KD layout");
  uint32_t* size = sc.m7.as<uint32_t>();
  uint32_t* pos = size + (total + 1);
  uint32_t* cnt = pos + (total + 1);
  uint32_t* off = cnt + (total + 1);
  uint32_t* ltmp = off + (total + 2);
  uint32_t* ltot = ltmp + scan_tmp_words((uint64_t)total + 2) + 4;
  const int levels = (int)level_lo.size() - 1;
  for (int hi = levels; hi > 0;) {  // the deepest kLayoutLevels first
    const int d = std::min(hi, kLayoutLevels), lv = hi - d;
    count_launch();
    const auto k = d == 3 ? k_sizes<3> : d == 2 ? k_sizes<2> : k_sizes<1>;
    k<<<grid(level_lo[lv + 1] - level_lo[lv]), kThreads, 0, st>>>(T, level_lo[lv], level_lo[lv + 1], size, total, err);
    hi = lv;
  }
  KD_TRY(cudaMemsetAsync(pos, 0, 4, st), "KD layout");
  for (int lv = 0; lv < levels; lv += kLayoutLevels) {
    count_launch();
    k_positions<<<grid(level_lo[lv + 1] - level_lo[lv]), kThreads, 0, st>>>(T, level_lo[lv], level_lo[lv + 1], size,
                                                                            pos, total);
  }
  count_launch();
  k_leaf_counts<<<grid((uint64_t)total + 1), kThreads, 0, st>>>(T, total, pos, cnt);
  launch_scan_excl(cnt, off, (uint64_t)total + 1, ltmp, ltot, st);
  uint32_t n_idx = 0;
  KD_TRY(cudaMemcpyAsync(&n_idx, ltot, 4, cudaMemcpyDeviceToHost, st), "KD layout");
  KD_TRY(cudaStreamSynchronize(st), "KD layout");
  KD_TRY(a.kd_nodes.ensure((size_t)total * 16), "KD nodes");
  KD_TRY(a.kd_idx.ensure((size_t)(n_idx ? n_idx : 1) * 4), "KD indices");
  count_launch();
  k_write_nodes<<<grid(total), kThreads, 0, st>>>(T, total, pos, off, poolbuf.as<uint32_t>(), a.kd_nodes.as<int4>(),
                                                  a.kd_idx.as<int32_t>(), n_idx, (uint32_t)(poolbuf.cap / 4), err);
  KD_TRY(cudaGetLastError(), "KD write");
  a.n_nodes = total;
  a.n_slots = n_idx;
  a.max_depth = (uint32_t)depth0;
  return {};
}

}  // namespace rq
