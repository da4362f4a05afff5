// Median BVH build on the GPU: constructBVHNew (accelerators.h:246-337),
// level by level.
//
// Per node the reference takes the union of the primitive boxes, seeds the
// centroid bounds with it (:275-277), picks the longest axis (:279, GeMaximumAxis
// :190-199), and if the centroids straddle the axis midpoint (:298-311) puts the
// floor(n/2) smallest centroids on the left (std::nth_element, :312-318); a node
// of one primitive is a leaf.  Degenerate nodes (all centroids on one side of
// the midpoint, or a zero-extent axis) become one leaf holding the whole range;
// the reference there keeps a single primitive or recurses without end.  Ties
// at the median are broken by primitive id; the reference leaves them to
// libstdc++'s nth_element.
//
// Method: the primitive ids are sorted once per axis by (centroid, id) with the
// engine's radix sort.  A level is a set of disjoint position ranges
// (segments) shared by the three lists.  Per level, four launches: segment
// boxes; one block for the split decisions, node numbering, parent links and
// the next level's segments; and a stable partition of the three lists (sides
// and tile counts, then the scatter).  The leaves end up as position ranges
// of the x-sorted list, which becomes the slot order.  Internal nodes are
// numbered breadth-first, left before right.  The level counts stay on the
// device (no host round trip per level), and once every segment holds at most
// kFinishSpan primitives the remaining levels of each run inside one block
// (k_finish, in shared memory).
//
// Bound: short launches' latency on small scenes (7 levels of 4 launches on
// 36k spheres), gathers of boxes and centroids by list order on large ones.
// GB300, rebuild of 36k spheres 796 -> 301 us, of a 498k-triangle terrain
// 1568 -> 613 us (first: 13 launches a level and two passes of a serial finish).
#include <algorithm>
#include <atomic>

#include "rq_build.hpp"
#include "rq_device.cuh"

namespace rq {
namespace {

constexpr int kThreads = 256;
constexpr uint32_t kRoot = 0xFFFFFFFFu;

// Ascending float order as unsigned keys; -0 and +0 map to the same key.
__device__ __forceinline__ uint32_t float_key(float f) {
  uint32_t b = __float_as_uint(__fadd_rn(f, 0.0f));
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

struct Segs {
  uint32_t* start;
  uint32_t* end;
  uint32_t* parent;  // node << 1 | side, kRoot for the root
  int32_t* box;      // 6 ordered ints
  uint32_t* half;    // elements on the left when the segment splits, else 0
  uint32_t* dim;
  uint32_t* rank;    // splitting segments before it
  uint32_t* lefts;   // left elements of the segments before it
  uint32_t* skey;    // first right element of the split list: its centroid key
  uint32_t* sid;     // and its primitive
};
constexpr size_t kSegWords = 15;

__global__ void __launch_bounds__(kThreads) k_prim_info(int kind, const float* __restrict__ verts,
                                                        const uint32_t* __restrict__ idx,
                                                        const float4* __restrict__ sph, uint32_t n,
                                                        float* __restrict__ aabb, float* __restrict__ cen,
                                                        uint32_t* __restrict__ keys, int32_t* __restrict__ seg_id,
                                                        Segs top, uint32_t* __restrict__ ctl) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  seg_id[p] = 0;
  if (p == 0) {  // level 0: one segment, the root
    top.start[0] = 0u;
    top.end[0] = n;
    top.parent[0] = kRoot;
    for (int k = 0; k < 3; ++k) { top.box[k] = ordered_pos_inf(); top.box[3 + k] = ordered_neg_inf(); }
    ctl[0] = 1u;
    ctl[1] = 0u;
  }
  float lo[3], hi[3], c[3];
  if (kind == kTriangles) {
    const float* a = verts + 3 * (size_t)__ldg(idx + 3 * (size_t)p);
    const float* b = verts + 3 * (size_t)__ldg(idx + 3 * (size_t)p + 1);
    const float* d = verts + 3 * (size_t)__ldg(idx + 3 * (size_t)p + 2);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      float x = __ldg(a + k), y = __ldg(b + k), z = __ldg(d + k);
      lo[k] = fminf(fminf(x, y), z);
      hi[k] = fmaxf(fmaxf(x, y), z);
      c[k] = __fdiv_rn(__fadd_rn(__fadd_rn(x, y), z), 3.0f);
    }
  } else {
    float4 s = __ldg(sph + p);
    float sc[3] = {s.x, s.y, s.z};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      lo[k] = __fsub_rn(sc[k], s.w);
      hi[k] = __fadd_rn(sc[k], s.w);
      c[k] = sc[k];
    }
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    aabb[6 * (size_t)p + k] = lo[k];
    aabb[6 * (size_t)p + 3 + k] = hi[k];
    cen[3 * (size_t)p + k] = c[k];
    keys[(size_t)k * n + p] = float_key(c[k]);
  }
}

// Segment boxes: one block reduces one slice of kBoundsSlice positions of a
// segment; one slice per segment stores directly, several use atomics (the
// boxes start empty).
constexpr uint32_t kBoundsSlice = kThreads * 8;
__global__ void __launch_bounds__(kThreads) k_seg_bounds(const uint32_t* __restrict__ list0,
                                                         const float* __restrict__ aabb,
                                                         const uint32_t* __restrict__ start,
                                                         const uint32_t* __restrict__ end, const uint32_t* S_dev,
                                                         uint32_t slices, int32_t* __restrict__ box) {
  const uint32_t seg = blockIdx.x / slices, slice = blockIdx.x % slices;
  if (seg >= *S_dev) return;
  const uint32_t s = __ldg(start + seg), e = __ldg(end + seg);
  const uint32_t b = s + slice * kBoundsSlice;
  if (b >= e) return;
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t p = b + threadIdx.x + (uint32_t)(kThreads * k);
    if (p < e) {
      const float2* q = reinterpret_cast<const float2*>(aabb + 6 * (size_t)__ldg(list0 + p));
      const float2 x = __ldg(q), y = __ldg(q + 1), z = __ldg(q + 2);
      lo[0] = fminf(lo[0], x.x); lo[1] = fminf(lo[1], x.y); lo[2] = fminf(lo[2], y.x);
      hi[0] = fmaxf(hi[0], y.y); hi[1] = fmaxf(hi[1], z.x); hi[2] = fmaxf(hi[2], z.y);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    for (int a = 0; a < 3; ++a) {
      lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
      hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
    }
  __shared__ float sm[kThreads / 32][6];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0)
    for (int a = 0; a < 3; ++a) { sm[w][a] = lo[a]; sm[w][3 + a] = hi[a]; }
  __syncthreads();
  if (threadIdx.x < 6) {
    const int a = threadIdx.x;
    float v = sm[0][a];
    for (int q = 1; q < kThreads / 32; ++q) v = a < 3 ? fminf(v, sm[q][a]) : fmaxf(v, sm[q][a]);
    int32_t* bx = box + 6 * (size_t)seg + a;
    if (slices == 1) *bx = float_to_ordered(v);
    else if (a < 3) atomicMin(bx, float_to_ordered(v));
    else atomicMax(bx, float_to_ordered(v));
  }
}

// The split decision of one segment (constructBVHNew's rules), given its
// box and the centroids of its first and last element along each axis (the
// segment's range of that axis' sorted list).  Shared by the level kernel
// and the in-block subtree builder so both decide with the same operations.
// The reference counts the centroids below the midpoint (:298-311) only to
// see whether some but not all are: on the sorted list, whether the first
// is and the last is not (counting them by binary search was 12% of a build).
struct SplitDecision {
  uint32_t split, half, dim;  // half: elements on the left (m / 2) when split
};
__device__ __forceinline__ SplitDecision decide_split(const float* box_lo, const float* box_hi, const float* cfirst,
                                                      const float* clast, uint32_t m) {
  SplitDecision d{0u, 0u, 0u};
  if (m <= 1) return d;
  float lo[3], hi[3];
  for (int a = 0; a < 3; ++a) {
    // centroid bounds seeded with the node bounds (:275-277); the extremes of
    // the centroids along axis a are the ends of that axis' sorted list
    lo[a] = cfirst[a] < box_lo[a] ? cfirst[a] : box_lo[a];
    hi[a] = clast[a] > box_hi[a] ? clast[a] : box_hi[a];
  }
  float ax = __fsub_rn(hi[0], lo[0]), ay = __fsub_rn(hi[1], lo[1]), az = __fsub_rn(hi[2], lo[2]);
  d.dim = (ax > ay && ax > az) ? 0u : (ay > az ? 1u : 2u);
  const float dlo = d.dim == 0 ? lo[0] : d.dim == 1 ? lo[1] : lo[2], dhi = d.dim == 0 ? hi[0] : d.dim == 1 ? hi[1] : hi[2];
  if (dhi != dlo) {
    const float pmid = __fdiv_rn(__fadd_rn(dlo, dhi), 2.0f);
    const float f = d.dim == 0 ? cfirst[0] : d.dim == 1 ? cfirst[1] : cfirst[2];
    const float l = d.dim == 0 ? clast[0] : d.dim == 1 ? clast[1] : clast[2];
    if (f < pmid && !(l < pmid)) {
      d.split = 1;
      d.half = m / 2;
    }
  }
  return d;
}

// Exclusive prefix over the block's threads (blockDim a multiple of 32, at
// most 1024) and the total; tmp: 33 words.
__device__ __forceinline__ unsigned long long block_prefix(unsigned long long v, unsigned long long* tmp,
                                                           unsigned long long& total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  unsigned long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (uint32_t)o) x += y;
  }
  if (lane == 31) tmp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const unsigned long long own = lane < nw ? tmp[lane] : 0ull;
    unsigned long long w = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= (uint32_t)o) w += y;
    }
    tmp[lane] = w - own;
    if (lane == 31) tmp[32] = w;
  }
  __syncthreads();
  const unsigned long long before = tmp[warp];
  total = tmp[32];
  __syncthreads();  // tmp may be reused
  return before + x - v;
}

// One level of segments, one block: the split decisions, the numbering of
// the splitting segments (their nodes, breadth first) and of their left
// elements, the links into the parents' nodes, and the next level's segments
// with empty boxes.  ctl[2 * level] = segments of the level, ctl[2 * level
// + 1] = the level's first node index; the next level's pair is written.
// (Five launches before: decision, three of a scan, links.)
__global__ void __launch_bounds__(1024) k_seg_level(Segs g, uint32_t* ctl, int level, const uint32_t* __restrict__ lists,
                                                    uint32_t n, const float* __restrict__ cen, Segs next,
                                                    float4* __restrict__ nodes, float* __restrict__ root) {
  __shared__ unsigned long long tmp[33];
  const uint32_t S = ctl[2 * level], node_base = ctl[2 * level + 1];
  unsigned long long run = 0;  // splitting segments (high word) and left elements so far
  for (uint32_t k0 = 0; k0 < S; k0 += blockDim.x) {
    const uint32_t k = k0 + threadIdx.x;
    const bool live = k < S;
    uint32_t s = 0, e = 0;
    float lo[3] = {0.f, 0.f, 0.f}, hi[3] = {0.f, 0.f, 0.f};
    SplitDecision d{0u, 0u, 0u};
    if (live) {
      s = g.start[k];
      e = g.end[k];
      float cf[3], cl[3];
      for (int a = 0; a < 3; ++a) {
        lo[a] = ordered_to_float(g.box[6 * (size_t)k + a]);
        hi[a] = ordered_to_float(g.box[6 * (size_t)k + 3 + a]);
        cf[a] = __ldg(cen + 3 * (size_t)lists[(size_t)a * n + s] + a);
        cl[a] = __ldg(cen + 3 * (size_t)lists[(size_t)a * n + e - 1] + a);
      }
      d = decide_split(lo, hi, cf, cl, e - s);
    }
    unsigned long long total;
    const unsigned long long at = run + block_prefix(((unsigned long long)d.split << 32) | d.half, tmp, total);
    run += total;
    if (!live) continue;
    const uint32_t rank = (uint32_t)(at >> 32), node = node_base + rank, mid = s + d.half;
    g.half[k] = d.half;
    g.dim[k] = d.dim;
    g.rank[k] = rank;
    g.lefts[k] = (uint32_t)at;
    const uint32_t pw = g.parent[k];
    if (pw == kRoot) {
      for (int a = 0; a < 3; ++a) { root[a] = lo[a]; root[3 + a] = hi[a]; }
    } else {
      const uint32_t pn = pw >> 1, side = pw & 1u;
      nodes[4 * (size_t)pn + side] = make_float4(lo[0], hi[0], lo[1], hi[1]);
      reinterpret_cast<float2*>(nodes + 4 * (size_t)pn + 2)[side] = make_float2(lo[2], hi[2]);
      int* link = reinterpret_cast<int*>(nodes + 4 * (size_t)pn + 3);
      link[side] = d.split ? (int)node : ~(int)s;
      link[2 + side] = d.split ? 0 : (int)(e - s);
    }
    if (d.split) {
      const uint32_t r = 2 * rank, m = lists[(size_t)d.dim * n + mid];
      g.skey[k] = float_key(__ldg(cen + 3 * (size_t)m + d.dim));
      g.sid[k] = m;
      next.start[r] = s;      next.end[r] = mid;     next.parent[r] = node << 1;
      next.start[r + 1] = mid; next.end[r + 1] = e;  next.parent[r + 1] = (node << 1) | 1u;
      for (int a = 0; a < 3; ++a) {
        next.box[6 * (size_t)r + a] = next.box[6 * (size_t)r + 6 + a] = ordered_pos_inf();
        next.box[6 * (size_t)r + 3 + a] = next.box[6 * (size_t)r + 9 + a] = ordered_neg_inf();
      }
    }
  }
  if (threadIdx.x == 0) {
    ctl[2 * level + 2] = 2 * (uint32_t)(run >> 32);
    ctl[2 * level + 3] = node_base + (uint32_t)(run >> 32);
  }
}

// Stable partition of the three lists inside every splitting segment: an
// element goes left when it precedes the segment's first right element in
// the split list's order (centroid, primitive), so its side needs no table.
// k_part_count takes the sides of a tile of one list (ballot words and the
// tile's left count), k_partition the tile's left elements before it (the
// earlier tiles' counts, or their prefix sum, and the counts inside the tile)
// and scatters.
// (Six launches before: marks, flags, three of a 3n scan, scatter.)
constexpr int kPartItems = 4;  // 8 / 4 / 2: 303 / 301 / 281 us (36k spheres), 2314 / 2303 / 2481 (2.7M triangles)
constexpr uint32_t kPartRun = 32 * kPartItems;               // positions per warp
constexpr uint32_t kPartTile = kPartRun * (kThreads / 32);  // positions per block
// Up to here every block of k_partition adds up its list's earlier tiles
// itself, above a prefix sum of the counts (three launches) does, or the reads
// grow with the square of the primitives.  Rebuild with sums in the blocks /
// with the prefix sum: 2.7M spheres 2765 / 2922 us, 8M 8851 / 8946, 14M 18539 /
// 18470, 30M 48520 / 47380, 60M 114960 / 105740.
constexpr uint32_t kPartSelf = 8192;  // tiles

__global__ void __launch_bounds__(kThreads) k_part_count(Segs g, const int32_t* __restrict__ seg_id,
                                                         const uint32_t* __restrict__ lists, uint32_t n,
                                                         uint32_t tiles, const float* __restrict__ cen,
                                                         uint32_t* __restrict__ sides, uint32_t* __restrict__ counts) {
  __shared__ uint32_t wsum[kThreads / 32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t a = blockIdx.x / tiles, tile = blockIdx.x - a * tiles;
  const uint32_t p0 = tile * kPartTile + warp * kPartRun, words = (n + 31) / 32;
  uint32_t total = 0, v[kPartItems], half[kPartItems], dim[kPartItems];
  int32_t k[kPartItems];
  bool left[kPartItems];
  // loads of all rounds together, one dependent step at a time
#pragma unroll
  for (int j = 0; j < kPartItems; ++j) {
    const uint32_t p = p0 + 32 * j + lane;
    k[j] = p < n ? __ldg(seg_id + p) : -1;
    v[j] = p < n ? __ldg(lists + (size_t)a * n + p) : 0u;
  }
#pragma unroll
  for (int j = 0; j < kPartItems; ++j) {
    half[j] = k[j] >= 0 ? __ldg(g.half + k[j]) : 0u;
    dim[j] = k[j] >= 0 ? __ldg(g.dim + k[j]) : 0u;
  }
#pragma unroll
  for (int j = 0; j < kPartItems; ++j) {
    left[j] = false;
    if (half[j]) {
      if (dim[j] == a) {
        left[j] = p0 + 32 * j + lane < __ldg(g.start + k[j]) + half[j];
      } else {
        const uint32_t c = float_key(__ldg(cen + 3 * (size_t)v[j] + dim[j])), sk = __ldg(g.skey + k[j]);
        left[j] = c < sk || (c == sk && v[j] < __ldg(g.sid + k[j]));
      }
    }
  }
#pragma unroll
  for (int j = 0; j < kPartItems; ++j) {
    const uint32_t m = __ballot_sync(0xffffffffu, left[j]);
    const uint32_t w = (p0 >> 5) + (uint32_t)j;
    if (lane == 0 && w < words) sides[(size_t)a * words + w] = m;
    total += __popc(m);
  }
  if (lane == 0) wsum[warp] = total;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0;
    for (int w = 0; w < kThreads / 32; ++w) t += wsum[w];
    counts[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(kThreads) k_partition(Segs g, const int32_t* __restrict__ seg_id,
                                                        const uint32_t* __restrict__ in, uint32_t n, uint32_t tiles,
                                                        const uint32_t* __restrict__ sides,
                                                        const uint32_t* __restrict__ counts,
                                                        const uint32_t* __restrict__ offs,
                                                        uint32_t* __restrict__ out, int32_t* __restrict__ next_seg) {
  __shared__ uint32_t wsum[kThreads / 32], wleft[kThreads / 32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = (1u << lane) - 1u;
  const uint32_t a = blockIdx.x / tiles, tile = blockIdx.x - a * tiles;
  const uint32_t p0 = tile * kPartTile + warp * kPartRun, words = (n + 31) / 32;
  uint32_t side[kPartItems], mine = 0, before = 0;
#pragma unroll
  for (int j = 0; j < kPartItems; ++j) {
    const uint32_t w = (p0 >> 5) + (uint32_t)j;
    side[j] = w < words ? __ldg(sides + (size_t)a * words + w) : 0u;
    mine += __popc(side[j]);
  }
  if (offs) {  // the counts' prefix sum over all three lists
    if (threadIdx.x == 0) before = __ldg(offs + blockIdx.x) - __ldg(offs + a * tiles);
  } else {
    for (uint32_t t = threadIdx.x; t < tile; t += kThreads) before += __ldg(counts + a * tiles + t);
  }
  before = __reduce_add_sync(0xffffffffu, before);
  if (lane == 0) {
    wsum[warp] = before;
    wleft[warp] = mine;
  }
  __syncthreads();
  uint32_t L = 0;  // left elements of the list before the warp's next 32
  for (uint32_t w = 0; w < kThreads / 32; ++w) L += wsum[w] + (w < warp ? wleft[w] : 0u);
#pragma unroll
  for (int j = 0; j < kPartItems; ++j) {
    const uint32_t p = p0 + 32 * j + lane;
    if (p < n) {
      const uint32_t v = __ldg(in + (size_t)a * n + p);
      const int32_t k = __ldg(seg_id + p);
      const uint32_t half = k >= 0 ? __ldg(g.half + k) : 0u;
      uint32_t np = p;
      int32_t child = -1;
      if (half) {
        const uint32_t s = __ldg(g.start + k), lb = L + __popc(side[j] & lt) - __ldg(g.lefts + k);
        const bool left = (side[j] >> lane) & 1u;
        np = left ? s + lb : s + half + ((p - s) - lb);
        child = (int32_t)(2 * __ldg(g.rank + k)) + (left ? 0 : 1);
      }
      if (np < n) {  // always, while the three lists hold the same sets
        out[(size_t)a * n + np] = v;
        if (a == 0) next_seg[np] = child;
      }
    }
    L += __popc(side[j]);
  }
}

// ---------------------------------------------------------------- small subtrees
// Segments of at most kFinishSpan primitives finish inside one block each:
// the block loads the segment's three sorted lists (as local indices), boxes
// and centroids into shared memory and runs the same levels there, a thread
// for every kFinishSpan / kFinishThreads positions: segment boxes by segmented
// warp reductions and shared atomics, one thread a segment for the decision,
// and the stable partition of the lists by ballots.  Internal nodes are
// numbered breadth first over the whole tree, so the block writes its nodes
// to scratch, numbered breadth first inside the subtree, and counts them per
// level (counts[d * S_bound + b]); an exclusive scan of that level-major
// table gives every subtree's first index at every level, and k_place moves
// the nodes there.  (The block ran twice before, once to count, and gave
// every segment of at most 64 primitives to one thread: 109 us of a
// 36k-sphere build, 65 us now, and 329 us of a 498k-triangle one, 165 now.)
constexpr uint32_t kFinishSpan = 1024;  // 256 / 512 / 1024: 372 / 356 / 336 us (36k spheres), 702 / 643 / 633 (498k triangles)
constexpr int kFinishThreads = 512;
constexpr int kFinishDepth = 14;  // levels of a subtree of kFinishSpan leaves (median halving), with margin
constexpr uint32_t kFinishPer = kFinishSpan / kFinishThreads, kFinishWords = kFinishSpan / 32;
constexpr uint16_t kNoSeg = 0xFFFF;

struct FinishShared {
  uint32_t id[kFinishSpan];                 // global primitive id by local index
  float box[6][kFinishSpan];                // primitive boxes (lo xyz, hi xyz) by local index
  float cen[3][kFinishSpan];                // centroids by local index
  uint16_t list[2][3][kFinishSpan];         // the three sorted lists, local indices, double buffered
  uint16_t seg[2][kFinishSpan];             // segment of every position
  uint8_t left[kFinishSpan];                // side of a primitive in its splitting segment
  uint16_t start[2][kFinishSpan], end[2][kFinishSpan];
  uint32_t parent[2][kFinishSpan];          // local node << 1 | side
  int32_t sbox[6][kFinishSpan];             // segment boxes, ordered ints
  uint16_t half[kFinishSpan], rank[kFinishSpan], lefts[kFinishSpan];
  uint8_t dim[kFinishSpan];
  uint32_t words[3][kFinishWords];          // left elements per 32 positions of each list
  unsigned long long tmp[33];
};

__global__ void __launch_bounds__(kFinishThreads) k_finish(Segs g, const uint32_t* S_dev, uint32_t S_bound,
                                                          uint32_t* lists0, const uint32_t* __restrict__ lists1,
                                                          const uint32_t* __restrict__ lists2,
                                                          const float* __restrict__ aabb, const float* __restrict__ cen,
                                                          uint32_t* loc, uint32_t* counts, float4* __restrict__ local,
                                                          float4* __restrict__ nodes, float* __restrict__ root,
                                                          uint32_t* err) {
  extern __shared__ __align__(16) unsigned char finish_smem[];
  FinishShared& sh = *reinterpret_cast<FinishShared*>(finish_smem);
  const uint32_t b = blockIdx.x, t = threadIdx.x, lane = t & 31u, lt = (1u << lane) - 1u;
  if (b >= *S_dev) return;  // its counts are zero
  const uint32_t s = g.start[b], e = g.end[b], cnt = e - s;
  if (cnt > kFinishSpan) {  // the level loop stops only when every segment fits
    if (t == 0) atomicOr(err, kErrCorrupt);
    return;
  }
  float4* mine = local + 4 * (size_t)s;  // at most cnt - 1 nodes
  for (uint32_t i = t; i < cnt; i += kFinishThreads) {
    const uint32_t gid = lists0[s + i];
    sh.id[i] = gid;
    loc[gid] = i;
    const float2* q = reinterpret_cast<const float2*>(aabb + 6 * (size_t)gid);
    const float2 x = __ldg(q), y = __ldg(q + 1), z = __ldg(q + 2);
    sh.box[0][i] = x.x; sh.box[1][i] = x.y; sh.box[2][i] = y.x;
    sh.box[3][i] = y.y; sh.box[4][i] = z.x; sh.box[5][i] = z.y;
    for (int a = 0; a < 3; ++a) sh.cen[a][i] = __ldg(cen + 3 * (size_t)gid + a);
    sh.list[0][0][i] = (uint16_t)i;
    sh.seg[0][i] = 0;
  }
  if (t == 0) {
    sh.start[0][0] = 0;
    sh.end[0][0] = (uint16_t)cnt;
  }
  __syncthreads();  // loc of this block's ids is visible to the block
  for (uint32_t i = t; i < cnt; i += kFinishThreads) {
    sh.list[0][1][i] = (uint16_t)loc[__ldg(lists1 + s + i)];
    sh.list[0][2][i] = (uint16_t)loc[__ldg(lists2 + s + i)];
  }
  int cb = 0;
  uint32_t nseg = 1, level_base = 0;
  for (int d = 0; nseg > 0; ++d, cb ^= 1) {
    if (d >= kFinishDepth) {
      if (t == 0) atomicOr(err, kErrCorrupt);
      return;
    }
    for (uint32_t j = t; j < nseg; j += kFinishThreads)
      for (int a = 0; a < 3; ++a) {
        sh.sbox[a][j] = ordered_pos_inf();
        sh.sbox[3 + a][j] = ordered_neg_inf();
      }
    __syncthreads();
    // segment boxes: 32 consecutive positions a warp and round
#pragma unroll
    for (uint32_t r = 0; r < kFinishPer; ++r) {
      const uint32_t i = r * kFinishThreads + t;
      const uint32_t k = i < cnt ? sh.seg[cb][i] : kNoSeg;
      int32_t v[6];
      if (k != kNoSeg) {
        const uint32_t x = sh.list[cb][0][i];
        for (int a = 0; a < 6; ++a) v[a] = float_to_ordered(sh.box[a][x]);
      }
      const uint32_t k0 = __shfl_sync(0xffffffffu, k, 0);
      if (__all_sync(0xffffffffu, k == k0)) {
        if (k0 != kNoSeg) {
          for (int a = 0; a < 3; ++a) {
            v[a] = __reduce_min_sync(0xffffffffu, v[a]);
            v[3 + a] = __reduce_max_sync(0xffffffffu, v[3 + a]);
          }
          if (lane == 0)
            for (int a = 0; a < 3; ++a) {
              atomicMin(&sh.sbox[a][k0], v[a]);
              atomicMax(&sh.sbox[3 + a][k0], v[3 + a]);
            }
        }
      } else if (k != kNoSeg) {
        for (int a = 0; a < 3; ++a) {
          atomicMin(&sh.sbox[a][k], v[a]);
          atomicMax(&sh.sbox[3 + a][k], v[3 + a]);
        }
      }
    }
    __syncthreads();
    // decisions, numbering, links, next level's segments
    unsigned long long run = 0;
    for (uint32_t j0 = 0; j0 < nseg; j0 += kFinishThreads) {
      const uint32_t j = j0 + t;
      const bool live = j < nseg;
      uint32_t st = 0, en = 0;
      float lo[3] = {0.f, 0.f, 0.f}, hi[3] = {0.f, 0.f, 0.f};
      SplitDecision dd{0u, 0u, 0u};
      if (live) {
        st = sh.start[cb][j];
        en = sh.end[cb][j];
        float cf[3], cl[3];
        for (int a = 0; a < 3; ++a) {
          lo[a] = ordered_to_float(sh.sbox[a][j]);
          hi[a] = ordered_to_float(sh.sbox[3 + a][j]);
          cf[a] = sh.cen[a][sh.list[cb][a][st]];
          cl[a] = sh.cen[a][sh.list[cb][a][en - 1]];
        }
        dd = decide_split(lo, hi, cf, cl, en - st);
      }
      unsigned long long total;
      const unsigned long long at = run + block_prefix(((unsigned long long)dd.split << 32) | dd.half, sh.tmp, total);
      run += total;
      if (live) {
        const uint32_t rank = (uint32_t)(at >> 32), node = level_base + rank;
        sh.half[j] = (uint16_t)dd.half;
        sh.dim[j] = (uint8_t)dd.dim;
        sh.rank[j] = (uint16_t)rank;
        sh.lefts[j] = (uint16_t)at;
        const uint32_t pw = d == 0 ? g.parent[b] : sh.parent[cb][j];
        if (pw == kRoot) {
          for (int a = 0; a < 3; ++a) { root[a] = lo[a]; root[3 + a] = hi[a]; }
        } else {
          // the subtree's root hangs below a node of the levels above, the rest below local nodes
          float4* into = (d == 0 ? nodes : mine) + 4 * (size_t)(pw >> 1);
          const uint32_t side = pw & 1u;
          into[side] = make_float4(lo[0], hi[0], lo[1], hi[1]);
          reinterpret_cast<float2*>(into + 2)[side] = make_float2(lo[2], hi[2]);
          int* link = reinterpret_cast<int*>(into + 3);
          link[side] = dd.split ? (int)node : ~(int)(s + st);
          link[2 + side] = dd.split ? 0 : (int)(en - st);
        }
        if (dd.split) {
          const uint32_t r = 2 * rank;
          sh.start[cb ^ 1][r] = (uint16_t)st;
          sh.end[cb ^ 1][r] = sh.start[cb ^ 1][r + 1] = (uint16_t)(st + dd.half);
          sh.end[cb ^ 1][r + 1] = (uint16_t)en;
          sh.parent[cb ^ 1][r] = node << 1;
          sh.parent[cb ^ 1][r + 1] = (node << 1) | 1u;
        }
      }
    }
    const uint32_t nsplit = (uint32_t)(run >> 32);
    if (t == 0) counts[(size_t)d * S_bound + b] = nsplit;
    __syncthreads();
    for (uint32_t i = t; i < cnt; i += kFinishThreads) {  // sides, from the split list's order
      const uint32_t k = sh.seg[cb][i];
      if (k != kNoSeg && sh.half[k])
        sh.left[sh.list[cb][sh.dim[k]][i]] = i < (uint32_t)sh.start[cb][k] + sh.half[k] ? 1 : 0;
    }
    __syncthreads();
    uint32_t side[3][kFinishPer];
#pragma unroll
    for (uint32_t r = 0; r < kFinishPer; ++r) {
      const uint32_t i = r * kFinishThreads + t;
      const uint32_t k = i < cnt ? sh.seg[cb][i] : kNoSeg;
      const bool splits = k != kNoSeg && sh.half[k];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        side[a][r] = __ballot_sync(0xffffffffu, splits && sh.left[sh.list[cb][a][i]]);
        if (lane == 0) sh.words[a][i >> 5] = __popc(side[a][r]);
      }
    }
    __syncthreads();
    if (t < 96) {  // exclusive prefix of each list's words, one warp a list
      const uint32_t a = t >> 5, own = lane < kFinishWords ? sh.words[a][lane] : 0u;
      uint32_t x = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
      }
      if (lane < kFinishWords) sh.words[a][lane] = x - own;
    }
    static_assert(kFinishWords <= 32 && kFinishThreads >= 96, "one warp prefixes a list's words");
    __syncthreads();
#pragma unroll
    for (uint32_t r = 0; r < kFinishPer; ++r) {
      const uint32_t i = r * kFinishThreads + t;
      if (i < cnt) {
        const uint32_t k = sh.seg[cb][i];
        const uint32_t half = k != kNoSeg ? sh.half[k] : 0u;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          uint32_t np = i;
          uint16_t child = kNoSeg;
          if (half) {
            const uint32_t st = sh.start[cb][k], lb = sh.words[a][i >> 5] + __popc(side[a][r] & lt) - sh.lefts[k];
            const bool left = (side[a][r] >> lane) & 1u;
            np = left ? st + lb : st + half + ((i - st) - lb);
            child = (uint16_t)(2 * sh.rank[k] + (left ? 0 : 1));
          }
          if (np < cnt) {  // always
            sh.list[cb ^ 1][a][np] = sh.list[cb][a][i];
            if (a == 0) sh.seg[cb ^ 1][np] = child;
          }
        }
      }
    }
    level_base += nsplit;
    nseg = 2 * nsplit;
    __syncthreads();
  }
  for (uint32_t i = t; i < cnt; i += kFinishThreads) lists0[s + i] = sh.id[sh.list[cb][0][i]];
}

// The subtrees' nodes from scratch to their places in the whole tree.
__global__ void __launch_bounds__(kThreads) k_place(Segs g, const uint32_t* S_dev, uint32_t S_bound,
                                                    const uint32_t* __restrict__ counts,
                                                    const uint32_t* __restrict__ offs, const uint32_t* base_dev,
                                                    uint32_t node_cap, const float4* __restrict__ local,
                                                    float4* __restrict__ nodes, uint32_t* err) {
  __shared__ uint32_t first[kFinishDepth + 1], shift[kFinishDepth];  // local index of a level's first node; what its nodes move by
  const uint32_t b = blockIdx.x, t = threadIdx.x;
  if (b >= *S_dev) return;
  if (t < kFinishDepth) {
    uint32_t f = 0;
    for (uint32_t d = 0; d < t; ++d) f += __ldg(counts + (size_t)d * S_bound + b);
    first[t] = f;
    shift[t] = *base_dev + __ldg(offs + (size_t)t * S_bound + b) - f;
    if (t == kFinishDepth - 1) first[kFinishDepth] = f + __ldg(counts + (size_t)t * S_bound + b);
  }
  __syncthreads();
  const uint32_t total = first[kFinishDepth];
  auto place = [&](uint32_t i) {
    uint32_t d = 0;
#pragma unroll
    for (int q = 1; q < kFinishDepth; ++q) d += first[q] <= i ? 1u : 0u;
    return i + shift[d];
  };
  const float4* mine = local + 4 * (size_t)g.start[b];
  for (uint32_t i = t; i < 4 * total; i += kThreads) {
    float4 v = __ldg(mine + i);
    if ((i & 3u) == 3u) {
      const int l = __float_as_int(v.x), r = __float_as_int(v.y);
      if (l >= 0) v.x = __int_as_float((int)place((uint32_t)l));
      if (r >= 0) v.y = __int_as_float((int)place((uint32_t)r));
    }
    const uint32_t at = place(i >> 2);
    if (at >= node_cap) {
      atomicOr(err, kErrCorrupt);  // indices come from the scan of the blocks' counts
      continue;
    }
    nodes[4 * (size_t)at + (i & 3u)] = v;
  }
  if (t == 0 && total && g.parent[b] != kRoot)
    reinterpret_cast<int*>(nodes + 4 * (size_t)(g.parent[b] >> 1) + 3)[g.parent[b] & 1u] = (int)place(0);
}

#define MB_TRY(call, what)                                           \
  do {                                                               \
    cudaError_t e_ = (call);                                         \
    if (e_ != cudaSuccess) return BuildResult::cuda_error(e_, what); \
  } while (0)

Segs segs_at(uint32_t* base, uint32_t cap) {
  Segs g;
  uint32_t** words[] = {&g.start, &g.end, &g.parent, &g.half, &g.dim, &g.rank, &g.lefts, &g.skey, &g.sid};
  for (size_t k = 0; k < 9; ++k) *words[k] = base + k * cap;
  g.box = reinterpret_cast<int32_t*>(base + 9 * (size_t)cap);  // 6 words per segment
  return g;
}

inline unsigned grid(uint64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

}  // namespace

BuildResult build_median_bvh(const SceneView& s, AccelBuffers& a, BuildScratch& sc, uint32_t* err,
                             cudaStream_t st) {
  const uint32_t n = s.n;
  const size_t payload = s.kind == kTriangles ? 48 : 16;
  MB_TRY(a.nodes.ensure((size_t)(n > 1 ? n - 1 : 1) * 64), "BVH nodes");
  MB_TRY(a.prims.ensure((size_t)n * payload), "BVH payload");
  MB_TRY(a.order.ensure((size_t)n * 4), "BVH order");
  MB_TRY(a.root.ensure(32), "BVH root");
  // working memory; the levels above the in-block finish hold segments of
  // more than kFinishSpan primitives and their children: every level's count
  // is at most cap (a power of two of halvings)
  uint32_t cap = 1;
  for (uint32_t size = n; size > kFinishSpan; size = (size + 1) / 2) cap *= 2;
  const uint32_t tiles = (n + kPartTile - 1) / kPartTile;
  MB_TRY(sc.m0.ensure((size_t)n * 9 * 4), "BVH scratch");              // aabb (6) + centroid (3)
  MB_TRY(sc.m1.ensure((size_t)n * 6 * 4), "BVH scratch");              // lists, double buffered
  MB_TRY(sc.m2.ensure((size_t)n * 3 * 4), "BVH scratch");              // sort keys
  const uint64_t cells = 3 * (uint64_t)tiles;
  MB_TRY(sc.m3.ensure(((size_t)((n + 31) / 32) * 3 + 2 * cells + scan_tmp_words(cells) + 8) * 4), "BVH scratch");  // sides, tile counts and their prefix
  MB_TRY(sc.m4.ensure((size_t)n * 8), "BVH scratch");                  // segment of every position, double buffered
  MB_TRY(sc.m5.ensure((size_t)cap * kSegWords * 4), "BVH scratch");    // segments, this level
  MB_TRY(sc.m6.ensure((size_t)cap * kSegWords * 4), "BVH scratch");    // segments, next level
  MB_TRY(sc.vals.ensure((size_t)n * 64), "BVH scratch");               // the subtrees' nodes before they are placed
  float* aabb = sc.m0.as<float>();
  float* cen = aabb + 6 * (size_t)n;
  uint32_t* lists = sc.m1.as<uint32_t>();
  uint32_t* lists_alt = lists + 3 * (size_t)n;
  uint32_t* keys = sc.m2.as<uint32_t>();
  uint32_t* sides = sc.m3.as<uint32_t>();
  uint32_t* tile_counts = sides + 3 * (size_t)((n + 31) / 32);
  uint32_t* tile_offs = tiles > kPartSelf ? tile_counts + cells : nullptr;
  uint32_t* tile_tmp = tile_counts + 2 * cells;
  int32_t* seg_id = sc.m4.as<int32_t>();
  int32_t* next_seg = seg_id + n;
  Segs cur = segs_at(sc.m5.as<uint32_t>(), cap), nxt = segs_at(sc.m6.as<uint32_t>(), cap);

  // Level 0: one segment, the root.  The host runs a fixed number of levels
  // (median splits halve the largest segment) with upper bounds for the
  // segment counts and sizes; the counts themselves and each level's first
  // node index stay on the device (ctl), so the levels run without a host
  // round trip.
  MB_TRY(sc.m7.ensure(2 * 72 * 4), "BVH scratch");
  uint32_t* ctl = sc.m7.as<uint32_t>();
  count_launch();
  k_prim_info<<<grid(n), kThreads, 0, st>>>(s.kind, s.verts, s.idx, s.sph, n, aabb, cen, keys, seg_id, cur, ctl);
  MB_TRY(cudaGetLastError(), "BVH prim info");
  {  // the three lists in one set of launches (12 radix passes one by one were 17% of a small build)
    BuildResult r = sort_pairs(keys, lists, n, 4, true, sc, err, st, 3, n, true);
    if (!r.ok()) return r;
  }
  uint32_t S = 1, max_size = n;  // upper bounds of this level's segments and their sizes
  int level = 0;
  for (;; ++level) {
    if (level > 64) return BuildResult::error(RQ_ERROR_INVALID_ARGUMENT, "median BVH deeper than 64 levels");
    if (max_size <= kFinishSpan) break;  // every segment finishes inside one block
    const uint32_t slices = (max_size + kBoundsSlice - 1) / kBoundsSlice;
    count_launch(4);
    k_seg_bounds<<<S * slices, kThreads, 0, st>>>(lists, aabb, cur.start, cur.end, ctl + 2 * level, slices, cur.box);
    k_seg_level<<<1, S < 1024u ? (S + 31) / 32 * 32 : 1024u, 0, st>>>(cur, ctl, level, lists, n, cen, nxt,
                                                                      a.nodes.as<float4>(), a.root.as<float>());
    k_part_count<<<3 * tiles, kThreads, 0, st>>>(cur, seg_id, lists, n, tiles, cen, sides, tile_counts);
    if (tile_offs) launch_scan_excl(tile_counts, tile_offs, cells, tile_tmp, tile_tmp + scan_tmp_words(cells) + 4, st);
    k_partition<<<3 * tiles, kThreads, 0, st>>>(cur, seg_id, lists, n, tiles, sides, tile_counts, tile_offs, lists_alt,
                                                next_seg);
    MB_TRY(cudaGetLastError(), "BVH level");
    std::swap(lists, lists_alt);
    std::swap(seg_id, next_seg);
    std::swap(cur, nxt);
    S *= 2;
    max_size = (max_size + 1) / 2;
  }
  // The remaining segments (level `level`, at most S, each of at most
  // kFinishSpan primitives): build, scan, place.
  {
    int dev = 0;
    MB_TRY(cudaGetDevice(&dev), "BVH finish");
    static std::atomic<uint64_t> attr_set{0};  // devices whose k_finish allows its shared memory
    const uint64_t bit = 1ull << (dev & 63);
    if (!(attr_set.load() & bit)) {
      MB_TRY(cudaFuncSetAttribute(k_finish, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FinishShared)),
             "BVH finish");
      attr_set.fetch_or(bit);
    }
    const uint64_t cells = (uint64_t)kFinishDepth * S;  // levels x subtrees
    MB_TRY(sc.keys.ensure((2 * cells + scan_tmp_words(cells) + 8) * 4), "BVH scratch");
    uint32_t* counts = sc.keys.as<uint32_t>();
    uint32_t* offs = counts + cells;
    uint32_t* ftmp = offs + cells;
    uint32_t* ftotal = ftmp + scan_tmp_words(cells) + 4;
    const uint32_t* S_dev = ctl + 2 * level;
    const uint32_t* base_dev = ctl + 2 * level + 1;
    MB_TRY(cudaMemsetAsync(counts, 0, cells * 4, st), "BVH finish");
    count_launch(2);
    k_finish<<<S, kFinishThreads, sizeof(FinishShared), st>>>(
        cur, S_dev, S, lists, lists + n, lists + 2 * (size_t)n, aabb, cen, reinterpret_cast<uint32_t*>(next_seg), counts,
        sc.vals.as<float4>(), a.nodes.as<float4>(), a.root.as<float>(), err);
    launch_scan_excl(counts, offs, cells, ftmp, ftotal, st);
    k_place<<<S, kThreads, 0, st>>>(cur, S_dev, S, counts, offs, base_dev, n > 1 ? n - 1 : 1, sc.vals.as<const float4>(),
                                    a.nodes.as<float4>(), err);
    MB_TRY(cudaGetLastError(), "BVH finish");
    MB_TRY(cudaMemcpyAsync(ctl + 2 * 71, ftotal, 4, cudaMemcpyDeviceToDevice, st), "BVH nodes");
  }
  uint32_t h_nodes[2] = {0u, 0u};
  MB_TRY(cudaMemcpyAsync(&h_nodes[0], ctl + 2 * level + 1, 4, cudaMemcpyDeviceToHost, st), "BVH nodes");
  MB_TRY(cudaMemcpyAsync(&h_nodes[1], ctl + 2 * 71, 4, cudaMemcpyDeviceToHost, st), "BVH nodes");
  MB_TRY(cudaStreamSynchronize(st), "BVH nodes");
  const uint32_t node_base = h_nodes[0] + h_nodes[1];
  // slot order = the x-sorted list; gather the payload in that order
  MB_TRY(cudaMemcpyAsync(a.order.p, lists, (size_t)n * 4, cudaMemcpyDeviceToDevice, st), "BVH order");
  launch_prims_gather(s.kind, s.verts, s.idx, s.sph, a.order.as<uint32_t>(), n, a.prims.as<float4>(), st);
  MB_TRY(cudaGetLastError(), "BVH payload");
  a.n_nodes = node_base;
  a.n_slots = n;
  a.max_depth = 0;
  return {};
}

}  // namespace rq
