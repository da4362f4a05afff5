// Persistent, work-stealing traversal of many structures in one launch.
//
// Rays of all structures lie back to back; ray_off (n_views + 1 entries)
// gives each structure's range.  The grid is sized to what the SMs hold at
// once; each warp takes 32 consecutive rays (spheres: 64) at a time from a
// global counter until none are left, so long and short structures, coherent and incoherent
// rays share the GPU without a tail per structure.  Each ray finds its
// structure by binary search over ray_off and walks it with the same FAST
// walk as a one-structure query (identical results; the binary walk shares
// the warp's lanes, walk_warp, whose rays may belong to different
// structures).  64 scenes, 8M random rays: closest hit 2798 us with one lane a
// ray, 2230 now, any hit 2271 and 1870 (256 rays per counter access were 9 and
// 6% slower than 32, 64: 6 and 1%); 7 / 8 / 9 blocks of 128 per SM 2327 / 2230 /
// 2359 (closest hit: 9 spill), 1872 at 8 and 1870 at 9 (any hit).  32 scenes of
// 5k spheres, 3.2M random rays, whose walks are short: 32 / 64 / 128 / 256 rays
// a turn 127 / 115 / 116 / 119 us, any hit 118 / 102 / 107 / 109.
//
// Launch shapes (block size, traversal stack depth) are template choices that
// rq_plan_create times on the caller's rays; a stack too shallow for a tree
// reports RQ_ERROR_STACK_OVERFLOW and the tuner drops that shape.
#include "trace_device.cuh"

namespace rq {
namespace {

// UNIT: every structure of the launch has single-primitive leaves (batched
// LBVH builds): 4-byte stack entries.
template <int KIND, bool ANY, int W, int STACK, int BLOCK, bool UNIT = false>
__global__ void __launch_bounds__(BLOCK, W == 2 ? (ANY ? 1152 : 1024) / BLOCK : 1) k_trace_batched(const Bvh2View* __restrict__ views,
                                                         const uint32_t* __restrict__ roff, uint32_t n_views,
                                                         const float4* __restrict__ rays, uint32_t n,
                                                         float4* __restrict__ hits, uint32_t* __restrict__ occ,
                                                         uint32_t* __restrict__ work, uint32_t* err,
                                                         const uint32_t* __restrict__ perm, bool loose) {
  __shared__ WarpShare<ANY, true, UNIT> share[W == 2 ? BLOCK / 32 : 1];
  const uint32_t lane = threadIdx.x & 31;
  constexpr uint32_t kGrab = KIND == kSpheres ? 64u : 32u;  // rays a warp takes at a time
  uint32_t base = 0, taken = kGrab;                         // taken: how many of them it has begun
  uint32_t again = 0;  // closest hits in doubt, walked once more without sharing
  for (;;) {
    if (ANY || again == 0u) {
      if (taken == kGrab) {
        if (lane == 0) base = atomicAdd(work, kGrab);
        base = __shfl_sync(0xffffffffu, base, 0);
        taken = 32u;
      } else {
        base += 32u;
        taken += 32u;
      }
    }
    if (base >= n) return;  // the whole warp leaves together
    const uint32_t w = base + lane;  // work index; the ray itself through perm
    const uint32_t r = (perm && w < n) ? __ldg(perm + w) : w;
    bool occluded = false;
    if constexpr (W == 2) {
      // the warp's rays share its lanes (walk_warp); rays that need the
      // exact box test are walked on their own first
      Bvh2View v{};
      Ray ray = {{0.f, 0.f, 0.f}, {0.f, 0.f, 1.f}, 0.f, 0.f};
      SlabRay sr = {};
      bool walk = w < n && (ANY || again == 0u || (again >> lane & 1u));
      if (walk) {
        v = views[segment_of(roff, n_views, r)];
        ray = load_ray(rays, r);
        sr = slab_ray(ray.o, ray.d);
      }
      Closest c = {ray.tmax, kMiss, 0.f, 0.f};
      bool exact_hit = false;
      if (walk && zero_dir(sr)) {
        uint32_t visits = 0, tests = 0;
        exact_hit = walk_bvh2_form<KIND, ANY, false, STACK, true, UNIT>(v, ray, sr, c, visits, tests, err);
        if (!ANY) store_hit(hits, r, c);
        walk = false;
      }
      __syncwarp();
      const bool own = walk;
      if constexpr (!ANY && KIND == kSpheres) {  // their lanes are their own, and rounds only cost them
        uint32_t visits = 0, tests = 0;
        if (walk) walk_bvh2_form<KIND, ANY, false, STACK, false, UNIT>(v, ray, sr, c, visits, tests, err);
        __syncwarp();
      } else {
        occluded = walk_warp<KIND, ANY, UNIT, STACK, true, true>(v, ray, sr, walk, false, again != 0u || loose, c,
                                                                 share[threadIdx.x >> 5], err);
      }
      if (!ANY && own) store_hit(hits, r, c);
      if (!ANY) again = __ballot_sync(0xffffffffu, own && occluded);
      occluded = occluded || exact_hit;
    } else if (w < n) {
      const Bvh2View v = views[segment_of(roff, n_views, r)];
      const Ray ray = load_ray(rays, r);
      Closest c = {ray.tmax, kMiss, 0.f, 0.f};
      uint32_t visits = 0, tests = 0;
      if (W == 4) {
        const Bvh4View v4{v.nodes, v.prims, v.order, v.root, v.n_internal, v.n_slots};
        occluded = walk_bvh4<KIND, ANY, false, STACK>(v4, ray, c, visits, tests, err);
      } else {
        const Bvh8View v8{v.nodes, v.prims, v.order, v.root, v.n_internal, v.n_slots};
        occluded = walk_bvh8<KIND, ANY, false, STACK>(v8, ray, c, visits, tests, err);
      }
      if (!ANY) store_hit(hits, r, c);
    }
    if (ANY) {
      if (perm) {  // bits of scattered rays: set one by one in the zeroed words
        if (occluded) atomicOr(occ + (r >> 5), 1u << (r & 31));
      } else {
        const uint32_t bits = __ballot_sync(0xffffffffu, occluded);
        if (lane == 0) occ[base >> 5] = bits;
      }
    }
  }
}

template <int KIND, bool ANY, int W, int STACK, int BLOCK>
cudaError_t launch_shape(const BatchedTrace& t, cudaStream_t s) {
  auto k = (W == 2 && t.unit) ? k_trace_batched<KIND, ANY, W, STACK, BLOCK, true>
                              : k_trace_batched<KIND, ANY, W, STACK, BLOCK, false>;
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, BLOCK, 0);
  if (e != cudaSuccess) return e;
  int sms = 0;
  int dev = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  const uint64_t want_warps = ((uint64_t)t.n + 31) / 32;
  uint64_t blocks = (uint64_t)(per_sm > 0 ? per_sm : 1) * sms;
  const uint64_t enough = (want_warps * 32 + BLOCK - 1) / BLOCK;  // no more warps than work blocks
  if (blocks > enough) blocks = enough;
  if (blocks < 1) blocks = 1;
  if ((e = cudaMemsetAsync(t.work, 0, 4, s)) != cudaSuccess) return e;
  if (ANY && t.perm && (e = cudaMemsetAsync(t.occ, 0, (size_t)((t.n + 31) / 32) * 4, s)) != cudaSuccess) return e;
  count_launch();
  k<<<(unsigned)blocks, BLOCK, 0, s>>>(t.views, t.roff, t.n_views, t.rays, t.n, t.hits, t.occ, t.work, t.err,
                                       t.perm, t.loose);
  return cudaGetLastError();
}

// Per-scene ray order keys: (scene << 15) | octant of the direction (3
// bits) | 12-bit Morton code of the origin, quantised to 16 cells per axis in
// the scene's root box.  Sorted stably, rays stay grouped by scene and, within
// a scene, by direction octant and origin cell (the original order within a
// cell).
__device__ __forceinline__ uint32_t spread4(uint32_t v) {  // 4 bits -> every third bit
  v &= 15u;
  return (v & 1u) | ((v & 2u) << 2) | ((v & 4u) << 4) | ((v & 8u) << 6);
}

__global__ void __launch_bounds__(256) k_batch_ray_keys(const Bvh2View* __restrict__ views,
                                                        const uint32_t* __restrict__ roff, uint32_t n_views,
                                                        const float4* __restrict__ rays, uint32_t n,
                                                        uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t sc = segment_of(roff, n_views, i);
  const float* root = views[sc].root;
  const float4 a = __ldg(rays + 2 * (size_t)i), b = __ldg(rays + 2 * (size_t)i + 1);
  const float o[3] = {a.x, a.y, a.z};
  uint32_t q[3];
  for (int k = 0; k < 3; ++k) {
    const float lo = __ldg(root + k), ext = __ldg(root + 3 + k) - lo;
    float u = ext > 0.f ? (o[k] - lo) / ext : 0.f;
    u = fminf(fmaxf(u * 16.f, 0.f), 15.f);
    q[k] = (uint32_t)u;
  }
  const uint32_t oct = (b.x < 0.f ? 4u : 0u) | (b.y < 0.f ? 2u : 0u) | (b.z < 0.f ? 1u : 0u);
  const uint32_t morton = (spread4(q[0]) << 2) | (spread4(q[1]) << 1) | spread4(q[2]);
  keys[i] = (sc << 15) | (oct << 12) | morton;
  vals[i] = i;
}

template <int KIND, bool ANY, int W>
cudaError_t dispatch_shape(const BatchedTrace& t, int block, int deep, cudaStream_t s) {
  constexpr int kShallow = W == 4 ? 48 : W == 8 ? 16 : 32, kDeep = W == 4 ? 96 : W == 8 ? 32 : 64;
  if (block == 256) {
    return deep ? launch_shape<KIND, ANY, W, kDeep, 256>(t, s) : launch_shape<KIND, ANY, W, kShallow, 256>(t, s);
  }
  return deep ? launch_shape<KIND, ANY, W, kDeep, 128>(t, s) : launch_shape<KIND, ANY, W, kShallow, 128>(t, s);
}

template <int KIND, bool ANY>
cudaError_t dispatch_width(const BatchedTrace& t, int block, int deep, cudaStream_t s) {
  if (t.width == 8) return dispatch_shape<KIND, ANY, 8>(t, block, deep, s);
  return t.width == 4 ? dispatch_shape<KIND, ANY, 4>(t, block, deep, s) : dispatch_shape<KIND, ANY, 2>(t, block, deep, s);
}

}  // namespace

int batched_stack_entries(int width, int deep) {
  return width == 4 ? (deep ? 96 : 48) : width == 8 ? (deep ? 32 : 16) : (deep ? 64 : 32);
}

int batch_key_bits(uint32_t n_views) {
  int b = 0;
  while (b < 32 && ((uint64_t)1 << b) < n_views) ++b;
  return 15 + b;
}

void launch_batch_ray_keys(const BatchedTrace& t, uint32_t* keys, uint32_t* vals, cudaStream_t s) {
  if (t.n == 0) return;
  count_launch();
  k_batch_ray_keys<<<(t.n + 255) / 256, 256, 0, s>>>(t.views, t.roff, t.n_views, t.rays, t.n, keys, vals);
}

cudaError_t launch_trace_batched(const BatchedTrace& t, int block, int deep, cudaStream_t s) {
  if (t.n == 0) return cudaSuccess;
  if (block != 128 && block != 256) return cudaErrorInvalidValue;
  if (t.kind == kTriangles)
    return t.any ? dispatch_width<kTriangles, true>(t, block, deep, s) : dispatch_width<kTriangles, false>(t, block, deep, s);
  return t.any ? dispatch_width<kSpheres, true>(t, block, deep, s) : dispatch_width<kSpheres, false>(t, block, deep, s);
}

}  // namespace rq
