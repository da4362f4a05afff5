// Stable LSD radix sort of (key, value) pairs, 8-bit digits, one kernel per
// digit pass ("onesweep": local ranking + decoupled look-back across tiles).
// Replaces radixSort (accelerators.h:348-369), which sorts a by-value copy and
// so has no effect: the order produced here is the stable order by key, ties
// in input order, which is what that LSD routine computes.
//
// Per pass and tile of 4,096 keys: keys are ranked stably inside each warp
// (eight ballots give a key's peers), warp counts are prefixed per digit, the
// tile's digit counts are published for later tiles, and each digit's global
// offset is found by walking back over earlier tiles, eight of them a round
// trip (bounded wait; a wait that gives up marks the tile as failed and later
// tiles abort instead of waiting).  Keys are staged in shared memory in digit
// order so the global writes are contiguous runs.
//
// Bound: a pass over a short input is a chain of latencies (tile number, load,
// ranking, look-back, store: about 6 us), over a long one the ranking's
// instructions.  GB300, four passes with histogram and clearing, first
// version (256 threads x 15 keys, __match_any_sync, one predecessor a round
// trip with a sleep between polls) against this one: 36k pairs 66 -> 43 us,
// 82k 68 -> 45, 1M 105 -> 74, 10M 550 -> 405, 40M 1917 -> 1407.  Peers by
// __match_any_sync instead of ballots: 1M 87, 40M 1794.  512 x 8 keys
// measures as 256 x 16 and 512 x 10, 1024 x 4 is slower (1M 97).
#include "rq_device.cuh"
#include "rq_internal.hpp"

namespace rq {
namespace {

constexpr int kThreads = 256;
constexpr uint32_t kFlagAgg = 1u << 30;
constexpr uint32_t kFlagPrefix = 2u << 30;
constexpr uint32_t kFlagAbort = 3u << 30;
constexpr uint32_t kValueMask = (1u << 30) - 1;
constexpr uint32_t kSpinLimit = 1u << 20;  // polls of the same eight predecessors' words before giving up
constexpr int kThreads32 = 512, kItems32 = 8;      // 32-bit keys: tiles of 4,096
constexpr int kThreadsSmall = 256, kItemsSmall = 8;  // short 32-bit sorts: tiles of 2,048
constexpr int kThreads64 = 512, kItems64 = 6;      // 64-bit keys: tiles of 3,072
constexpr uint32_t kSmallSort = 300000;  // 2,048-key tiles up to here: 165k pairs 45 us in 2,048s, 53 in 4,096s; 500k 55 / 53
constexpr uint32_t kStallSpin = 256;       // polls of the test hook's never-set word

template <typename K>
__global__ void __launch_bounds__(kThreads) k_histogram(const K* __restrict__ keys, uint32_t n,
                                                        int passes, uint32_t* __restrict__ hist, size_t stride) {
  __shared__ uint32_t sh[sizeof(K)][256];
  keys += blockIdx.y * stride;
  hist += blockIdx.y * kSortHistWords;
  for (int i = threadIdx.x; i < (int)sizeof(K) * 256; i += blockDim.x) (&sh[0][0])[i] = 0;
  __syncthreads();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    K k = __ldg(keys + i);
    for (int p = 0; p < passes; ++p) atomicAdd(&sh[p][(uint32_t)(k >> (8 * p)) & 255u], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x) {
    uint32_t v = (&sh[0][0])[i];
    if (v) atomicAdd(&hist[i], v);
  }
}

constexpr int kWin = 8;  // predecessors a digit's look-back reads at once

// One pass over one tile of T * I keys, 256 digits.  The staging arrays share
// the warp counts' memory: every key's place in the tile is in a register
// before the first key is staged.
template <typename K, int T, int I>
struct __align__(16) OnesweepSmem {
  static_assert(T >= 256, "one thread per digit");
  static constexpr int kTile = T * I, kW = T / 32;
  union {
    uint32_t warp_hist[kW][256];
    struct {
      K keys[kTile];
      uint32_t vals[kTile];
    } stage;
  };
  uint32_t digit_start[256];
  uint32_t global_base[256];  // digit's global offset of this tile, less digit_start
  unsigned long long scan_tmp[8];
  uint32_t tile;
  int abort;
};

__device__ __forceinline__ uint32_t load_status(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void store_status(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

template <typename K, int T, int I>
__global__ void __launch_bounds__(T) k_onesweep(const K* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                K* __restrict__ kout, uint32_t* __restrict__ vout, uint32_t n,
                                                int shift, const uint32_t* __restrict__ hist, uint32_t* status,
                                                uint32_t* tile_counter, uint32_t* err, const uint32_t* stall,
                                                size_t stride, size_t status_stride) {
  // blockIdx.y: one of several sorts of the same length, `stride` apart
  kin += blockIdx.y * stride;
  if (vin) vin += blockIdx.y * stride;
  kout += blockIdx.y * stride;
  vout += blockIdx.y * stride;
  hist += blockIdx.y * kSortHistWords;
  status += blockIdx.y * status_stride;
  tile_counter += blockIdx.y * kSortCounterWords;
  using Smem = OnesweepSmem<K, T, I>;
  constexpr int kTile = Smem::kTile, kW = Smem::kW;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  if (tid == 0) {
    sm.tile = atomicAdd(tile_counter, 1u);
    sm.abort = 0;
  }
  for (int i = tid; i < kW * 256; i += T) (&sm.warp_hist[0][0])[i] = 0;
  __syncthreads();
  const uint32_t tile = sm.tile;
  const uint64_t base = (uint64_t)tile * kTile;
  const uint32_t valid = (uint64_t)n - base < (uint64_t)kTile ? (uint32_t)(n - base) : (uint32_t)kTile;

  // Warp-striped load: element order (warp, item, lane) = input order.
  const uint32_t first = (uint32_t)warp * (32 * I) + lane;
  K keys[I];
  uint32_t vals[I], rank[I];
#pragma unroll
  for (int k = 0; k < I; ++k) {
    const uint32_t x = first + (uint32_t)k * 32;
    keys[k] = x < valid ? __ldg(kin + base + x) : K(0);
  }
#pragma unroll
  for (int k = 0; k < I; ++k) {
    const uint32_t x = first + (uint32_t)k * 32;
    vals[k] = x < valid ? (vin ? __ldg(vin + base + x) : (uint32_t)base + x) : 0u;
  }

  // Stable rank within the warp, item by item.
#pragma unroll
  for (int k = 0; k < I; ++k) {
    const bool ok = first + (uint32_t)k * 32 < valid;
    const uint32_t d = (uint32_t)(keys[k] >> shift) & 255u;
    uint32_t peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const bool bit = (d >> q) & 1u;
      const uint32_t m = __ballot_sync(0xffffffffu, bit);
      peers &= bit ? m : ~m;
    }
    const uint32_t below = __popc(peers & ((1u << lane) - 1u));
    uint32_t b = 0;
    if (ok && below == 0) {
      b = sm.warp_hist[warp][d];
      sm.warp_hist[warp][d] = b + __popc(peers);
    }
    b = __shfl_sync(0xffffffffu, b, ok ? __ffs(peers) - 1 : lane);
    rank[k] = b + below;
    __syncwarp();
  }
  __syncthreads();

  // Digit t: prefix over warps, tile count, published at once so that later
  // tiles can proceed.
  const uint32_t t = tid;
  uint32_t count = 0, excl = 0;
  unsigned long long scan = 0, own = 0;
  uint32_t* st = status + t;
  if (tid < 256) {
#pragma unroll
    for (int w = 0; w < kW; ++w) {
      const uint32_t c = sm.warp_hist[w][t];
      sm.warp_hist[w][t] = count;
      count += c;
    }
    store_status(st + (size_t)tile * 256, (tile == 0 ? kFlagPrefix : kFlagAgg) | count);
    // exclusive scans of the digit counts, of the whole input (high word)
    // and of the tile (low word), together
    own = ((unsigned long long)__ldg(hist + t) << 32) | count;
    scan = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, scan, o);
      if (lane >= o) scan += y;
    }
    if (lane == 31) sm.scan_tmp[warp] = scan;
  }
  __syncthreads();
  if (tid < 256) {
    unsigned long long before = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) before += w < warp ? sm.scan_tmp[w] : 0ull;
    scan += before - own;
    sm.digit_start[t] = (uint32_t)scan;
  }
  __syncthreads();
  // Every key's place in the tile, then (the counts are read) staging.
#pragma unroll
  for (int k = 0; k < I; ++k) {
    const uint32_t d = (uint32_t)(keys[k] >> shift) & 255u;
    rank[k] += sm.digit_start[d] + sm.warp_hist[warp][d];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < I; ++k) {
    if (first + (uint32_t)k * 32 < valid) {
      sm.stage.keys[rank[k]] = keys[k];
      sm.stage.vals[rank[k]] = vals[k];
    }
  }

  // Decoupled look-back for digit t, kWin predecessors per round trip.
  if (tid < 256) {
    bool failed = false;
    if (tile > 0) {
      // Test hook (stall != null): tile 1 first waits on a word that nothing
      // sets, so its bounded wait gives up as a lost predecessor's would.
      if (stall && tile == 1)
        failed = !spin_until([&] { return *reinterpret_cast<const volatile uint32_t*>(stall) != 0u; }, kStallSpin);
      uint32_t polls = 0;
      for (int32_t j = (int32_t)tile - 1; j >= 0 && !failed;) {
        uint32_t sum = 0;
        bool stop = false, wait = false;
#pragma unroll
        for (int q = 0; q < kWin; ++q) {
          const uint32_t v = j >= q ? load_status(st + (size_t)(j - q) * 256) : kFlagPrefix;
          const uint32_t f = v & ~kValueMask;
          if (stop || wait) continue;
          wait = f == 0u;
          failed = f == kFlagAbort;
          stop = f == kFlagPrefix || failed;
          sum += v & kValueMask;
        }
        if (wait) {  // bounded: back to back at first, then with pauses
          if (++polls > kSpinLimit) failed = true;
          if (polls > 64u) __nanosleep(100);
          continue;
        }
        excl += sum;
        if (stop) break;
        j -= kWin;
        polls = 0;  // the limit is for one window's words
      }
      if (failed) {
        store_status(st + (size_t)tile * 256, kFlagAbort);
        sm.abort = 1;
        atomicOr(err, kErrTimeout);
      } else {
        store_status(st + (size_t)tile * 256, kFlagPrefix | ((excl + count) & kValueMask));
      }
    }
    sm.global_base[t] = (uint32_t)(scan >> 32) + excl - (uint32_t)scan;
  }
  __syncthreads();
  if (sm.abort) return;

#pragma unroll
  for (int k = 0; k < I; ++k) {
    const uint32_t i = tid + (uint32_t)k * T;
    if (i < valid) {
      const K key = sm.stage.keys[i];
      const uint32_t gpos = sm.global_base[(uint32_t)(key >> shift) & 255u] + i;
      if (gpos < n) {
        kout[gpos] = key;
        vout[gpos] = sm.stage.vals[i];
      }
    }
  }
}

// Sorted pairs land back in keys / vals, unless vals_out is given: then the
// final pass's buffers are left as they are and *vals_out names the one that
// holds the sorted values (keys end in the matching key buffer).  count:
// sorts of n pairs each, `stride` pairs apart in every buffer.  identity:
// the values are 0 .. n - 1 and vals need not hold them yet.
template <typename K, int T, int I>
void onesweep_passes(K* keys, uint32_t* vals, uint32_t n, int passes, K* keys_alt, uint32_t* vals_alt,
                     const uint32_t* hist, uint32_t* status, uint32_t* counters, uint32_t* err, cudaStream_t s,
                     uint32_t** vals_out, const uint32_t* stall, uint32_t count, size_t stride, bool identity) {
  using Smem = OnesweepSmem<K, T, I>;
  static_assert(sizeof(Smem) <= 48 * 1024, "onesweep shared memory over the default limit");
  const uint32_t tile = T * I;
  const uint32_t tiles = (n + tile - 1) / tile;
  K* src_k = keys;
  uint32_t* src_v = vals;
  K* dst_k = keys_alt;
  uint32_t* dst_v = vals_alt;
  for (int p = 0; p < passes; ++p) {
    count_launch();
    k_onesweep<K, T, I><<<dim3(tiles, count), T, sizeof(Smem), s>>>(
        src_k, p == 0 && identity ? nullptr : src_v, dst_k, dst_v, n, 8 * p, hist + 256 * p,
        status + (size_t)p * tiles * 256, counters + p, err, p == 0 ? stall : nullptr, stride,
        (size_t)passes * tiles * 256);
    K* tk = src_k; src_k = dst_k; dst_k = tk;
    uint32_t* tv = src_v; src_v = dst_v; dst_v = tv;
  }
  if (vals_out) {
    *vals_out = src_v;
    return;
  }
  if (src_k != keys)
    for (uint32_t c = 0; c < count; ++c) {
      cudaMemcpyAsync(keys + c * stride, src_k + c * stride, (size_t)n * sizeof(K), cudaMemcpyDeviceToDevice, s);
      cudaMemcpyAsync(vals + c * stride, src_v + c * stride, (size_t)n * 4, cudaMemcpyDeviceToDevice, s);
    }
}

void onesweep32(uint32_t* keys, uint32_t* vals, uint32_t n, int passes, const SortScratch& sc, uint32_t* err,
                cudaStream_t s, uint32_t** vals_out, uint32_t count, size_t stride, bool identity) {
  const auto run = n <= kSmallSort ? onesweep_passes<uint32_t, kThreadsSmall, kItemsSmall>
                                   : onesweep_passes<uint32_t, kThreads32, kItems32>;
  run(keys, vals, n, passes, sc.keys_alt, sc.vals_alt, sc.hist, sc.status, sc.counters, err, s, vals_out, sc.stall,
      count, stride, identity);
}

template <typename K>
void histogram(const K* keys, uint32_t n, int passes, uint32_t* hist, cudaStream_t s, uint32_t count, size_t stride) {
  if (n == 0) return;
  uint32_t g = (n + kThreads * 8 - 1) / (kThreads * 8);
  if (g > 2048) g = 2048;
  count_launch();
  k_histogram<K><<<dim3(g, count), kThreads, 0, s>>>(keys, n, passes, hist, stride);
}

}  // namespace

uint32_t sort_tiles(uint32_t n) {
  const uint32_t tile = n <= kSmallSort ? kThreadsSmall * kItemsSmall : kThreads32 * kItems32;
  return (n + tile - 1) / tile;
}

size_t sort_status_words(uint32_t n, int passes) {
  return (size_t)passes * sort_tiles(n) * 256;
}

void launch_histogram(const uint32_t* keys, uint32_t n, int passes, uint32_t* hist, cudaStream_t s, uint32_t count,
                      size_t stride) {
  histogram<uint32_t>(keys, n, passes, hist, s, count, stride);
}

void launch_onesweep(uint32_t* keys, uint32_t* vals, uint32_t n, int passes, const SortScratch& sc,
                     uint32_t* err, cudaStream_t s, uint32_t count, size_t stride, bool identity) {
  if (n <= 1) return;
  onesweep32(keys, vals, n, passes, sc, err, s, nullptr, count, stride, identity);
}

uint32_t* launch_onesweep_vals(uint32_t* keys, uint32_t* vals, uint32_t n, int passes, const SortScratch& sc,
                               uint32_t* err, cudaStream_t s) {
  if (n <= 1) return vals;
  uint32_t* out = vals;
  onesweep32(keys, vals, n, passes, sc, err, s, &out, 1, 0, false);
  return out;
}

size_t sort_status_words64(uint32_t n, int passes) {
  return (size_t)passes * ((n + kThreads64 * kItems64 - 1) / (kThreads64 * kItems64)) * 256;
}

void launch_histogram64(const uint64_t* keys, uint32_t n, int passes, uint32_t* hist, cudaStream_t s) {
  histogram<uint64_t>(keys, n, passes, hist, s, 1, 0);
}

void launch_onesweep64(uint64_t* keys, uint32_t* vals, uint32_t n, int passes, uint64_t* keys_alt,
                       uint32_t* vals_alt, const uint32_t* hist, uint32_t* status, uint32_t* counters,
                       uint32_t* err, cudaStream_t s) {
  if (n <= 1) return;
  onesweep_passes<uint64_t, kThreads64, kItems64>(keys, vals, n, passes, keys_alt, vals_alt, hist, status, counters,
                                                  err, s, nullptr, nullptr, 1, 0, false);
}

}  // namespace rq
