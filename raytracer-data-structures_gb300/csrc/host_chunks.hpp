// The chunks in which a host-buffer query is streamed (host code only).
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

namespace rq {

constexpr uint32_t kPipeChunk = 1u << 21;  // rays per chunk at most: 64 MB up, 32 MB (or 256 KB of bits) down
constexpr uint32_t kPipeMin = 1u << 19;
constexpr uint32_t kPipeHead = 1u << 18;  // smallest first chunk, unless that is a quarter of the rays

// Chunks of a query of n rays, in order: doubling ones where it begins a
// train (nothing is being traced yet: a short first upload), full ones, then
// halving ones where it ends it (nothing follows: a short last traversal and
// download).  None is larger than kPipeChunk, the most a device slot holds,
// and every one but the last is a multiple of 32 rays, so occlusion words
// never straddle chunks.
inline std::vector<uint32_t> chunk_plan(uint32_t n, bool begins, bool ends) {
  std::vector<uint32_t> plan;
  const uint32_t least = std::min(n / 4, std::max(kPipeHead, n / 16)) & ~31u;
  const uint64_t head = std::clamp(least, 32u, kPipeChunk);
  for (uint64_t left = n, size = begins ? head : kPipeChunk; left > 0; size *= 2) {
    size = std::min<uint64_t>(size, kPipeChunk);
    if (ends && left <= 2 * size) size = std::max(head, (left / 2) & ~uint64_t(31));
    const uint64_t take = std::min(size, left);
    plan.push_back((uint32_t)take);
    left -= take;
  }
  return plan;
}

}  // namespace rq
