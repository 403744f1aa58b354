// Document masks of packed sequences, block-wise: the smallest and largest document id of every 64 positions, and the set
// of tiles a CTA has to walk.  Two blocks whose id ranges do not meet hold no visible (query, key) pair, whatever the
// order of the ids; with documents laid out one after the other that leaves the blocks of the same document.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "tile_math.h"

namespace kf {
namespace docblk {

constexpr int ROWS = 64;                       // positions per range
constexpr int MASK_BYTES = 256;                // one bit per tile: up to 2048 tiles
__host__ __device__ constexpr bool fits(int tiles) { return tiles <= MASK_BYTES * 8; }
__host__ __device__ constexpr int n_blocks(int S) { return (S + ROWS - 1) / ROWS; }

// Range over `n` consecutive blocks (those past the end hold nothing).
__device__ __forceinline__ int2 merged(const int2* rg, int n64, int first, int n) {
  int2 r = make_int2(0x7fffffff, -0x7fffffff - 1);
  for (int i = 0; i < n; ++i)
    if (first + i < n64) {
      const int2 v = rg[first + i];
      r.x = min(r.x, v.x);
      r.y = max(r.y, v.y);
    }
  return r;
}

__device__ __forceinline__ tilemath::IdRange ids(int2 r) { return {r.x, r.y}; }

// One bit per tile for which walked(j) holds; called by all threads of the block, which synchronise before the mask is read.
template <typename Walked>
__device__ __forceinline__ void build_mask(uint32_t* mask, int tiles, Walked walked) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  for (int w = warp; w * 32 < tiles; w += warps) {
    const int j = w * 32 + lane;
    const uint32_t bits = __ballot_sync(0xffffffffu, j < tiles && walked(j));
    if (lane == 0) mask[w] = bits;
  }
}

// First set bit at or after j, or `tiles`.
__device__ __forceinline__ int next(const uint32_t* mask, int j, int tiles) {
  while (j < tiles) {
    const uint32_t rest = mask[j >> 5] >> (j & 31);
    if (rest) return j + __ffs(rest) - 1;
    j = (j | 31) + 1;
  }
  return tiles;
}

__device__ __forceinline__ int count(const uint32_t* mask, int tiles) {
  int n = 0;
  for (int w = 0; w * 32 < tiles; ++w) n += __popc(mask[w]);
  return n;
}

}  // namespace docblk
}  // namespace kf
