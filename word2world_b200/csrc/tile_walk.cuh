// Shared machinery of the per-tile pixel loops (forward blend, both backward
// pixel passes).
//
// A tile is cut into eight 8x4 pixel blocks, one warp each: warp w owns
// columns 8*(w & 1) .. +7, rows 4*(w >> 1) .. +3, lane l its pixel
// (l & 7, l >> 3) inside the block.
#pragma once

#include "common.cuh"

namespace w2w {

constexpr int kRecVec = 3;  // float4s of an entry staged in shared memory

// Pixel of this thread in tile `tile` of a grid `gw` tiles wide.
struct TilePixel {
  int X0, Y0, px, py, warp, lane, bx, by;  // (bx, by): top-left pixel of the warp's block
  // warp: this thread's 8x4 block of the tile (0..7)
  __device__ __forceinline__ TilePixel(int tile, int gw, int block) {
    warp = block;
    lane = threadIdx.x & 31;
    X0 = (tile % gw) * kTile;
    Y0 = (tile / gw) * kTile;
    bx = X0 + kBlockW * (warp & 1);
    by = Y0 + kBlockH * (warp >> 1);
    px = bx + (lane & 7);
    py = by + (lane >> 3);
  }
  __device__ __forceinline__ TilePixel(int tile, int gw) : TilePixel(tile, gw, int(threadIdx.x >> 5)) {}
};

// Tiles are processed heaviest first: CTA b takes tile order[b], where order
// lists the tiles by decreasing weight (tile_order_kernel: the list length
// from `ranges`, or `counts` when given), so the heaviest start in the first
// wave instead of wherever the raster order puts them.
// `zero`, when given, is cleared over num_tiles entries on the way (the
// blend's per-tile maximum, which its CTAs then combine), and `counter`, when
// given, set to zero (the persistent blend's queue).
__global__ void tile_order_kernel(const uint2* ranges, const uint32_t* counts, int num_tiles, uint32_t* order,
                                  uint32_t* zero, uint32_t* counter);

// Block masks the forward blend leaves for the backward passes: for every
// tile and 8x4 block one bit per list position, set when the entry may reach
// the block (block_mask), packed into words of 32 positions counted from the
// tile's first one.  A tile of n entries has 8 rows (one per block) of
// ceil(n / 32) words; its rows start at word mask_row(...), which keeps the
// tiles' regions apart without a prefix over them: a tile's list starts at
// position x, and floor(x / 32) + tile grows by at least ceil(n / 32) from one
// tile to the next.  A state the blend did not write (a replayed list) has the
// binning header's flag clear, and the backward tests every entry itself.
__host__ __device__ __forceinline__ size_t mask_row(uint32_t first, int tile, int n, int block) {
  return 8 * (size_t(first >> 5) + size_t(tile)) + size_t(block) * size_t((n + 31) >> 5);
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src) {
  const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// All but this thread's newest kPending groups of copies have landed (and are
// visible to it).
template <int kPending>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(kPending) : "memory");
}

}  // namespace w2w
