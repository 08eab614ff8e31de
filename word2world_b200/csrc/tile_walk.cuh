// Shared machinery of the per-tile pixel loops (forward blend, both backward
// pixel passes).
//
// A tile is cut into eight 8x4 pixel blocks, one warp each: warp w owns
// columns 8*(w & 1) .. +7, rows 4*(w >> 1) .. +3, lane l its pixel
// (l & 7, l >> 3) inside the block.
#pragma once

#include "common.cuh"

namespace w2w {


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
// lists the tiles by decreasing list length (quarter-octave buckets; order
// within a bucket is arbitrary), so the heaviest start in the first wave
// instead of wherever the raster order puts them.  The sort's histogram writes
// it (sort.cu), or a kernel of its own where there is no sort (blend.cu).  The
// backward takes the same order: sorting the tiles again by the
// contributor counts the blend found cost 3 us a view and won nothing (378
// against 383 us of backward per 4 views at 500k, 93 against 90 at 16k).
constexpr int kTileBuckets = 130;
__device__ __forceinline__ int tile_bucket(uint32_t n) {
  if (n == 0) return 0;
  const int e = 31 - __clz(n);
  const uint32_t q = e >= 2 ? (n >> (e - 2)) & 3u : (n << (2 - e)) & 3u;
  return 1 + 4 * e + int(q);
}
// First position of each bucket, the heaviest first, by one warp (32 buckets a step).
__device__ __forceinline__ void bucket_positions(const uint32_t* cnt, uint32_t* pos) {
  const int lane = threadIdx.x & 31;
  uint32_t before = 0;
  for (int b0 = kTileBuckets - 1; b0 >= 0; b0 -= 32) {
    const int b = b0 - lane;
    const uint32_t c = b >= 0 ? cnt[b] : 0u;
    uint32_t x = c;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t o = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += o;
    }
    if (b >= 0) pos[b] = before + x - c;
    before += __shfl_sync(0xffffffffu, x, 31);
  }
}

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

// The reference's Gaussian value (gaussEval.h:7-29) in two halves: the
// mahalanobis numerator, then exp(-0.5 * num / det) with negative distances
// mapped to 1000.
__device__ __forceinline__ float gauss_num(float px, float py, float mx, float my, float cxx, float cxy, float cyy) {
  using namespace fp;
  const float dx = sub(px, mx), dy = sub(py, my);
  const float tX = d2<BL_TX>(dx, cyy, dy, cxy);
  const float tY = s2<BL_TY>(-dx, cxy, dy, cxx);
  return s2<BL_NUM>(tX, dx, tY, dy);
}
__device__ __forceinline__ float gauss_from_m(float m) {
  if (m < 0.0f) m = 1000.0f;
  return expf(mul(-0.5f, m));
}

// The forward's Gaussian values of a lane's entry -- mean (mx, my), covariance
// and determinant c = (cxx, cxy, cyy, det) -- at pixels of the block at
// (bx, by): emit(p, value) for the lane's 32 / kLanes pixels p (a lane per entry
// and 4 / kLanes pixel rows: lane l takes entry l % (32 / kLanes)).  The entry
// stays in registers, so its reciprocal determinant and the per-row and
// per-column products are computed once; a row's pixels go through each stage
// together, so their divisions and exponentials overlap.
//
// Per value the arithmetic is gauss_num's and gauss_from_m's, with the quotient
// by the determinant from div_markstein.  That holds while the variances are in
// [2^-20, 2^20], the determinant's magnitude in [2^-27, 2^20] (the projection drops
// those below 1e-8; a needle's is often lost to cancellation, and then as likely
// below 0) and the mean is not within 2^-12 of a pixel in both coordinates without
// being on it: then a numerator is 0 or above 2^-126 in magnitude (each of its two
// nested sums of products cancels to no less than 2^-47 of its terms) and below
// 2^72, its quotient neither underflows nor overflows and keeps its sign, and one
// too small for div_markstein's range (2^-60) still gives exp(-quotient / 2) = 1.
// Any other entry is evaluated with the IEEE division, pixel by pixel, which took
// 606 us a 512x512 render of 50k needles when half of them fell to it.
template <int kLanes, typename Emit>
__device__ __forceinline__ void gauss_values(float mx, float my, float4 c, float bx, float by, Emit&& emit) {
  constexpr int kRows = 4 / kLanes;
  const int r0 = (int(threadIdx.x & 31u) / (32 / kLanes)) * kRows;
  const float fx = fabsf(mx - rintf(mx)), fy = fabsf(my - rintf(my));
  auto in = [](float v) { return v >= 0x1p-20f && v <= 0x1p20f; };
  if (fabsf(c.w) >= 0x1p-27f && fabsf(c.w) <= 0x1p20f && in(c.x) && in(c.z) && fabsf(mx) <= 0x1p24f && fabsf(my) <= 0x1p24f &&
      (fmaxf(fx, fy) >= 0x1p-12f || fmaxf(fx, fy) == 0.0f)) {
    const float y = rcp_markstein(c.w);
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      float num[8], g[8];
#pragma unroll
      for (int col = 0; col < 8; ++col)
        num[col] = gauss_num(bx + float(col), by + float(r0 + r), mx, my, c.x, c.y, c.z);
#pragma unroll
      for (int col = 0; col < 8; ++col) num[col] = div_markstein_y(num[col], c.w, y);
#pragma unroll
      for (int col = 0; col < 8; ++col) g[col] = expf(mul(-0.5f, num[col]));
#pragma unroll
      for (int col = 0; col < 8; ++col) emit(8 * (r0 + r) + col, num[col] < 0.0f ? 0.0f : g[col]);
    }
  } else {
#pragma unroll 1
    for (int p = 8 * r0; p < 8 * (r0 + kRows); ++p) {
      const float num = gauss_num(bx + float(p & 7), by + float(p >> 3), mx, my, c.x, c.y, c.z);
      emit(p, gauss_from_m(div(num, c.w)));
    }
  }
}

}  // namespace w2w
