// Backward pass.
//
// Per-pixel pass (reference backward.cu:521-665): one warp, and one CTA, per 8x4
// pixel block, its pixels walking the tile's list back to front, recomputing each
// pair's alpha from the stored state (final transmittance and last-contributor
// index) instead of storing per-pair values.  Each entry's sums over the block's
// pixels are formed by its own lane and added with one atomic each (the reference
// issues ten atomics per pixel-Gaussian pair).  A block starts at its pixels'
// largest contributor count: entries past it are skipped by every pixel.
//
// Per-Gaussian pass: the reference's computeCov2DCUDA (backward.cu:27-227) and
// backwardPreprocessingKernel (backward.cu:229-519) fused into one thread per
// Gaussian.
//
// grad_mode 0 reproduces the reference's formulas, including where they are
// not the derivative of its forward (+0.3 on the 2-D covariance, a 1.3*tan box
// clamp, colour-clamp masks, SH_C2[2] = 0.3154 and all 16 SH bands).  grad_mode
// 1 is the exact derivative of the forward: the pair set is re-derived with the
// forward's own Gaussian evaluation and the forward's final transmittance.
#include "common.cuh"
#include "kernels.h"
#include "tile_walk.cuh"

#include <cfloat>
#include <type_traits>

namespace w2w {
namespace {

// ---------------------------------------------------------------------------
// Per-pixel pass.  One warp, and one CTA, per 8x4 pixel block, walking its
// block's part of the tile's list back to front, the entries its block mask
// names packed into groups of 32:
//
//   1. lane j gathers entry j's record (the next group's loads are in flight
//      while this one is worked on) and evaluates it at the block's 32 pixels:
//      alpha and Gaussian value of every pair, 0 where the pair is skipped,
//      into two 32 x 32 tables;
//   2. every lane runs its pixel through the group's entries in order -- the
//      transmittance chain, which needs no decisions: a skipped pair's alpha is
//      0 -- and puts two numbers per pair in their place: u, from which every
//      geometric gradient of the pair follows, and w, its colour weight;
//   3. lane j sums entry j over the block's 32 pixels (the moments of u over the
//      pixel offsets, and w times each upstream plane), turns the sums into the
//      entry's gradients and adds each with one atomic.
//
// A group of up to 16 (8) entries spreads steps 1 and 3 over two (four) lanes
// per entry.
//
// What bounds it: instruction issue, and for scenes that leave SMs idle the
// busiest warp's chain.  About 20 + 18 + 13 instructions per entry in the three
// steps.  A shuffle tree per entry (ten values through 21 shuffles per pair of
// entries, with their products computed per pixel) cost about 60 for step 3
// alone; evaluating the pairs in step 2, four entries at a time, left the
// busiest warps waiting for each one's exponential and reciprocal (119 us
// against 96 per view at 500k / 512x512, 30 against 23 at 16k / 256x256).
// One-warp CTAs give a block's slot back when it ends; an eight-warp CTA held
// its registers until the slowest of its blocks had ended.  Cutting the
// heaviest tiles' walks into segments, each replaying the chain behind it, no
// longer pays: a replay costs steps 1 and 2, three quarters of the work (470
// us per 4 views at 500k without, 678 with half an SM count of tiles cut).
//
// A skipped pair's zeros keep it out of the chain and the sums by
// multiplication, as long as all that they meet is finite.  kSelect: they are
// left out by selection (a pair's w is 0 only where it was skipped), for blocks
// whose view has a value that is not tame (GeomHeader::wild) or whose pixels
// have such an upstream gradient.  A whole walk is compiled either way: a test
// per group of entries instead, its loops the same, cost 1 to 3 % of a step (1M
// Gaussians 1364 -> 1385 us, a batch of six scenes 1012 -> 1040).
// ---------------------------------------------------------------------------
constexpr int kGroup = 32;        // entries per group
constexpr int kSteps = 8;         // of them in flight through a pixel's chain
constexpr int kWindow = 512;      // list positions whose mask bits are expanded together, 16 per lane
constexpr int kTableStride = 36;  // floats per pixel row: rows start on 16 bytes, 8 rows cover the banks

// A warp's shared memory.
struct __align__(16) BwdWarp {
  float alpha[32 * kTableStride];  // [pixel of the block][entry of the group]: alpha, then w
  float value[32 * kTableStride];  // the Gaussian value, then u
  float4 up[32];                   // per pixel: upstream dL/dcolour and dL/ddepth
  float4 dc[kGroup];               // per entry: depth and colour
  uint32_t last[32];               // per pixel: contributor count
  uint32_t queue[kWindow + kGroup];  // list positions waiting, highest first: under a group, and one window's
};

// Positions [lo, top) of a block's part of a tile's list, highest first, in
// groups of up to 32.  words: the block's mask row, or null (each entry is
// tested against the block here).  A lane expands 16 positions' bits of a
// window at the offset a scan over the lanes gives it: about 80 instructions
// per 512 positions, where taking the words one by one cost 40 per 32 and was
// the longest walks' largest part (91k of 222k cycles).
template <bool kWide>
struct BlockWalk {
  const uint32_t* words;
  const float* record;
  const uint32_t* list;   // the tile's first list entry
  uint32_t num_records;
  int bx, by, lo, top, window, head, tail;
  uint32_t ahead;  // the lane's mask word of the next window to expand

  // Window w's mask word of this lane (two lanes share one).
  __device__ __forceinline__ uint32_t load(int w) const {
    const int lane = threadIdx.x & 31;
    const int i = w * (kWindow / 32) + (lane >> 1);
    if (words != nullptr) return w >= (lo >> 9) && 32 * i < top ? __ldg(words + i) : 0u;
    uint32_t mine = 0u;
    for (int k = 0; k < kWindow / 32 && w >= (lo >> 9); ++k) {
      const int pos = kWindow * w + 32 * k + lane;
      bool reach = false;
      if (pos >= lo && pos < top) {
        const uint32_t id = __ldg(list + pos);
        if (id < num_records) {
          float4 r0, r1;  // the blend's record
          ldg32<kWide>(record + 16 * size_t(id), r0, r1);
          reach = block_test(r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, bx, by);
        }
      }
      const uint32_t b = __ballot_sync(0xffffffffu, reach);
      if ((lane >> 1) == k) mine = b;
    }
    return mine;
  }
  __device__ __forceinline__ void start(int lo_, int top_) {
    static_assert(kWindow == 512, "window index");
    lo = lo_;
    top = top_;
    head = tail = 0;
    window = top > lo ? (top - 1) >> 9 : -1;
    ahead = window >= 0 ? load(window) : 0u;
  }
  // Queues positions until a group waits or none are left; returns the next
  // group's size (its positions: queue[head, head + size)).  Warp-collective;
  // the caller has synchronised the warp after its last read of the queue.
  __device__ __forceinline__ int fill(uint32_t* queue) {
    const int lane = threadIdx.x & 31;
    while (tail - head < kGroup && window >= 0 && window >= (lo >> 9)) {
      if (head > 0) {  // what waits moves to the front
        const uint32_t v = head + lane < tail ? queue[head + lane] : 0u;
        __syncwarp();
        queue[lane] = v;
        tail -= head;
        head = 0;
        __syncwarp();
      }
      const int base = kWindow * window + 16 * lane;
      uint32_t bits = (lane & 1) ? ahead >> 16 : ahead & 0xffffu;
      if (top - base < 16) bits &= top > base ? (1u << (top - base)) - 1u : 0u;
      if (lo - base > 0) bits &= lo - base < 16 ? 0xffffffffu << (lo - base) : 0u;
      --window;
      ahead = window >= 0 ? load(window) : 0u;
      int n = __popc(bits), from = n;  // from: this lane's bits and those of the lanes above
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_down_sync(0xffffffffu, from, d);
        if (lane + d < 32) from += o;
      }
      int at = tail + from - n;
      while (bits != 0u) {
        const int b = 31 - __clz(bits);
        queue[at++] = uint32_t(base + b);
        bits ^= 1u << b;
      }
      tail += __shfl_sync(0xffffffffu, from, 0);
    }
    __syncwarp();
    return min(tail - head, kGroup);
  }
};

// A group in flight: the lane's entry.
struct GroupLoad {
  float4 q0, q1, q2;  // Chain::gather's
  uint32_t id = ~0u, pos = ~0u;
  int count = 0;
};

// Pixel-loop prologue shared by both modes: this thread's pixel, its
// upstream gradients and contributor count, the warp's walk length.
struct BwdPixel {
  int tile;
  TilePixel tp;
  bool inside;
  size_t pix;
  uint2 range;
  int walk;  // list positions [0, walk) may hold contributors of this warp's pixels
  uint32_t last;
  float dLp0 = 0.f, dLp1 = 0.f, dLp2 = 0.f, dLd = 0.f, dLa = 0.f;
  int W, H;         // this tile's image size
  const float* bg;
  __device__ __forceinline__ BwdPixel(const BackwardArgs& a, int tile_, int local_tile, int block, int W_, int H_,
                                      size_t pbase, const float* bg_)
      : tile(tile_), tp(local_tile, (W_ + kTile - 1) / kTile, block), W(W_), H(H_), bg(bg_) {
    inside = tp.px < W && tp.py < H;
    range = a.ranges[tile];
    const size_t hw = size_t(W) * H;
    pix = inside ? pbase + size_t(tp.py) * W + tp.px : 0;
    last = inside ? a.n_contrib[pix] : 0u;
    walk = int(min(__reduce_max_sync(0xffffffffu, last), range.y - range.x));
    if (inside) {
      // colour planes: an image's three planes sit together at 3 * pbase
      const size_t cp = 3 * pbase + (pix - pbase);
      dLp0 = a.dL_dcolor[cp];
      dLp1 = a.dL_dcolor[hw + cp];
      dLp2 = a.dL_dcolor[2 * hw + cp];
      dLd = a.dL_ddepth != nullptr ? a.dL_ddepth[pix] : 0.f;  // absent: no loss on depth / alpha
      dLa = a.dL_dalpha != nullptr ? a.dL_dalpha[pix] : 0.f;
    }
  }
};

// The reference's pair test and Gaussian value: power from the conic, skipped
// when positive or below alpha 1/255, alpha = min(0.99, o G).  q0 = (mx, my,
// conic a, conic b), q1 = (conic c, opacity, _, _).  The roundings of the
// power are written out, so that a pair at a threshold is decided the same
// whatever the compiler shares between the pixels of a row or a column: one
// decided differently changes every gradient behind it by 1/255.
__device__ __forceinline__ bool ref_eval(float4 q0, float4 q1, float pxf, float pyf, float& G, float& alpha) {
  const float dx = sub(q0.x, pxf), dy = sub(q0.y, pyf);
  const float quad = fma(mul(q0.z, dx), dx, mul(mul(q1.x, dy), dy));
  const float power = fma(-0.5f, quad, -mul(mul(q0.w, dx), dy));
  G = expf(power);
  alpha = fminf(0.99f, mul(q1.y, G));
  return power <= 0.0f && alpha >= 1.0f / 255.0f;
}

// The ten (nine without a depth loss) sums of an entry over its lanes' pixels.
constexpr int kSums = 10;
template <int kLanes>
__device__ __forceinline__ void combine_lanes(float (&v)[kSums]) {
#pragma unroll
  for (int d = 32 / kLanes; d < 32; d <<= 1)
#pragma unroll
    for (int k = 0; k < kSums; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], d);
}

// Nothing to add: mostly an entry that no pixel of the block took.  Each sum
// counts: the others may cancel (a Gaussian centred between two pixels under an
// upstream gradient of opposite signs has a mean gradient and nothing else).
__device__ __forceinline__ bool all_zero(const float (&v)[kSums]) {
  bool zero = true;
#pragma unroll
  for (int k = 0; k < kSums; ++k) zero = zero && v[k] == 0.f;
  return zero;
}

// Reference formulas (backward.cu:552-663) for one pixel; entries (mx, my,
// conic a, conic b), (conic c, opacity, depth, r), (g, b, _, _).
// The reference keeps the colour, depth and alpha composited behind the current
// entry per channel and multiplies their differences by the upstream planes;
// the chain is linear in them, so one number serves: B, the upstream-weighted
// composite behind the entry.  kDA: a loss reaches depth or alpha.
template <bool kDA>
struct RefChain {
  float T, B = 0.f, tf_bg;  // tf_bg: T_final times (background . upstream colour)
  __device__ __forceinline__ RefChain(const BackwardArgs& a, const BwdPixel& p) {
    const float tf = p.inside ? 1.0f - a.out_alpha[p.pix] : 0.0f;
    T = tf;
    tf_bg = tf * (p.bg[0] * p.dLp0 + p.bg[1] * p.dLp1 + p.bg[2] * p.dLp2);
  }
  template <bool kWide>
  static __device__ __forceinline__ void gather(const BackwardArgs& a, GroupLoad& g) {
    const float* r = a.bwd_record + 16 * size_t(g.id);
    ldg32<kWide>(r, g.q0, g.q1);
    g.q2 = __ldg(reinterpret_cast<const float4*>(r) + 2);
  }
  static __device__ __forceinline__ float4 depth_colour(const GroupLoad& g) {
    return make_float4(g.q1.z, g.q1.w, g.q2.x, g.q2.y);
  }
  template <int kLanes>
  static __device__ __forceinline__ void evaluate(BwdWarp& s, const GroupLoad& g, float bx, float by) {
    constexpr int kEntries = 32 / kLanes, kRows = 4 / kLanes;
    const int lane = int(threadIdx.x & 31u), e = lane % kEntries, r0 = (lane / kEntries) * kRows;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const uint4 l0 = *reinterpret_cast<const uint4*>(s.last + 8 * (r0 + r));
      const uint4 l1 = *reinterpret_cast<const uint4*>(s.last + 8 * (r0 + r) + 4);
      const uint32_t last[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        float G, alpha;
        const bool ok = ref_eval(g.q0, g.q1, bx + float(c), by + float(r0 + r), G, alpha) && g.pos < last[c];
        const int at = (8 * (r0 + r) + c) * kTableStride + e;
        s.alpha[at] = ok ? alpha : 0.f;
        s.value[at] = ok ? G : 0.f;
      }
    }
  }

  // kSteps entries of the pixel's chain: alphas and values become w and u.  T
  // in [~1e-4, 1] (the forward stops before T < 1e-4) and 1 - alpha in [0.01,
  // 1]: T / (1 - alpha) from the correctly rounded reciprocal and one remainder
  // correction; exactly T where alpha is 0.
  template <bool kSelect>
  __device__ __forceinline__ void steps(const BwdPixel& p, const float4* dc, float (&alpha)[kSteps],
                                        float (&value)[kSteps]) {
    float q[kSteps], y[kSteps];
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
      const float4 c = dc[k];
      q[k] = c.y * p.dLp0 + c.z * p.dLp1 + c.w * p.dLp2;
      if constexpr (kDA) q[k] += c.x * p.dLd + p.dLa;
      y[k] = rcp_markstein(1.f - alpha[k]);
    }
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
      const float t = T * y[k];
      T = fma(fma(-(1.f - alpha[k]), t, T), y[k], t);
      const float d = q[k] - B;
      const bool skip = kSelect && alpha[k] == 0.f;
      B = skip ? B : B + alpha[k] * d;
      value[k] = skip ? 0.f : value[k] * (d * T - tf_bg * y[k]);
      alpha[k] *= T;
    }
  }

  // The lane's entry over its pixels, and its atomics.
  template <int kLanes, bool kSelect>
  static __device__ __forceinline__ void reduce(const BackwardArgs& a, const BwdWarp& s, const GroupLoad& g, float bx,
                                                float by, float hW, float hH) {
    constexpr int kEntries = 32 / kLanes, kRows = 4 / kLanes;
    const int lane = int(threadIdx.x & 31u), e = lane % kEntries, r0 = (lane / kEntries) * kRows;
    float S = 0.f, Sx = 0.f, Sy = 0.f, Sxx = 0.f, Sxy = 0.f, Syy = 0.f, c0 = 0.f, c1 = 0.f, c2 = 0.f, cd = 0.f;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const float dy = g.q0.y - (by + float(r0 + r));
      float rs = 0.f, rx = 0.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int px = 8 * (r0 + r) + c;
        const float u = s.value[px * kTableStride + e], w = s.alpha[px * kTableStride + e];
        if (kSelect && w == 0.f) continue;
        const float4 up = s.up[px];
        const float dx = g.q0.x - (bx + float(c)), t = u * dx;
        rs += u;
        rx += t;
        Sxx += t * dx;
        c0 += w * up.x;
        c1 += w * up.y;
        c2 += w * up.z;
        if constexpr (kDA) cd += w * up.w;
      }
      S += rs;
      Sx += rx;
      Sxy += dy * rx;
      const float t = dy * rs;
      Sy += t;
      Syy += t * dy;
    }
    float v[kSums] = {S, Sx, Sy, Sxx, Sxy, Syy, c0, c1, c2, cd};
    combine_lanes<kLanes>(v);
    if (lane >= g.count || g.id >= uint32_t(a.P)) return;
    if (all_zero(v)) return;
    const float A = g.q0.z, B = g.q0.w, C = g.q1.x, o = g.q1.y, h = -0.5f * o;
    const size_t id = g.id;
    atomicAdd(a.dL_dcolors + 3 * id, v[6]);
    atomicAdd(a.dL_dcolors + 3 * id + 1, v[7]);
    atomicAdd(a.dL_dcolors + 3 * id + 2, v[8]);
    if constexpr (kDA) atomicAdd(a.acc_depth + id, v[9]);
    atomicAdd(a.dL_dmean2D + 3 * id, -o * hW * (A * v[1] + B * v[2]));
    atomicAdd(a.dL_dmean2D + 3 * id + 1, -o * hH * (C * v[2] + B * v[1]));
    atomicAdd(a.acc_cov + 4 * id, h * v[3]);
    atomicAdd(a.acc_cov + 4 * id + 1, h * v[4]);
    atomicAdd(a.acc_cov + 4 * id + 3, h * v[5]);
    atomicAdd(a.dL_dopacity + id, v[0]);
  }
};

// Exact derivative of the forward blend for one pixel; entries (mx, my, opacity,
// _), (cxx, cxy, cyy, det), (depth, r, g, b).  The suffix sums behind the
// current entry (colour including the background, depth, weight) enter only
// through their upstream-weighted sum D.
struct ExactChain {
  float T, D;
  __device__ __forceinline__ ExactChain(const BackwardArgs& a, const BwdPixel& p) {
    T = p.inside ? a.T_final[p.pix] : 0.0f;
    D = T * (p.bg[0] * p.dLp0 + p.bg[1] * p.dLp1 + p.bg[2] * p.dLp2);
  }
  template <bool kWide>
  static __device__ __forceinline__ void gather(const BackwardArgs& a, GroupLoad& g) {
    const float* r = a.record + 16 * size_t(g.id);
    float4 o;
    ldg32<kWide>(r, g.q0, o);
    g.q0.z = o.w;
    ldg32<kWide>(r + 8, g.q1, g.q2);
  }
  static __device__ __forceinline__ float4 depth_colour(const GroupLoad& g) { return g.q2; }
  // The forward's own Gaussian values and decisions; the value is 0 where
  // alpha is clamped to 0.99, past which no gradient goes.
  template <int kLanes>
  static __device__ __forceinline__ void evaluate(BwdWarp& s, const GroupLoad& g, float bx, float by) {
    const int e = int(threadIdx.x & 31u) % (32 / kLanes);
    gauss_values<kLanes>(g.q0.x, g.q0.y, g.q1, bx, by, [&](int p, float v) {
      const float og = mul(g.q0.z, v), al = fminf(0.99f, og);  // 0.99 for NaN (an infinite opacity times 0)
      const bool ok = al >= 1.0f / 255.0f && g.pos < s.last[p];
      s.alpha[p * kTableStride + e] = ok ? al : 0.f;
      s.value[p * kTableStride + e] = ok && og < 0.99f ? v : 0.f;
    });
  }
  template <bool kSelect>
  __device__ __forceinline__ void steps(const BwdPixel& p, const float4* dc, float (&alpha)[kSteps],
                                        float (&value)[kSteps]) {
    float q[kSteps], ia[kSteps];
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
      const float4 c = dc[k];
      q[k] = c.y * p.dLp0 + c.z * p.dLp1 + c.w * p.dLp2 + c.x * p.dLd + p.dLa;
      ia[k] = rcp_markstein(1.0f - alpha[k]);  // 1 - alpha in [0.01, 1]
    }
#pragma unroll
    for (int k = 0; k < kSteps; ++k) {
      T *= ia[k];  // transmittance in front of this entry
      const bool skip = kSelect && alpha[k] == 0.f;
      value[k] = skip ? 0.f : value[k] * (q[k] * T - D * ia[k]);
      alpha[k] *= T;
      D = skip ? D : D + q[k] * alpha[k];
    }
  }

  // With e = cyy dx - cxy dy and f = cxx dy - cxy dx (offsets from the mean),
  // d(num / det) = 2 (e, f) / det over the offsets and -(e e, 2 e f, f f) / det^2
  // over the covariance.
  template <int kLanes, bool kSelect>
  static __device__ __forceinline__ void reduce(const BackwardArgs& a, const BwdWarp& s, const GroupLoad& g, float bx,
                                                float by, float hW, float hH) {
    constexpr int kEntries = 32 / kLanes, kRows = 4 / kLanes;
    const int lane = int(threadIdx.x & 31u), en = lane % kEntries, r0 = (lane / kEntries) * kRows;
    float S = 0.f, Se = 0.f, Sf = 0.f, See = 0.f, Sef = 0.f, Sff = 0.f, c0 = 0.f, c1 = 0.f, c2 = 0.f, cd = 0.f;
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
      const float dy = (by + float(r0 + r)) - g.q0.y, ey = -g.q1.y * dy, fy = g.q1.x * dy;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int px = 8 * (r0 + r) + c;
        const float u = s.value[px * kTableStride + en], w = s.alpha[px * kTableStride + en];
        if (kSelect && w == 0.f) continue;
        const float4 up = s.up[px];
        const float dx = (bx + float(c)) - g.q0.x;
        const float e = g.q1.z * dx + ey, f = fy - g.q1.y * dx;
        const float te = u * e, tf = u * f;
        S += u;
        Se += te;
        Sf += tf;
        See += te * e;
        Sef += te * f;
        Sff += tf * f;
        c0 += w * up.x;
        c1 += w * up.y;
        c2 += w * up.z;
        cd += w * up.w;
      }
    }
    float v[kSums] = {S, Se, Sf, See, Sef, Sff, c0, c1, c2, cd};
    combine_lanes<kLanes>(v);
    if (lane >= g.count || g.id >= uint32_t(a.P)) return;
    if (all_zero(v)) return;
    // |det| >= 1e-8 (the projection drops a smaller one): rcp_markstein's rounding
    // depends on the significand alone while det, its approximate reciprocal and
    // the remainder are normal numbers, so this is the correctly rounded 1/det.
    // An infinite opacity is clamped at every pixel: the geometric sums are 0.
    const float idet = rcp_markstein(g.q1.w), k1 = (fabsf(g.q0.z) <= FLT_MAX ? g.q0.z : 0.f) * idet, k2 = k1 * idet;
    const size_t id = g.id;
    atomicAdd(a.dL_dcolors + 3 * id, v[6]);
    atomicAdd(a.dL_dcolors + 3 * id + 1, v[7]);
    atomicAdd(a.dL_dcolors + 3 * id + 2, v[8]);
    atomicAdd(a.acc_depth + id, v[9]);
    atomicAdd(a.dL_dmean2D + 3 * id, k1 * hW * v[1]);
    atomicAdd(a.dL_dmean2D + 3 * id + 1, k1 * hH * v[2]);
    atomicAdd(a.acc_cov + 4 * id, 0.5f * k2 * v[3]);
    atomicAdd(a.acc_cov + 4 * id + 1, k2 * v[4]);
    atomicAdd(a.acc_cov + 4 * id + 2, 0.5f * k2 * v[5]);
    atomicAdd(a.dL_dopacity + id, v[0]);
  }
};

// Pixel-loop prologue for block `block` of tile `tile`: the call's image, or
// its batch item's.
__device__ __forceinline__ BwdPixel make_bwd_pixel(const BackwardArgs& a, int tile, int block) {
  if (a.items == nullptr) return BwdPixel(a, tile, tile, block, a.W, a.H, 0, a.bg);
  const BatchItem& it = a.items[find_item_tile(a.items, a.num_items, uint32_t(tile))];
  return BwdPixel(a, tile, tile - int(it.tile_base), block, it.W, it.H, size_t(it.pix_base), it.bg);
}

template <typename Chain, bool kWide>
__global__ void __launch_bounds__(32, 16) render_bwd_kernel(BackwardArgs a) {
  grid_wait();
  __shared__ BwdWarp s;
  const int tile = int(a.order[blockIdx.x / 8]);  // heaviest first
  const int lane = int(threadIdx.x), block = int(blockIdx.x) % 8;
  const BwdPixel p = make_bwd_pixel(a, tile, block);
  if (p.walk <= 0) return;
  s.up[lane] = make_float4(p.dLp0, p.dLp1, p.dLp2, p.dLd);
  s.last[lane] = p.last;
  Chain ch(a, p);
  const float bx = float(p.tp.bx), by = float(p.tp.by);
  const float hW = 0.5f * float(p.W), hH = 0.5f * float(p.H);
  const uint32_t* list = a.point_list + p.range.x;
  BlockWalk<kWide> walk;
  // the blend's block masks, when this binning state has them
  const bool use_masks = a.masks_valid != nullptr && *a.masks_valid != 0u;
  walk.words = use_masks ? a.masks + mask_row(p.range.x, tile, int(p.range.y - p.range.x), block) : nullptr;
  walk.record = a.record;
  walk.list = list;
  walk.num_records = uint32_t(a.P);
  walk.bx = p.tp.bx;
  walk.by = p.tp.by;

  // The next group's positions and ids (the lanes' entries as the chain's
  // evaluate spreads them).  An id of num_records or more -- a list left
  // inconsistent by a sort whose bounded wait ran out, which its error word
  // reports -- is skipped, never read.
  auto pack = [&](GroupLoad& g) {
    __syncwarp();
    g.count = walk.fill(s.queue);
    const int e = g.count > 16 ? lane : g.count > 8 ? lane & 15 : lane & 7;
    g.pos = e < g.count ? s.queue[walk.head + e] : ~0u;  // past every pixel's last contributor
    walk.head += g.count;
    g.id = e < g.count ? __ldg(list + g.pos) : ~0u;
  };
  auto gather = [&](GroupLoad& g) {
    // opacity 0, in gauss_values' range: contributes nothing
    g.q0 = make_float4(-1024.f, -1024.f, 0.f, 0.f);
    g.q1 = make_float4(1.f, 0.f, 1.f, 1.f);
    g.q2 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (g.id < uint32_t(a.P)) Chain::template gather<kWide>(a, g);
    else g.pos = ~0u;
  };
  auto run = [&](auto select) {
    constexpr bool kSelect = decltype(select)::value;
    walk.start(0, p.walk);
    GroupLoad g, next;
    pack(g);
    gather(g);
    if (g.count > 0) pack(next);
    while (g.count > 0) {
      const int count = g.count;
      if (count > 16) Chain::template evaluate<1>(s, g, bx, by);
      else if (count > 8) Chain::template evaluate<2>(s, g, bx, by);
      else Chain::template evaluate<4>(s, g, bx, by);
      s.dc[lane] = Chain::depth_colour(g);
      GroupLoad after;
      gather(next);                     // the next group's records and
      if (next.count > 0) pack(after);  // the ids of the one after it are in flight below
      __syncwarp();
      float* al = s.alpha + lane * kTableStride;
      float* va = s.value + lane * kTableStride;
      for (int e = 0; e < count; e += kSteps) {
        float4* xa = reinterpret_cast<float4*>(al + e);
        float4* xv = reinterpret_cast<float4*>(va + e);
        const float4 a0 = xa[0], a1 = xa[1], v0 = xv[0], v1 = xv[1];
        float x[kSteps] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        float v[kSteps] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
        ch.template steps<kSelect>(p, s.dc + e, x, v);
        xa[0] = make_float4(x[0], x[1], x[2], x[3]);
        xa[1] = make_float4(x[4], x[5], x[6], x[7]);
        xv[0] = make_float4(v[0], v[1], v[2], v[3]);
        xv[1] = make_float4(v[4], v[5], v[6], v[7]);
      }
      __syncwarp();
      if (count > 16) Chain::template reduce<1, kSelect>(a, s, g, bx, by, hW, hH);
      else if (count > 8) Chain::template reduce<2, kSelect>(a, s, g, bx, by, hW, hH);
      else Chain::template reduce<4, kSelect>(a, s, g, bx, by, hW, hH);
      __syncwarp();
      g = next;
      next = after;
    }
  };
  const bool plain = *a.wild == 0u && tame(p.dLp0) && tame(p.dLp1) && tame(p.dLp2) && tame(p.dLd) && tame(p.dLa) &&
                     tame(p.bg[0]) && tame(p.bg[1]) && tame(p.bg[2]);
  if (__all_sync(0xffffffffu, plain)) run(std::false_type{});
  else run(std::true_type{});
}

// ---------------------------------------------------------------------------
// Per-Gaussian passes: one thread per Gaussian, with the SH rows (up to 48
// floats each) moved between global and shared memory by the whole warp, so
// that global loads and stores are contiguous 128-byte runs instead of one
// 192-byte-strided row per thread.
// ---------------------------------------------------------------------------
constexpr int kGaussThreads = 128;
constexpr int kGaussRow = 52;  // floats of shared memory per Gaussian (store_rows; the staged rows need 49)

__device__ __forceinline__ int sh_stride(int M) {
  const int r = 3 * (M < 16 ? M : 16);
  return r | 1;
}

// Rows [i0, i0 + n) of shs ([P, M, 3]), first min(M, 16) coefficients, into
// s (row g at g * stride).  Warp-collective.
__device__ __forceinline__ void sh_stage_in(const float* shs, int M, int i0, int n, float* s, int stride) {
  constexpr int kInFlight = 8;  // loads issued before their stores
  const int rs = 3 * (M < 16 ? M : 16), rg = 3 * M, lane = threadIdx.x & 31;
  if (M == 16 && n == 32 && aligned16(shs)) {
    stage_span(shs + size_t(i0) * 48, 48, s, stride, 0);
    __syncwarp();
    return;
  }
  if (rs > 0) {
    const int total = n * rs;
    int g = 0, c = lane;
    while (c >= rs) { c -= rs; ++g; }
    for (int e0 = 0; e0 < total; e0 += 32 * kInFlight) {
      float v[kInFlight];
      int dst[kInFlight];
#pragma unroll
      for (int k = 0; k < kInFlight; ++k) {
        const bool ok = e0 + 32 * k + lane < total;
        v[k] = ok ? __ldg(shs + size_t(i0 + g) * rg + c) : 0.f;
        dst[k] = ok ? g * stride + c : -1;
        c += 32;
        while (c >= rs) { c -= rs; ++g; }
      }
#pragma unroll
      for (int k = 0; k < kInFlight; ++k)
        if (dst[k] >= 0) s[dst[k]] = v[k];
    }
  }
  __syncwarp();
}

// 32 rows of dL/dSH (48 floats each) of 16-byte aligned arrays: each lane puts
// its products into s, and the warp writes them out as contiguous 16-byte
// pieces, without the index arithmetic of a lane per output element.  s holds
// 32 rows of 52 floats (an odd number of 16-byte pieces), which start at
// conflict-free banks.
__device__ __forceinline__ void store_rows(float* dsh, float* s, const float (&basis)[16], const float (&cf)[3],
                                           bool active) {
  const int lane = threadIdx.x & 31;
  float4* s4 = reinterpret_cast<float4*>(s);
#pragma unroll
  for (int q = 0; q < 12; ++q) {
    float o[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) o[w] = active ? basis[(4 * q + w) / 3] * cf[(4 * q + w) % 3] : 0.f;
    s4[13 * lane + q] = make_float4(o[0], o[1], o[2], o[3]);
  }
  __syncwarp();
  float4* dst = reinterpret_cast<float4*>(dsh);
#pragma unroll
  for (int q = 0; q < 12; ++q) {
    const int f = 32 * q + lane, g = f / 12;
    dst[f] = s4[f + g];  // piece f % 12 of row g at 13 g
  }
}

// The same for the raw path's arrays: rows of 3 and of 45 floats, both odd, lie
// in s as they lie in memory.
__device__ __forceinline__ void store_rows_raw(float* ddc, float* dac, float* s, const float (&basis)[16],
                                               const float (&cf)[3], bool active) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) s[3 * lane + ch] = active ? basis[0] * cf[ch] : 0.f;
#pragma unroll
  for (int e = 0; e < 45; ++e) s[kRawAc + 45 * lane + e] = active ? basis[1 + e / 3] * cf[e % 3] : 0.f;
  __syncwarp();
  const float4* s4 = reinterpret_cast<const float4*>(s);
  if (lane < 24) reinterpret_cast<float4*>(ddc)[lane] = s4[lane];
  float4* dst = reinterpret_cast<float4*>(dac);
#pragma unroll
  for (int q = 0; q < 12; ++q)
    if (32 * q + lane < 360) dst[32 * q + lane] = s4[kRawAc / 4 + 32 * q + lane];
}

// dsh rows [i0, i0 + n) ([P, M, 3]) = basis[k] * cf[ch] (k < 16; 0 beyond),
// written contiguously; each thread's factors pass through s.  Warp-collective.
__device__ __forceinline__ void sh_store_outer(float* dsh, int M, int i0, int n, float* s, const float (&basis)[16],
                                               const float (&cf)[3], bool active) {
  constexpr int kRow = 21;  // 16 basis + 3 colour factors, odd stride
  const int lane = threadIdx.x & 31, rg = 3 * M;
  __syncwarp();  // the SH rows in s have been read
  if (M == 16 && n == 32 && aligned16(dsh)) {
    store_rows(dsh + size_t(i0) * 48, s, basis, cf, active);
    return;
  }
#pragma unroll
  for (int k = 0; k < 16; ++k) s[lane * kRow + k] = active ? basis[k] : 0.f;
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) s[lane * kRow + 16 + ch] = active ? cf[ch] : 0.f;
  __syncwarp();
  if (rg > 0) {
    constexpr int kInFlight = 8;
    const int total = n * rg;
    int g = 0, c = lane;
    while (c >= rg) { c -= rg; ++g; }
    for (int e0 = 0; e0 < total; e0 += 32 * kInFlight) {
      float v[kInFlight];
      size_t dst[kInFlight];
#pragma unroll
      for (int q = 0; q < kInFlight; ++q) {
        const int k = c / 3, ch = c - 3 * k;
        const bool ok = e0 + 32 * q + lane < total;
        v[q] = ok && k < 16 ? s[g * kRow + k] * s[g * kRow + 16 + ch] : 0.f;
        dst[q] = ok ? size_t(i0 + g) * rg + c : ~size_t(0);
        c += 32;
        while (c >= rg) { c -= rg; ++g; }
      }
#pragma unroll
      for (int q = 0; q < kInFlight; ++q)
        if (dst[q] != ~size_t(0)) dsh[dst[q]] = v[q];
    }
  }
}

// The raw path's SH rows: coefficient 0 from sh_dc ([P, 1, 3]), the rest from
// sh_ac ([P, M - 1, 3]).  Same staging as sh_stage_in.  Warp-collective.
// Returns true for full rows that are on their way asynchronously as they lie in
// memory (sh_ac only, 45 floats a row): copy_wait and a warp barrier complete
// them.
__device__ __forceinline__ bool sh_stage_in_raw(const float* dc, const float* ac, int M, int i0, int n, float* s,
                                                int stride) {
  constexpr int kInFlight = 8;
  const int rs = 3 * (M < 16 ? M : 16), ra = 3 * (M - 1), lane = threadIdx.x & 31;
  if (M == 16 && n == 32 && aligned16(ac)) {
    copy_span_async(s, ac + size_t(i0) * 45, 32 * 45);
    return true;
  }
  if (rs > 0) {
    const int total = n * rs;
    int g = 0, c = lane;
    while (c >= rs) { c -= rs; ++g; }
    for (int e0 = 0; e0 < total; e0 += 32 * kInFlight) {
      float v[kInFlight];
      int dst[kInFlight];
#pragma unroll
      for (int k = 0; k < kInFlight; ++k) {
        const bool ok = e0 + 32 * k + lane < total;
        v[k] = !ok ? 0.f : c < 3 ? __ldg(dc + size_t(i0 + g) * 3 + c) : __ldg(ac + size_t(i0 + g) * ra + (c - 3));
        dst[k] = ok ? g * stride + c : -1;
        c += 32;
        while (c >= rs) { c -= rs; ++g; }
      }
#pragma unroll
      for (int k = 0; k < kInFlight; ++k)
        if (dst[k] >= 0) s[dst[k]] = v[k];
    }
  }
  __syncwarp();
  return false;
}

// sh_store_outer for the raw path: coefficient 0 to ddc, the rest to dac.
__device__ __forceinline__ void sh_store_outer_raw(float* ddc, float* dac, int M, int i0, int n, float* s,
                                                   const float (&basis)[16], const float (&cf)[3], bool active) {
  constexpr int kRow = 21;
  const int lane = threadIdx.x & 31, rg = 3 * M, ra = 3 * (M - 1);
  __syncwarp();  // the SH rows in s have been read
  if (M == 16 && n == 32 && aligned16(ddc) && aligned16(dac)) {
    store_rows_raw(ddc + size_t(i0) * 3, dac + size_t(i0) * 45, s, basis, cf, active);
    return;
  }
#pragma unroll
  for (int k = 0; k < 16; ++k) s[lane * kRow + k] = active ? basis[k] : 0.f;
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) s[lane * kRow + 16 + ch] = active ? cf[ch] : 0.f;
  __syncwarp();
  if (rg > 0) {
    constexpr int kInFlight = 8;
    const int total = n * rg;
    int g = 0, c = lane;
    while (c >= rg) { c -= rg; ++g; }
    for (int e0 = 0; e0 < total; e0 += 32 * kInFlight) {
      float v[kInFlight];
      float* dst[kInFlight];
#pragma unroll
      for (int q = 0; q < kInFlight; ++q) {
        const int k = c / 3, ch = c - 3 * k;
        const bool ok = e0 + 32 * q + lane < total;
        v[q] = ok && k < 16 ? s[g * kRow + k] * s[g * kRow + 16 + ch] : 0.f;
        dst[q] = !ok ? nullptr : c < 3 ? ddc + size_t(i0 + g) * 3 + c : dac + size_t(i0 + g) * ra + (c - 3);
        c += 32;
        while (c >= rg) { c -= rg; ++g; }
      }
#pragma unroll
      for (int q = 0; q < kInFlight; ++q)
        if (dst[q] != nullptr) *dst[q] = v[q];
    }
  }
}

// A batched call's SH rows of the warp's elements [i0, i0 + n): one scene's
// contiguous rows when all n belong to one item (sh_stage_in's spans), else
// each thread its own row (the warp spans scenes).  Warp-collective.
__device__ __forceinline__ void batch_sh_stage_in(const BackwardArgs& a, int i0, int n, float* s, int stride) {
  const int lane = threadIdx.x & 31;
  const int first = find_item_elem(a.items, a.num_items, uint32_t(i0));
  const int last = find_item_elem(a.items, a.num_items, uint32_t(i0 + n - 1));
  if (first == last) {
    const BatchItem& it = a.items[first];
    sh_stage_in(it.shs, a.M, i0 - int(it.elem_base), n, s, stride);
    return;
  }
  const int rs = 3 * (a.M < 16 ? a.M : 16);
  if (lane < n) {
    const int i = i0 + lane;
    const BatchItem& it = a.items[find_item_elem(a.items, a.num_items, uint32_t(i))];
    const float* row = it.shs + size_t(i - int(it.elem_base)) * 3 * a.M;
    for (int c = 0; c < rs; ++c) s[lane * stride + c] = __ldg(row + c);
  }
  __syncwarp();
}

// Per-Gaussian, reference formulas (backward.cu:27-227 then :229-519)
__constant__ float kSH_C2[5] = {1.0925484305920792f, -1.0925484305920792f, 0.31539156525252005f,
                                -1.0925484305920792f, 0.5462742152960396f};
__constant__ float kSH_C3[7] = {-0.5900435899266435f, 2.890611442640554f, -0.4570457994644658f,
                                0.3731763325901154f,  -0.4570457994644658f, 1.445305721320277f,
                                -0.5900435899266435f};

// The scene and camera of one element: the call's, or its batch item's.
struct GView {
  const float* means3D;
  const float* scales;
  const float* rotations;
  const float* mats;  // view (16), projection (16), camera position (3)
  int gi;             // index within the scene
  int W, degree;
  float h_x, h_y, tan_fovx, tan_fovy, focal_x, scale_modifier;
  const float* svec = nullptr;  // raw scales / quaternions (then scales / rotations are unused)
  const float* quat = nullptr;

  // the activated scale k and rotation (w, x, y, z).  The raw path's
  // rotation multiplies by the reciprocal of the clamped norm (the forward
  // divides, bit-exact with torch; here it only enters gradients, and the two
  // differ by at most an ulp)
  __device__ __forceinline__ float scale(int k) const {
    return svec != nullptr ? expf(__ldg(&svec[3 * gi + k])) : __ldg(&scales[3 * gi + k]);
  }
  __device__ __forceinline__ float4 rotation() const {
    if (quat != nullptr) {
      const float4 q = load_quat(quat, gi);
      const float w = q.x, x = q.y, y = q.z, z = q.w;
      const float inv = __frcp_rn(fmaxf(sqrtf((w * w + y * y) + (x * x + z * z)), 1e-12f));
      return make_float4(w * inv, x * inv, y * inv, z * inv);
    }
    return load_quat(rotations, gi);
  }
};

// Element i (global index) of batch item `it`.
__device__ __forceinline__ GView item_gview(const BatchItem& it, int i) {
  return GView{it.means3D, it.scales, it.rotations, it.view, i - int(it.elem_base), it.W, it.degree, it.h_x, it.h_y,
               it.tan_fovx, it.tan_fovy, it.h_x, it.scale_modifier};
}

__device__ __forceinline__ GView make_gview(const BackwardArgs& a, int i, const float* s_mats) {
  GView g;
  if (a.items == nullptr) {
    g = GView{a.means3D, a.scales, a.rotations, s_mats, i, a.W, a.degree, a.h_x, a.h_y, a.tan_fovx, a.tan_fovy,
              a.focal_x, a.scale_modifier};
    g.svec = a.svec;
    g.quat = a.quat;
  } else {
    g = item_gview(a.items[find_item_elem(a.items, a.num_items, uint32_t(i))], i);
  }
  return g;
}

// The per-Gaussian outputs of one element (kept in registers; the kernels
// store them, or sum them over a group's views).
struct GOut {
  float m3[3], cov[6], sc[3], rot[4];
};

__device__ __forceinline__ void store_gout(const BackwardArgs& a, int i, const GOut& o) {
  for (int k = 0; k < 3; ++k) a.dL_dmeans3D[3 * i + k] = o.m3[k];
  for (int k = 0; k < 6; ++k) a.dL_dcov3D[6 * i + k] = o.cov[k];
  for (int k = 0; k < 3; ++k) a.dL_dscales[3 * i + k] = o.sc[k];
  for (int k = 0; k < 4; ++k) a.dL_drotations[4 * i + k] = o.rot[k];
}

// One Gaussian (radius > 0) of the reference-formula pass, in two parts: the
// covariance and mean gradients (sd: dL/dmean so far), which need no SH
// coefficient, then every other output but dL_dsh, plus the SH basis and masked
// colour gradient dL_dsh is built from.
__device__ __forceinline__ void ref_gaussian_geometry(const BackwardArgs& a, int i, const GView& gv, GOut& o,
                                                      float (&dc)[6], float (&sd)[3]) {
  const float* mats = gv.mats;
  const float* view = mats;
  const float* proj = mats + 16;
  const float cx = __ldg(&gv.means3D[3 * gv.gi]), cy = __ldg(&gv.means3D[3 * gv.gi + 1]), cz = __ldg(&gv.means3D[3 * gv.gi + 2]);
  const float* pc = a.cov3D + 6 * size_t(i);  // read with __ldg below

  // ---- computeCov2DCUDA ----
  float vx = view[0] * cx + view[4] * cy + view[8] * cz + view[12];
  float vy = view[1] * cx + view[5] * cy + view[9] * cz + view[13];
  float vz = view[2] * cx + view[6] * cy + view[10] * cz + view[14];
  const float vw = view[3] * cx + view[7] * cy + view[11] * cz + view[15];
  const float w_inv = 1.0f / (vw + 1e-8f);
  vx *= w_inv;
  vy *= w_inv;
  vz *= w_inv;
  const float bound_x = 1.3f * gv.tan_fovx, bound_y = 1.3f * gv.tan_fovy;
  const float proj_x = vx / vz, proj_y = vy / vz;
  const float cpx = fminf(bound_x, fmaxf(-bound_x, proj_x));
  const float cpy = fminf(bound_y, fmaxf(-bound_y, proj_y));
  const float px = cpx * vz, py = cpy * vz;
  const float mask_x = (proj_x >= -bound_x && proj_x <= bound_x) ? 1.0f : 0.0f;
  const float mask_y = (proj_y >= -bound_y && proj_y <= bound_y) ? 1.0f : 0.0f;
  const float z_inv = 1.0f / vz, z_inv2 = z_inv * z_inv;
  const float h_x = gv.h_x, h_y = gv.h_y;
  // J (glm column-major J[col][row]) and T = W * J
  const float J[3][3] = {{h_x * z_inv, 0.f, -h_x * px * z_inv2}, {0.f, h_y * z_inv, -h_y * py * z_inv2}, {0.f, 0.f, 0.f}};
  const float Wv[3][3] = {{view[0], view[4], view[8]}, {view[1], view[5], view[9]}, {view[2], view[6], view[10]}};
  const float Vk[3][3] = {{__ldg(pc + 0), __ldg(pc + 1), __ldg(pc + 2)}, {__ldg(pc + 1), __ldg(pc + 3), __ldg(pc + 4)}, {__ldg(pc + 2), __ldg(pc + 4), __ldg(pc + 5)}};
  float T[3][3], tmp[3][3], c2[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int r = 0; r < 3; ++r) T[c][r] = Wv[0][r] * J[c][0] + Wv[1][r] * J[c][1] + Wv[2][r] * J[c][2];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int r = 0; r < 3; ++r) tmp[c][r] = Vk[r][0] * T[c][0] + Vk[r][1] * T[c][1] + Vk[r][2] * T[c][2];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int r = 0; r < 3; ++r) c2[c][r] = T[r][0] * tmp[c][0] + T[r][1] * tmp[c][1] + T[r][2] * tmp[c][2];
  c2[0][0] += 0.3f;
  c2[1][1] += 0.3f;
  const float ca = c2[0][0], cb = c2[0][1], cc = c2[1][1];
  const float den = ca * cc - cb * cb;
  const float dinv2 = 1.0f / (den * den + 1e-7f);
  const float gx = __ldg(&a.acc_cov[4 * i]), gy = __ldg(&a.acc_cov[4 * i + 1]), gz = __ldg(&a.acc_cov[4 * i + 3]);
  float ga = 0.f, gb = 0.f, gc = 0.f;
  if (dinv2 > 0) {
    ga = dinv2 * (-cc * cc * gx + 2.0f * cb * cc * gy + (den - ca * cc) * gz);
    gb = dinv2 * 2.0f * (cb * cc * gx - (den + 2.0f * cb * cb) * gy + ca * cb * gz);
    gc = dinv2 * (-ca * ca * gz + 2.0f * ca * cb * gy + (den - ca * cc) * gx);
    dc[0] = T[0][0] * T[0][0] * ga + T[0][0] * T[1][0] * gb + T[1][0] * T[1][0] * gc;
    dc[3] = T[0][1] * T[0][1] * ga + T[0][1] * T[1][1] * gb + T[1][1] * T[1][1] * gc;
    dc[5] = T[0][2] * T[0][2] * ga + T[0][2] * T[1][2] * gb + T[1][2] * T[1][2] * gc;
    dc[1] = 2.0f * (T[0][0] * T[0][1] * ga + (T[0][0] * T[1][1] + T[0][1] * T[1][0]) * gb * 0.5f + T[1][0] * T[1][1] * gc);
    dc[2] = 2.0f * (T[0][0] * T[0][2] * ga + (T[0][0] * T[1][2] + T[0][2] * T[1][0]) * gb * 0.5f + T[1][0] * T[1][2] * gc);
    dc[4] = 2.0f * (T[0][1] * T[0][2] * ga + (T[0][1] * T[1][2] + T[0][2] * T[1][1]) * gb * 0.5f + T[1][1] * T[1][2] * gc);
  } else {
    for (int k = 0; k < 6; ++k) dc[k] = 0.f;
  }
  for (int k = 0; k < 6; ++k) o.cov[k] = dc[k];
  const float gT00 = 2.0f * (T[0][0] * Vk[0][0] + T[0][1] * Vk[0][1] + T[0][2] * Vk[0][2]) * ga + (T[1][0] * Vk[0][0] + T[1][1] * Vk[0][1] + T[1][2] * Vk[0][2]) * gb;
  const float gT01 = 2.0f * (T[0][0] * Vk[1][0] + T[0][1] * Vk[1][1] + T[0][2] * Vk[1][2]) * ga + (T[1][0] * Vk[1][0] + T[1][1] * Vk[1][1] + T[1][2] * Vk[1][2]) * gb;
  const float gT02 = 2.0f * (T[0][0] * Vk[2][0] + T[0][1] * Vk[2][1] + T[0][2] * Vk[2][2]) * ga + (T[1][0] * Vk[2][0] + T[1][1] * Vk[2][1] + T[1][2] * Vk[2][2]) * gb;
  const float gT10 = 2.0f * (T[1][0] * Vk[0][0] + T[1][1] * Vk[0][1] + T[1][2] * Vk[0][2]) * gc + (T[0][0] * Vk[0][0] + T[0][1] * Vk[0][1] + T[0][2] * Vk[0][2]) * gb;
  const float gT11 = 2.0f * (T[1][0] * Vk[1][0] + T[1][1] * Vk[1][1] + T[1][2] * Vk[1][2]) * gc + (T[0][0] * Vk[1][0] + T[0][1] * Vk[1][1] + T[0][2] * Vk[1][2]) * gb;
  const float gT12 = 2.0f * (T[1][0] * Vk[2][0] + T[1][1] * Vk[2][1] + T[1][2] * Vk[2][2]) * gc + (T[0][0] * Vk[2][0] + T[0][1] * Vk[2][1] + T[0][2] * Vk[2][2]) * gb;
  const float gJ00 = Wv[0][0] * gT00 + Wv[0][1] * gT01 + Wv[0][2] * gT02;
  const float gJ02 = Wv[2][0] * gT00 + Wv[2][1] * gT01 + Wv[2][2] * gT02;
  const float gJ11 = Wv[1][0] * gT10 + Wv[1][1] * gT11 + Wv[1][2] * gT12;
  const float gJ12 = Wv[2][0] * gT10 + Wv[2][1] * gT11 + Wv[2][2] * gT12;
  const float z_inv3 = z_inv2 * z_inv;
  const float gvx = mask_x * (-h_x * z_inv2 * gJ02);
  const float gvy = mask_y * (-h_y * z_inv2 * gJ12);
  const float gvz = -h_x * z_inv2 * gJ00 - h_y * z_inv2 * gJ11 + 2.0f * h_x * px * z_inv3 * gJ02 +
                    2.0f * h_y * py * z_inv3 * gJ12;
  sd[0] = view[0] * gvx + view[1] * gvy + view[2] * gvz;
  sd[1] = view[4] * gvx + view[5] * gvy + view[6] * gvz;
  sd[2] = view[8] * gvx + view[9] * gvy + view[10] * gvz;

  // ---- backwardPreprocessingKernel ----
  const float cw = proj[3] * cx + proj[7] * cy + proj[11] * cz + proj[15];
  const float iw = 1.0f / (cw + 1e-7f);
  const float iw2 = iw * iw;
  const float ptx = (proj[0] * cx + proj[4] * cy + proj[8] * cz + proj[12]) * iw2;
  const float pty = (proj[1] * cx + proj[5] * cy + proj[9] * cz + proj[13]) * iw2;
  const float g2x = __ldg(&a.dL_dmean2D[3 * i]), g2y = __ldg(&a.dL_dmean2D[3 * i + 1]);
  sd[0] += (proj[0] * iw - proj[3] * ptx) * g2x + (proj[1] * iw - proj[3] * pty) * g2y;
  sd[1] += (proj[4] * iw - proj[7] * ptx) * g2x + (proj[5] * iw - proj[7] * pty) * g2y;
  sd[2] += (proj[8] * iw - proj[11] * ptx) * g2x + (proj[9] * iw - proj[11] * pty) * g2y;
  const float vzz = view[2] * cx + view[6] * cy + view[10] * cz + view[14];
  const float gd = __ldg(&a.acc_depth[i]);
  sd[0] += (view[2] - view[3] * vzz) * gd;
  sd[1] += (view[6] - view[7] * vzz) * gd;
  sd[2] += (view[10] - view[11] * vzz) * gd;
}

// sh_row: this Gaussian's SH coefficients (staged in shared memory), of which
// coefficient 0, whose basis value is constant, is not read.
__device__ __forceinline__ void ref_gaussian_rest(const BackwardArgs& a, int i, const GView& gv, const float* sh_row,
                                                  const float (&dc)[6], float (&sd)[3], float (&basis)[16],
                                                  float (&cf)[3], GOut& o) {
  const int M = a.M;
  const float* cam = gv.mats + 32;
  const float cx = __ldg(&gv.means3D[3 * gv.gi]), cy = __ldg(&gv.means3D[3 * gv.gi + 1]), cz = __ldg(&gv.means3D[3 * gv.gi + 2]);
  // SH (all 16 bands, colour-clamp masks)
  const float ox = cx - cam[0], oy = cy - cam[1], oz = cz - cam[2];
  const float msq = ox * ox + oy * oy + oz * oz;
  const float mag = sqrtf(msq + 1e-10f);
  const float im = 1.0f / mag;
  const float x = ox * im, y = oy * im, z = oz * im;
  const float x2 = x * x, y2 = y * y, z2 = z * z, xy = x * y, xz = x * z, yz = y * z;
  const float x2my2 = x2 - y2, tx2 = 3.0f * x2, ty2 = 3.0f * y2, fz2 = 4.0f * z2, wz2 = 2.0f * z2;
  for (int ch = 0; ch < 3; ++ch) cf[ch] = __ldg(&a.dL_dcolors[3 * i + ch]) * (__ldg(&a.clamped[3 * i + ch]) ? 0.0f : 1.0f);
  const float SH_C0 = 0.28209479177387814f, SH_C1 = 0.4886025119029199f;
  basis[0] = SH_C0; basis[1] = -SH_C1 * y; basis[2] = SH_C1 * z; basis[3] = -SH_C1 * x;
  basis[4] = kSH_C2[0] * xy; basis[5] = kSH_C2[1] * yz; basis[6] = kSH_C2[2] * (wz2 - x2 - y2);
  basis[7] = kSH_C2[3] * xz; basis[8] = kSH_C2[4] * x2my2;
  basis[9] = kSH_C3[0] * y * (tx2 - y2); basis[10] = kSH_C3[1] * xy * z; basis[11] = kSH_C3[2] * y * (fz2 - x2 - y2);
  basis[12] = kSH_C3[3] * z * (wz2 - tx2 - ty2); basis[13] = kSH_C3[4] * x * (fz2 - x2 - y2);
  basis[14] = kSH_C3[5] * z * x2my2; basis[15] = kSH_C3[6] * x * (x2 - ty2);
  auto SH = [&](int k, int ch) -> float { return k < M ? sh_row[3 * k + ch] : 0.0f; };
  float ag[3] = {0.f, 0.f, 0.f};
  auto dotc = [&](int k) { return SH(k, 0) * cf[0] + SH(k, 1) * cf[1] + SH(k, 2) * cf[2]; };
  ag[0] -= SH_C1 * dotc(3);
  ag[1] -= SH_C1 * dotc(1);
  ag[2] += SH_C1 * dotc(2);
  float d2x[3], d2y[3], d2z[3];
  for (int ch = 0; ch < 3; ++ch) {
    d2x[ch] = kSH_C2[0] * y * SH(4, ch) + kSH_C2[2] * (-2.0f * x) * SH(6, ch) + kSH_C2[3] * z * SH(7, ch) + kSH_C2[4] * (2.0f * x) * SH(8, ch);
    d2y[ch] = kSH_C2[0] * x * SH(4, ch) + kSH_C2[1] * z * SH(5, ch) + kSH_C2[2] * (-2.0f * y) * SH(6, ch) + kSH_C2[4] * (-2.0f * y) * SH(8, ch);
    d2z[ch] = kSH_C2[1] * y * SH(5, ch) + kSH_C2[2] * (4.0f * z) * SH(6, ch) + kSH_C2[3] * x * SH(7, ch);
  }
  ag[0] += d2x[0] * cf[0] + d2x[1] * cf[1] + d2x[2] * cf[2];
  ag[1] += d2y[0] * cf[0] + d2y[1] * cf[1] + d2y[2] * cf[2];
  ag[2] += d2z[0] * cf[0] + d2z[1] * cf[1] + d2z[2] * cf[2];
  const float f3x[7] = {kSH_C3[0] * 6.0f * xy, kSH_C3[1] * yz, kSH_C3[2] * (-2.0f * xy), kSH_C3[3] * (-6.0f * xz),
                        kSH_C3[4] * (fz2 - 3.0f * x2 - y2), kSH_C3[5] * 2.0f * xz, kSH_C3[6] * 3.0f * x2my2};
  const float f3y[7] = {kSH_C3[0] * 3.0f * (x2 - y2), kSH_C3[1] * xz, kSH_C3[2] * (fz2 - 3.0f * y2 - x2),
                        kSH_C3[3] * (-6.0f * yz), kSH_C3[4] * (-2.0f * xy), kSH_C3[5] * (-2.0f * yz),
                        kSH_C3[6] * (-6.0f * xy)};
  const float f3z[7] = {0.0f, kSH_C3[1] * xy, kSH_C3[2] * 8.0f * yz, kSH_C3[3] * 3.0f * (wz2 - x2 - y2),
                        kSH_C3[4] * 8.0f * xz, kSH_C3[5] * x2my2, 0.0f};
  float d3x[3] = {0.f, 0.f, 0.f}, d3y[3] = {0.f, 0.f, 0.f}, d3z[3] = {0.f, 0.f, 0.f};
  for (int k = 0; k < 7; ++k)
    for (int ch = 0; ch < 3; ++ch) {
      const float s = SH(9 + k, ch);
      d3x[ch] += f3x[k] * s;
      d3y[ch] += f3y[k] * s;
      d3z[ch] += f3z[k] * s;
    }
  ag[0] += d3x[0] * cf[0] + d3x[1] * cf[1] + d3x[2] * cf[2];
  ag[1] += d3y[0] * cf[0] + d3y[1] * cf[1] + d3y[2] * cf[2];
  ag[2] += d3z[0] * cf[0] + d3z[1] * cf[1] + d3z[2] * cf[2];
  const float im3 = im * im * im;
  const float rd[3] = {ox, oy, oz};
  for (int r = 0; r < 3; ++r) {
    float acc = 0.f;
    for (int c = 0; c < 3; ++c) acc += ((c == r ? msq : 0.0f) - rd[c] * rd[r]) * im3 * ag[c];
    sd[r] += acc;
  }
  o.m3[0] = sd[0];
  o.m3[1] = sd[1];
  o.m3[2] = sd[2];

  // ---- scale / rotation (backward.cu:446-518) ----
  const float4 qr = gv.rotation();
  const float qw = qr.x, qx = qr.y, qy = qr.z, qz = qr.w;
  const float xx = qx * qx, yy = qy * qy, zz = qz * qz;
  const float qxy = qx * qy, qxz = qx * qz, qyz = qy * qz;
  const float xw = qx * qw, yw = qy * qw, zw = qz * qw;
  const float sc[3] = {gv.scale(0), gv.scale(1), gv.scale(2)};
  const float sx = gv.scale_modifier * sc[0], sy = gv.scale_modifier * sc[1], sz = gv.scale_modifier * sc[2];
  const float m11 = sx * (1.f - 2.f * (yy + zz)), m12 = sx * 2.f * (qxy - zw), m13 = sx * 2.f * (qxz + yw);
  const float m21 = sy * 2.f * (qxy + zw), m22 = sy * (1.f - 2.f * (xx + zz)), m23 = sy * 2.f * (qyz - xw);
  const float m31 = sz * 2.f * (qxz - yw), m32 = sz * 2.f * (qyz + xw), m33 = sz * (1.f - 2.f * (xx + yy));
  const float g11 = dc[0], g12 = dc[1], g13 = dc[2], g22 = dc[3], g23 = dc[4], g33 = dc[5];
  const float a11 = 2.f * (m11 * g11 + m12 * g12 + m13 * g13);
  const float a12 = 2.f * (m11 * g12 + m12 * g22 + m13 * g23);
  const float a13 = 2.f * (m11 * g13 + m12 * g23 + m13 * g33);
  const float a21 = 2.f * (m21 * g11 + m22 * g12 + m23 * g13);
  const float a22 = 2.f * (m21 * g12 + m22 * g22 + m23 * g23);
  const float a23 = 2.f * (m21 * g13 + m22 * g23 + m23 * g33);
  const float a31 = 2.f * (m31 * g11 + m32 * g12 + m33 * g13);
  const float a32 = 2.f * (m31 * g12 + m32 * g22 + m33 * g23);
  const float a33 = 2.f * (m31 * g13 + m32 * g23 + m33 * g33);
  float ds[3] = {(1.f - 2.f * (yy + zz)) * a11 + 2.f * (qxy - zw) * a12 + 2.f * (qxz + yw) * a13,
                 2.f * (qxy + zw) * a21 + (1.f - 2.f * (xx + zz)) * a22 + 2.f * (qyz - xw) * a23,
                 2.f * (qxz - yw) * a31 + 2.f * (qyz + xw) * a32 + (1.f - 2.f * (xx + yy)) * a33};
  if (gv.svec != nullptr)  // raw path: scales = exp(svec)
    for (int k = 0; k < 3; ++k) ds[k] = ds[k] * sc[k];
  o.sc[0] = ds[0];
  o.sc[1] = ds[1];
  o.sc[2] = ds[2];
  float4 dq;
  dq.x = 4.f * (-sz * (a31 * yw - a32 * xw + a33 * qxy) + sy * (a21 * zw - a22 * qxz + a23 * yy) + sx * (a12 * zw - a13 * yw - a11 * qyz));
  dq.y = 4.f * (sz * (a31 * zw + a32 * zz - a33 * qyz) - sy * (a21 * yw + a22 * qxy + a23 * xx) + sx * (a12 * yy + a13 * zw + a11 * qxz));
  dq.z = 4.f * (-sz * (a31 * xx + a32 * xw + a33 * qxz) + sy * (a21 * zw + a22 * yy + a23 * yw) - sx * (a12 * xw + a13 * xx + a11 * qxy));
  dq.w = 4.f * (sz * (a31 * xw - a32 * xx + a33 * qxy) - sy * (a21 * qxz - a22 * zw + a23 * qyz) + sx * (a12 * qyz - a13 * zz + a11 * yy));
  if (gv.quat != nullptr) {  // raw path: rotation = q / max(|q|, 1e-12)
    const float4 qv = load_quat(gv.quat, gv.gi);
    const float q0 = qv.x, q1 = qv.y, q2 = qv.z, q3 = qv.w;
    const float n = sqrtf(q0 * q0 + q1 * q1 + q2 * q2 + q3 * q3);
    if (n > 1e-12f) {  // (g - r (r . g)) / n with r = q / n
      const float inv = __frcp_rn(n);
      const float rg = (q0 * dq.x + q1 * dq.y + q2 * dq.z + q3 * dq.w) * inv;
      dq = make_float4((dq.x - q0 * inv * rg) * inv, (dq.y - q1 * inv * rg) * inv, (dq.z - q2 * inv * rg) * inv,
                       (dq.w - q3 * inv * rg) * inv);
    } else {  // the norm is clamped to 1e-12 there: q / 1e-12 is linear in q
      dq = make_float4(dq.x * 1e12f, dq.y * 1e12f, dq.z * 1e12f, dq.w * 1e12f);
    }
  }
  o.rot[0] = dq.x;
  o.rot[1] = dq.y;
  o.rot[2] = dq.z;
  o.rot[3] = dq.w;
}

// Bound by memory: 556 bytes a Gaussian, 4.5 TB/s at 500k and 5 TB/s at 1M.  The
// raw SH rows arrive asynchronously under the covariance gradients, and dL/dSH
// leaves as products each lane forms for its own row (store_rows): 78 -> 62 us a
// view at 500k, 142 -> 112 us at 1M, against rows staged through registers and
// outputs whose factors every lane looked up by index.  8 CTAs per SM (64
// registers): more Gaussians' loads in flight.
__global__ void __launch_bounds__(kGaussThreads, 8) gaussians_ref_kernel(BackwardArgs a) {
  grid_wait();
  __shared__ __align__(16) float s_sh[kGaussThreads / 32][32 * kGaussRow];
  // view, projection, camera position: shared memory is never aliased by the
  // outputs, so these stay in place across the output stores
  __shared__ float s_mats[35];
  if (a.items == nullptr) {  // a batched call's matrices live in its item table
    if (threadIdx.x < 16) s_mats[threadIdx.x] = a.view[threadIdx.x];
    else if (threadIdx.x < 32) s_mats[threadIdx.x] = a.proj[threadIdx.x - 16];
    else if (threadIdx.x < 35) s_mats[threadIdx.x] = a.campos[threadIdx.x - 32];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  float* sw = s_sh[threadIdx.x >> 5];
  const int i0 = blockIdx.x * kGaussThreads + (threadIdx.x & ~31);
  if (i0 >= a.P) return;  // warp-uniform
  const int n = min(32, a.P - i0);
  const int i = i0 + lane;
  const int stride = sh_stride(a.M);
  const float* row = sw + lane * stride;
  if (a.items == nullptr) {
    if (a.sh_dc != nullptr) {
      if (sh_stage_in_raw(a.sh_dc, a.sh_ac, a.M, i0, n, sw, stride)) row = sw + 45 * lane - 3;
    } else {
      sh_stage_in(a.shs, a.M, i0, n, sw, stride);
    }
  } else {
    batch_sh_stage_in(a, i0, n, sw, stride);
  }
  const GView gv = make_gview(a, lane < n ? i : i0, s_mats);
  float basis[16], cf[3] = {0.f, 0.f, 0.f};
  const bool active = lane < n && a.radii[i] > 0;
  GOut o;
  float dcov[6], sd[3];
  if (active) ref_gaussian_geometry(a, i, gv, o, dcov, sd);
  copy_wait();
  __syncwarp();
  if (active) {
    ref_gaussian_rest(a, i, gv, row, dcov, sd, basis, cf, o);
    store_gout(a, i, o);
  } else if (lane < n) {
    for (int k = 0; k < 3; ++k) a.dL_dmeans3D[3 * i + k] = 0.f;
    for (int k = 0; k < 6; ++k) a.dL_dcov3D[6 * i + k] = 0.f;
    for (int k = 0; k < 3; ++k) a.dL_dscales[3 * i + k] = 0.f;
    for (int k = 0; k < 4; ++k) a.dL_drotations[4 * i + k] = 0.f;
  }
  // raw path: the accumulated opacity gradient through opacity = sigmoid(logit)
  if (a.logit != nullptr && lane < n) {
    const float y = __frcp_rn(1.f + expf(-__ldg(&a.logit[i])));  // sigmoid, within an ulp of the forward's
    a.dL_dopacity[i] = a.dL_dopacity[i] * (1.f - y) * y;
  }
  // densification statistics (gaussians_handler.py:116-118) in this pass, not
  // one of their own; atomic, because views on other streams may add too
  if (a.dens_accum != nullptr && lane < n && a.radii[i] > 0) {
    const float gx = a.dL_dmean2D[3 * i], gy = a.dL_dmean2D[3 * i + 1];
    atomicAdd(&a.dens_accum[i], __fsqrt_rn(__fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy))));
    atomicAdd(&a.dens_counter[i], 1.0f);
  }
  // dL_dsh[k][ch] = basis[k] * cf[ch] for the first min(M, 16) bands, 0 beyond
  if (a.dL_dsh_dc != nullptr) sh_store_outer_raw(a.dL_dsh_dc, a.dL_dsh_ac, a.M, i0, n, sw, basis, cf, active);
  else sh_store_outer(a.dL_dsh, a.M, i0, n, sw, basis, cf, active);
}

// Per-Gaussian, exact derivative of the forward.
// One Gaussian (radius > 0) of the exact-derivative pass: every output but
// dL_dsh, plus the outer-product factors of dL_dsh (see ref_gaussian).
__device__ __forceinline__ void exact_gaussian(const BackwardArgs& a, int i, const GView& gv, const float* sh_row,
                                               float (&basis)[16], float (&cf)[3], GOut& o) {
  const int M = a.M;
  const float* mats = gv.mats;
  const float* cam = mats + 32;
  const float* V = mats;
  const float* PM = mats + 16;
  const float m0 = __ldg(&gv.means3D[3 * gv.gi]), m1 = __ldg(&gv.means3D[3 * gv.gi + 1]), m2 = __ldg(&gv.means3D[3 * gv.gi + 2]);
  float gm[3] = {0.f, 0.f, 0.f};
  // screen position / depth: ndc = clip.xyz / (clip.w + 1e-5); dL_dmean2D already holds dL/dNDC
  float clip[4];
  for (int r = 0; r < 4; ++r) clip[r] = PM[r] * m0 + PM[4 + r] * m1 + PM[8 + r] * m2 + PM[12 + r];
  const float wi = 1.0f / (clip[3] + 1e-5f);
  const float gn0 = __ldg(&a.dL_dmean2D[3 * i]), gn1 = __ldg(&a.dL_dmean2D[3 * i + 1]), gn2 = __ldg(&a.acc_depth[i]);
  const float gcl[4] = {gn0 * wi, gn1 * wi, gn2 * wi, -(gn0 * clip[0] + gn1 * clip[1] + gn2 * clip[2]) * wi * wi};
  for (int c = 0; c < 3; ++c)
    for (int r = 0; r < 4; ++r) gm[c] += PM[4 * c + r] * gcl[r];
  // covariance chain
  float t[3];
  for (int r = 0; r < 3; ++r) t[r] = V[r] * m0 + V[4 + r] * m1 + V[8 + r] * m2 + V[12 + r];
  const float L = float(gv.W) / (2.0f * gv.focal_x);
  const float rx = t[0] / t[2], ry = t[1] / t[2];
  const float nn = sqrtf(rx * rx + ry * ry) / L;
  const bool clampd = nn > 1.0f;
  float txp = t[0], typ = t[1];
  if (clampd) { txp = rx / nn * t[2]; typ = ry / nn * t[2]; }
  const float tz = t[2], f = gv.focal_x;
  const float rgt[3] = {V[0], V[4], V[8]}, upv[3] = {V[1], V[5], V[9]}, fw[3] = {V[2], V[6], V[10]};
  float jx[3], jy[3];
  for (int k = 0; k < 3; ++k) {
    jx[k] = f * (rgt[k] / tz - txp * fw[k] / (tz * tz));
    jy[k] = f * (upv[k] / tz - typ * fw[k] / (tz * tz));
  }
  const float* pc = a.cov3D + 6 * size_t(i);  // read with __ldg below
  const float S[3][3] = {{__ldg(pc + 0), __ldg(pc + 1), __ldg(pc + 2)}, {__ldg(pc + 1), __ldg(pc + 3), __ldg(pc + 4)}, {__ldg(pc + 2), __ldg(pc + 4), __ldg(pc + 5)}};
  const float gxx = __ldg(&a.acc_cov[4 * i]), gxy = __ldg(&a.acc_cov[4 * i + 1]), gyy = __ldg(&a.acc_cov[4 * i + 2]);
  float Gf[3][3];
  for (int p = 0; p < 3; ++p)
    for (int q = 0; q < 3; ++q) Gf[p][q] = gxx * jx[p] * jx[q] + gyy * jy[p] * jy[q] + gxy * jx[p] * jy[q];
  o.cov[0] = Gf[0][0];
  o.cov[1] = Gf[0][1] + Gf[1][0];
  o.cov[2] = Gf[0][2] + Gf[2][0];
  o.cov[3] = Gf[1][1];
  o.cov[4] = Gf[1][2] + Gf[2][1];
  o.cov[5] = Gf[2][2];
  float Sjx[3], Sjy[3];
  for (int p = 0; p < 3; ++p) {
    Sjx[p] = S[p][0] * jx[0] + S[p][1] * jx[1] + S[p][2] * jx[2];
    Sjy[p] = S[p][0] * jy[0] + S[p][1] * jy[1] + S[p][2] * jy[2];
  }
  float gtxp = 0.f, gtyp = 0.f, gtz = 0.f;
  for (int k = 0; k < 3; ++k) {
    const float gjx = 2.f * gxx * Sjx[k] + gxy * Sjy[k];
    const float gjy = 2.f * gyy * Sjy[k] + gxy * Sjx[k];
    gtxp += gjx * (-f * fw[k] / (tz * tz));
    gtyp += gjy * (-f * fw[k] / (tz * tz));
    gtz += gjx * f * (-rgt[k] / (tz * tz) + 2.f * txp * fw[k] / (tz * tz * tz));
    gtz += gjy * f * (-upv[k] / (tz * tz) + 2.f * typ * fw[k] / (tz * tz * tz));
  }
  float gt[3];
  if (!clampd) {
    gt[0] = gtxp; gt[1] = gtyp; gt[2] = gtz;
  } else {
    const float r2 = t[0] * t[0] + t[1] * t[1], r1 = sqrtf(r2), r3 = r2 * r1;
    const float dxx = L * tz * t[1] * t[1] / r3, dxy = -L * tz * t[0] * t[1] / r3, dxz = L * t[0] / r1;
    const float dyx = -L * tz * t[0] * t[1] / r3, dyy = L * tz * t[0] * t[0] / r3, dyz = L * t[1] / r1;
    gt[0] = gtxp * dxx + gtyp * dyx;
    gt[1] = gtxp * dxy + gtyp * dyy;
    gt[2] = gtz + gtxp * dxz + gtyp * dyz;
  }
  for (int c = 0; c < 3; ++c)
    for (int r = 0; r < 3; ++r) gm[c] += V[4 * c + r] * gt[r];
  // Sigma = M M^T, M = R diag(s)
  const float4 qr = gv.rotation();
  const float w = qr.x, x = qr.y, y = qr.z, z = qr.w;
  const float R[3][3] = {{1.f - 2.f * (y * y + z * z), 2.f * (x * y - w * z), 2.f * (x * z + w * y)},
                         {2.f * (x * y + w * z), 1.f - 2.f * (x * x + z * z), 2.f * (y * z - w * x)},
                         {2.f * (x * z - w * y), 2.f * (y * z + w * x), 1.f - 2.f * (x * x + y * y)}};
  const float s[3] = {gv.scale(0), gv.scale(1), gv.scale(2)};
  float dM[3][3];
  for (int p = 0; p < 3; ++p)
    for (int k = 0; k < 3; ++k) {
      float acc = 0.f;
      for (int q = 0; q < 3; ++q) acc += 0.5f * (Gf[p][q] + Gf[q][p]) * R[q][k] * s[k];
      dM[p][k] = 2.f * acc;
    }
  for (int k = 0; k < 3; ++k) {
    float acc = 0.f;
    for (int p = 0; p < 3; ++p) acc += dM[p][k] * R[p][k];
    o.sc[k] = acc;
  }
  float dR[3][3];
  for (int p = 0; p < 3; ++p)
    for (int k = 0; k < 3; ++k) dR[p][k] = dM[p][k] * s[k];
  o.rot[0] = dR[0][1] * (-2.f * z) + dR[0][2] * (2.f * y) + dR[1][0] * (2.f * z) + dR[1][2] * (-2.f * x) +
                           dR[2][0] * (-2.f * y) + dR[2][1] * (2.f * x);
  o.rot[1] = dR[0][1] * (2.f * y) + dR[0][2] * (2.f * z) + dR[1][0] * (2.f * y) + dR[1][1] * (-4.f * x) +
                               dR[1][2] * (-2.f * w) + dR[2][0] * (2.f * z) + dR[2][1] * (2.f * w) + dR[2][2] * (-4.f * x);
  o.rot[2] = dR[0][0] * (-4.f * y) + dR[0][1] * (2.f * x) + dR[0][2] * (2.f * w) + dR[1][0] * (2.f * x) +
                               dR[1][2] * (2.f * z) + dR[2][0] * (-2.f * w) + dR[2][1] * (2.f * z) + dR[2][2] * (-4.f * y);
  o.rot[3] = dR[0][0] * (-4.f * z) + dR[0][1] * (-2.f * w) + dR[0][2] * (2.f * x) + dR[1][0] * (2.f * w) +
                               dR[1][1] * (-4.f * z) + dR[1][2] * (2.f * y) + dR[2][0] * (2.f * x) + dR[2][1] * (2.f * y);
  // colour: rgb = sum_k basis_k(dir) sh_k + 0.5 with the forward's constants
  const float v0 = m0 - cam[0], v1 = m1 - cam[1], v2 = m2 - cam[2];
  const float vn = sqrtf(v0 * v0 + v1 * v1 + v2 * v2);
  const float X = v0 / vn, Y = v1 / vn, Z = v2 / vn;
  const float gc0 = __ldg(&a.dL_dcolors[3 * i]), gc1 = __ldg(&a.dL_dcolors[3 * i + 1]), gc2 = __ldg(&a.dL_dcolors[3 * i + 2]);
  const float C1 = 0.4886025119029199f, C2a = 1.0925484305920792f, C2e = 0.5462742152960396f;
  const float C30 = 0.5900435899266435f, C31 = 2.890611442640554f, C32 = 0.4570457994644658f;
  const float C33 = 0.3731763325901154f, C35 = 1.445305721320277f;
  const float xx = X * X, yy = Y * Y, zz = Z * Z;
  float b[16], db[16][3];
  for (int k = 0; k < 16; ++k) db[k][0] = db[k][1] = db[k][2] = 0.f;
  b[0] = 0.28209479177387814f;
  b[1] = -C1 * Y; db[1][1] = -C1;
  b[2] = C1 * Z; db[2][2] = C1;
  b[3] = -C1 * X; db[3][0] = -C1;
  b[4] = C2a * X * Y; db[4][0] = C2a * Y; db[4][1] = C2a * X;
  b[5] = -C2a * Y * Z; db[5][1] = -C2a * Z; db[5][2] = -C2a * Y;
  b[6] = 0.3f * (2.f * zz - xx - yy); db[6][0] = -0.6f * X; db[6][1] = -0.6f * Y; db[6][2] = 1.2f * Z;
  b[7] = -C2a * X * Z; db[7][0] = -C2a * Z; db[7][2] = -C2a * X;
  b[8] = C2e * (xx - yy); db[8][0] = 2.f * C2e * X; db[8][1] = -2.f * C2e * Y;
  b[9] = -C30 * Y * (3.f * xx - yy); db[9][0] = -6.f * C30 * X * Y; db[9][1] = -C30 * (3.f * xx - 3.f * yy);
  b[10] = C31 * X * Y * Z; db[10][0] = C31 * Y * Z; db[10][1] = C31 * X * Z; db[10][2] = C31 * X * Y;
  b[11] = -C32 * Y * (4.f * zz - xx - yy); db[11][0] = 2.f * C32 * X * Y; db[11][1] = -C32 * (4.f * zz - xx - 3.f * yy); db[11][2] = -8.f * C32 * Y * Z;
  b[12] = C33 * Z * (2.f * zz - 3.f * xx - 3.f * yy); db[12][0] = -6.f * C33 * X * Z; db[12][1] = -6.f * C33 * Y * Z; db[12][2] = C33 * (6.f * zz - 3.f * xx - 3.f * yy);
  b[13] = -C32 * X * (4.f * zz - xx - yy); db[13][0] = -C32 * (4.f * zz - 3.f * xx - yy); db[13][1] = 2.f * C32 * X * Y; db[13][2] = -8.f * C32 * X * Z;
  b[14] = C35 * Z * (xx - yy); db[14][0] = 2.f * C35 * X * Z; db[14][1] = -2.f * C35 * Y * Z; db[14][2] = C35 * (xx - yy);
  b[15] = -C30 * X * (xx - 3.f * yy); db[15][0] = -C30 * (3.f * xx - 3.f * yy); db[15][1] = 6.f * C30 * X * Y;
  int de = gv.degree > 3 ? 3 : gv.degree;
  while (de > 0 && (de + 1) * (de + 1) > M) --de;
  const int nb = (de + 1) * (de + 1);
  const float* shd = sh_row;
  float gdir[3] = {0.f, 0.f, 0.f};
  for (int k = 0; k < nb; ++k) {
    const float sdot = shd[3 * k] * gc0 + shd[3 * k + 1] * gc1 + shd[3 * k + 2] * gc2;
    gdir[0] += sdot * db[k][0];
    gdir[1] += sdot * db[k][1];
    gdir[2] += sdot * db[k][2];
  }
  // dL_dsh = b[k] * gc for the bands the forward used, 0 beyond
  for (int k = 0; k < 16; ++k) basis[k] = k < nb ? b[k] : 0.f;
  cf[0] = gc0;
  cf[1] = gc1;
  cf[2] = gc2;
  const float dd[3] = {X, Y, Z};
  const float dot = dd[0] * gdir[0] + dd[1] * gdir[1] + dd[2] * gdir[2];
  for (int p = 0; p < 3; ++p) gm[p] += (gdir[p] - dd[p] * dot) / vn;
  o.m3[0] = gm[0];
  o.m3[1] = gm[1];
  o.m3[2] = gm[2];
}

__global__ void __launch_bounds__(kGaussThreads) gaussians_exact_kernel(BackwardArgs a) {
  grid_wait();
  __shared__ __align__(16) float s_sh[kGaussThreads / 32][32 * kGaussRow];
  // view, projection, camera position: shared memory is never aliased by the
  // outputs, so these stay in place across the output stores
  __shared__ float s_mats[35];
  if (a.items == nullptr) {  // a batched call's matrices live in its item table
    if (threadIdx.x < 16) s_mats[threadIdx.x] = a.view[threadIdx.x];
    else if (threadIdx.x < 32) s_mats[threadIdx.x] = a.proj[threadIdx.x - 16];
    else if (threadIdx.x < 35) s_mats[threadIdx.x] = a.campos[threadIdx.x - 32];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  float* sw = s_sh[threadIdx.x >> 5];
  const int i0 = blockIdx.x * kGaussThreads + (threadIdx.x & ~31);
  if (i0 >= a.P) return;  // warp-uniform
  const int n = min(32, a.P - i0);
  const int i = i0 + lane;
  const int stride = sh_stride(a.M);
  const GView gv = make_gview(a, lane < n ? i : i0, s_mats);
  if (a.items == nullptr) {
    sh_stage_in(a.shs, a.M, i0, n, sw, stride);
  } else {
    batch_sh_stage_in(a, i0, n, sw, stride);
  }
  float basis[16], cf[3] = {0.f, 0.f, 0.f};
  const bool active = lane < n && a.radii[i] > 0;
  if (active) {
    GOut o;
    exact_gaussian(a, i, gv, sw + lane * stride, basis, cf, o);
    store_gout(a, i, o);
  } else if (lane < n) {
    for (int k = 0; k < 3; ++k) a.dL_dmeans3D[3 * i + k] = 0.f;
    for (int k = 0; k < 6; ++k) a.dL_dcov3D[6 * i + k] = 0.f;
    for (int k = 0; k < 3; ++k) a.dL_dscales[3 * i + k] = 0.f;
    for (int k = 0; k < 4; ++k) a.dL_drotations[4 * i + k] = 0.f;
  }
  sh_store_outer(a.dL_dsh, a.M, i0, n, sw, basis, cf, active);
}

// ---------------------------------------------------------------------------
// Grouped per-Gaussian pass (batched calls): one thread per output row of a
// group (a scene, or a serving request), walking the group's items (views) in
// table order.  Each item's element is the single-view computation above; its
// outputs are summed in registers in item order, starting from zero, with
// explicit-rounding adds -- w2w_group_sum's order over the per-element
// outputs (the per-view arithmetic, inlined here, may fuse a multiply-add
// differently, so the two agree to a few ulps).  The SH rows are staged once per warp for
// all views of a scene (a view of another scene reads its own row from
// memory), and no per-element dL/dSH, dL/dmeans3D, dL/dscales, dL/drotations
// or dL/dcov3D is written.
// ---------------------------------------------------------------------------
template <int kMode>
__global__ void __launch_bounds__(kGaussThreads) gaussians_group_kernel(BackwardArgs a) {
  grid_wait();
  __shared__ __align__(16) float s_sh[kGaussThreads / 32][32 * kGaussRow];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  float* sw = s_sh[threadIdx.x >> 5];
  const long long row0 = (long long)blockIdx.x * kGaussThreads + (threadIdx.x & ~31);
  if (row0 >= a.group_rows) return;  // warp-uniform
  const int n = int(min(32LL, a.group_rows - row0));
  const uint32_t row = uint32_t(row0) + uint32_t(lane < n ? lane : 0);
  const uint32_t* gbase = a.group_tables;
  const uint32_t* iptr = gbase + (a.num_groups + 1);
  const uint32_t* ielem = iptr + (a.num_groups + 1);
  int lo = 0, hi = a.num_groups - 1;  // this row's group: the last g with gbase[g] <= row
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (__ldg(gbase + mid) <= row) lo = mid;
    else hi = mid - 1;
  }
  const int g = lo;
  const uint32_t r = row - __ldg(gbase + g);
  const uint32_t k0 = __ldg(iptr + g), k1 = __ldg(iptr + g + 1);
  const int M = a.M, rg = 3 * M, stride = sh_stride(M);
  const uint32_t e0 = k0 < k1 ? __ldg(ielem + k0) + r : uint32_t(a.P);
  const float* shs0 = e0 < uint32_t(a.P) ? a.items[find_item_elem(a.items, a.num_items, e0)].shs : nullptr;
  // the rows of the warp's first group's scene, contiguous when every lane is in that group
  if (__all_sync(full, g == __shfl_sync(full, g, 0) && shs0 != nullptr)) {
    sh_stage_in(shs0, M, int(__shfl_sync(full, r, 0)), n, sw, stride);
  } else {
    if (lane < n && shs0 != nullptr)
      for (int c = 0; c < 3 * (M < 16 ? M : 16); ++c) sw[lane * stride + c] = __ldg(shs0 + size_t(r) * rg + c);
    __syncwarp();
  }
  float am[3] = {0.f, 0.f, 0.f}, asc[3] = {0.f, 0.f, 0.f}, arot[4] = {0.f, 0.f, 0.f, 0.f}, aop = 0.f;
  float ash[48];
#pragma unroll
  for (int c = 0; c < 48; ++c) ash[c] = 0.f;
  for (uint32_t k = k0; lane < n && k < k1; ++k) {
    const uint32_t i = __ldg(ielem + k) + r;
    if (i >= uint32_t(a.P)) continue;  // a table pointing past the elements: nothing is read there
    const BatchItem& it = a.items[find_item_elem(a.items, a.num_items, i)];
    const GView gv = item_gview(it, int(i));
    if (a.radii[i] > 0) {
      const float* sh_row = it.shs == shs0 ? sw + lane * stride : it.shs + size_t(gv.gi) * rg;
      float basis[16], cf[3];
      GOut o;
      if (kMode == 1) exact_gaussian(a, int(i), gv, sh_row, basis, cf, o);
      else {
        float dcov[6], sd[3];
        ref_gaussian_geometry(a, int(i), gv, o, dcov, sd);
        ref_gaussian_rest(a, int(i), gv, sh_row, dcov, sd, basis, cf, o);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) am[c] = add(am[c], o.m3[c]);
#pragma unroll
      for (int c = 0; c < 3; ++c) asc[c] = add(asc[c], o.sc[c]);
#pragma unroll
      for (int c = 0; c < 4; ++c) arot[c] = add(arot[c], o.rot[c]);
#pragma unroll
      for (int b = 0; b < 16; ++b)
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) ash[3 * b + ch] = add(ash[3 * b + ch], mul(basis[b], cf[ch]));
    }
    aop = add(aop, a.dL_dopacity[i]);
  }
  if (lane < n) {
    for (int c = 0; c < 3; ++c) a.g_means3D[3 * size_t(row) + c] = am[c];
    for (int c = 0; c < 3; ++c) a.g_scales[3 * size_t(row) + c] = asc[c];
    for (int c = 0; c < 4; ++c) a.g_rotations[4 * size_t(row) + c] = arot[c];
    a.g_opacity[row] = aop;
  }
  // dL/dSH rows [row0, row0 + n) ([rows, M, 3], contiguous) through shared
  // memory, so the warp's stores are one contiguous run
  __syncwarp();  // every lane is done with the staged input rows
  if (lane < n) {
#pragma unroll
    for (int c = 0; c < 48; ++c)
      if (c < rg) sw[lane * stride + c] = ash[c];
    for (int c = 48; c < rg; ++c) sw[lane * stride + c] = 0.f;  // bands beyond the 16th (none for M <= 16)
  }
  __syncwarp();
  float* dst = a.g_sh + size_t(row0) * rg;
  const int total = n * rg;
  int gr = 0, c = lane;
  while (c >= rg) { c -= rg; ++gr; }
  for (int e = lane; e < total; e += 32) {
    dst[e] = sw[gr * stride + c];
    c += 32;
    while (c >= rg) { c -= rg; ++gr; }
  }
}

}  // namespace

void launch_backward_groups(const BackwardArgs& a, cudaStream_t stream) {
  if (a.group_rows <= 0 || a.num_groups <= 0) return;
  const long long blocks = (a.group_rows + kGaussThreads - 1) / kGaussThreads;
  stage_begin(kStBwdGaussians, stream);
  launch_after(a.grad_mode == 1 ? gaussians_group_kernel<1> : gaussians_group_kernel<0>, unsigned(blocks),
               kGaussThreads, 0, stream, a);
  stage_end(kStBwdGaussians, stream, 1);
}

void launch_backward_render(const BackwardArgs& a, cudaStream_t stream) {
  const int tiles = a.items ? a.total_tiles : ((a.W + kTile - 1) / kTile) * ((a.H + kTile - 1) / kTile);
  if (tiles <= 0) return;
  stage_begin(kStBwdRender, stream);
  const bool da = a.dL_ddepth != nullptr || a.dL_dalpha != nullptr;  // a loss reaches depth or alpha
  const bool wide = ((reinterpret_cast<uintptr_t>(a.record) | reinterpret_cast<uintptr_t>(a.bwd_record)) & 31u) == 0u;
  auto launch = [&](auto kernel, auto narrow) {
    if (wide) launch_after(kernel, unsigned(tiles * 8), 32, 0, stream, a);
    else launch_after(narrow, unsigned(tiles * 8), 32, 0, stream, a);
  };
  if (a.grad_mode == 1) launch(render_bwd_kernel<ExactChain, true>, render_bwd_kernel<ExactChain, false>);
  else if (da) launch(render_bwd_kernel<RefChain<true>, true>, render_bwd_kernel<RefChain<true>, false>);
  else launch(render_bwd_kernel<RefChain<false>, true>, render_bwd_kernel<RefChain<false>, false>);
  stage_end(kStBwdRender, stream, 1);
}

void launch_backward_gaussians(const BackwardArgs& a, cudaStream_t stream) {
  if (a.P <= 0) return;
  const int blocks = (a.P + kGaussThreads - 1) / kGaussThreads;
  stage_begin(kStBwdGaussians, stream);
  launch_after(a.grad_mode == 1 ? gaussians_exact_kernel : gaussians_ref_kernel, unsigned(blocks), kGaussThreads, 0,
               stream, a);
  stage_end(kStBwdGaussians, stream, 1);
}

}  // namespace w2w
