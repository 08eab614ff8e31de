// Backward pass.
//
// Per-pixel pass (reference backward.cu:521-665): one CTA per tile, pixels
// walk the tile's list back to front, recomputing each pair's alpha from the
// stored state (final transmittance and last-contributor index) instead of
// storing per-pair values.  Each entry's per-pixel contributions are summed
// across the warp with shuffles and added with one atomic per warp (the
// reference issues ten atomics per pixel-Gaussian pair).  A tile starts at its
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

#include <type_traits>

namespace w2w {
namespace {

// Heavy tiles: each warp's walk is cut into kSplitWays segments, one CTA per
// segment.  The CTA of a segment first replays the state recurrences of the
// entries behind it (alpha and the transmittance / suffix updates only: no
// gradients, no reduction, about kReplayCost of a full entry's work) to reach
// the state at its segment's end, then walks its segment in full.  All CTAs
// compute the state with the same code in the same order, so each starts from
// exactly the state a single walk would have reached; only the order of the
// atomic additions changes.  Segment lengths (from the back) make the
// segments' work equal: L_0 = W, L_i = W - kReplayCost * (L_0 + ... + L_{i-1}).
// kSplitWays (2 or 3) and the number of split tiles are run-time tuning
// knobs (W2W_TUNE_BWD_WAYS, W2W_TUNE_BWD_SPLIT); only the order of the atomic
// additions depends on them.
constexpr float kReplayCost = 0.22f;

// List positions [lo, hi) of segment k (0 = the back-most) of a walk of
// length `walk`.
template <int kSplitWays>
__device__ __forceinline__ void segment_of(int walk, int k, int& lo, int& hi) {
  float len[kSplitWays], before = 0.f, total = 0.f;
#pragma unroll
  for (int i = 0; i < kSplitWays; ++i) {
    len[i] = 1.0f - kReplayCost * before;
    before += len[i];
  }
  total = before;
  float b0 = 0.f, b1 = 0.f;
#pragma unroll
  for (int i = 0; i < kSplitWays; ++i) {
    if (i < k) b0 += len[i];
    if (i <= k) b1 += len[i];
  }
  hi = walk - int(float(walk) * (b0 / total));
  lo = k == kSplitWays - 1 ? 0 : walk - int(float(walk) * (b1 / total));
  lo = max(0, min(lo, hi));
}

// ---------------------------------------------------------------------------
// Per-pixel pass.  One warp, and one CTA, per 8x4 pixel block, walking its
// block's part of the tile's list back to front, the entries its block mask
// names packed into groups of 32:
//
//   1. lane j gathers entry j's record (the next group's loads are in flight
//      while this one is evaluated) and puts it in shared memory;
//   2. every lane evaluates the group's entries in order for its pixel -- the
//      transmittance chain -- and writes two numbers per pair: u, from which
//      every geometric gradient of the pair follows, and w, the pair's colour
//      weight;
//   3. the 32 x 32 table of (u, w) is read across: lane j sums entry j over the
//      block's 32 pixels (the moments of u over the pixel offsets, and w times
//      each upstream plane), turns the sums into the entry's gradients and adds
//      each with one atomic.
//
// What bounds it: instruction issue, and for scenes that leave SMs idle the
// busiest warp's chain.  Summing across the warp in step 3 costs about 12
// instructions per entry; a shuffle tree per entry (ten values through 21
// shuffles per pair of entries, with their products computed per pixel) cost
// about 60, and groups of 32 mask-selected entries replace list chunks of 32
// of which a quarter were evaluated.  Four entries are evaluated together: their
// exponentials and reciprocals overlap, and only the chain of T and B runs
// through them (two together: 128.8 us per view against 119.3, 500k Gaussians,
// 512x512).  One-warp CTAs give a block's slot back when it ends; an eight-warp
// CTA held its registers until the slowest of its blocks had ended (two warps:
// 125.5 us, four: 139.6 with two entries together).  Sixteen CTAs per SM (128
// registers): 283 us at 1M / 1024x1024 and 336 us for a 12-view batch, against
// 299 and 359 at 150 registers; the busiest warps' chain, which a full SM slows,
// makes 500k / 512x512 124 us against 119.
// ---------------------------------------------------------------------------
constexpr int kBwdWarps = 1;               // blocks (warps) per CTA
constexpr int kBwdParts = 8 / kBwdWarps;   // CTAs per tile (and segment)
constexpr int kGroup = 32;                 // entries per group, one per lane
constexpr int kIlp = 4;                    // entries evaluated together

// A warp's shared memory.  The rows of `uw` are one pair longer than the
// group, so that reading down a column touches every bank once.
struct __align__(16) BwdWarp {
  float4 rec[kGroup * kRecVec];  // the group's records; the third float4's w is the entry's list position
  float4 up[32];                 // per pixel: upstream dL/dcolour and dL/ddepth
  float2 uw[kGroup][33];
  uint32_t slot[kGroup];         // list positions of the group being packed
};

// Positions [lo, top) of a block's part of a tile's list, highest first, in
// groups of up to 32.  words: the block's mask row, or null (each entry is
// tested against the block here).
struct BlockWalk {
  const uint32_t* words;
  const float* record;
  const uint32_t* list;   // the tile's first list entry
  uint32_t num_records;
  int bx, by, lo, top, wi, wb;
  uint32_t bits, cache;

  __device__ __forceinline__ void start(int lo_, int top_) {
    lo = lo_;
    top = top_;
    wi = ((top - 1) >> 5) + 1;  // words [0, wi) are still to come
    wb = wi;
    bits = 0;
  }
  // Word w's bits inside [lo, top).
  __device__ __forceinline__ uint32_t word(int w) {
    const int lane = threadIdx.x & 31;
    uint32_t b;
    if (words != nullptr) {
      if (w < wb) {  // 32 words at a time, one per lane
        wb = max(w - 31, 0);
        cache = wb + lane <= w ? __ldg(words + wb + lane) : 0u;
      }
      b = __shfl_sync(0xffffffffu, cache, w - wb);
    } else {
      const int pos = 32 * w + lane;
      bool reach = false;
      if (pos >= lo && pos < top) {
        const uint32_t id = __ldg(list + pos);
        if (id < num_records) {
          const float4* r = reinterpret_cast<const float4*>(record) + 4 * size_t(id);
          const float4 r0 = __ldg(r), r1 = __ldg(r + 1);  // the blend's record
          reach = block_test(r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, bx, by);
        }
      }
      b = __ballot_sync(0xffffffffu, reach);
    }
    const int above = top - 32 * w, below = lo - 32 * w;
    if (above < 32) b &= (1u << above) - 1u;
    if (below > 0) b &= 0xffffffffu << below;
    return b;
  }
  // Packs the next group's positions into slot[0, count), highest first.
  // Warp-collective; the caller has synchronised the warp after its last read of slot.
  __device__ __forceinline__ int next(uint32_t* slot) {
    const int lane = threadIdx.x & 31;
    int count = 0;
    if (top <= lo) return 0;
    const int first = lo >> 5;
    while (true) {
      if (bits == 0u) {
        if (wi <= first) break;
        bits = word(--wi);
        continue;
      }
      const int n = __popc(bits), room = kGroup - count;
      const int rank = __popc((bits >> lane) >> 1);  // set bits above this lane's
      const bool mine = (bits >> lane) & 1u;
      if (mine && rank < room) slot[count + rank] = uint32_t(32 * wi + lane);
      if (n > room) {
        bits = __ballot_sync(0xffffffffu, mine && rank >= room);
        count = kGroup;
        break;
      }
      count += n;
      bits = 0u;
      if (count == kGroup) break;
    }
    __syncwarp();
    return count;
  }
};

// Entry records of a group in flight: lane j's entry.
struct GroupLoad {
  float4 r0, r1, r2;
  uint32_t id;
  int count;
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
// when positive or below alpha 1/255, alpha = min(0.99, o G).
__device__ __forceinline__ bool ref_eval(float4 q0, float4 q1, float pxf, float pyf, float& G, float& alpha) {
  const float dx = q0.x - pxf, dy = q0.y - pyf;
  const float power = -0.5f * (q0.z * dx * dx + q1.x * dy * dy) - q0.w * dx * dy;
  G = expf(power);
  alpha = fminf(0.99f, q1.y * G);
  return power <= 0.0f && alpha >= 1.0f / 255.0f;
}

// Reference formulas (backward.cu:552-663) for one pixel; slots
// (mx, my, conic a, conic b), (conic c, opacity, depth, r), (g, b, skip, position).
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
  // Gaussian id's record as its slot's three float4s
  static __device__ __forceinline__ void gather(const BackwardArgs& a, uint32_t id, float4& r0, float4& r1, float4& r2) {
    const float4* r = reinterpret_cast<const float4*>(a.bwd_record) + 4 * size_t(id);
    r0 = __ldg(r);
    r1 = __ldg(r + 1);
    r2 = __ldg(r + 2);
  }

  // kIlp entries, in order, at e (past the group's end: records that contribute
  // nothing); o: u, w of each.  The evaluations are independent and overlap;
  // only T and B run through the entries.  kFull false: state only (the entries
  // behind a split tile's segment).
  template <bool kFull>
  __device__ __forceinline__ void step(const float4* e, const BwdPixel& p, float pxf, float pyf, float2 (&o)[kIlp]) {
    float G[kIlp], al[kIlp], y[kIlp], q[kIlp];
    bool ok[kIlp];
#pragma unroll
    for (int k = 0; k < kIlp; ++k) {
      const float4 q0 = e[kRecVec * k], q1 = e[kRecVec * k + 1], q2 = e[kRecVec * k + 2];
      ok[k] = ref_eval(q0, q1, pxf, pyf, G[k], al[k]) && __float_as_uint(q2.w) < p.last;
      y[k] = rcp_markstein(1.f - al[k]);
      q[k] = q1.w * p.dLp0 + q2.x * p.dLp1 + q2.y * p.dLp2;
      if constexpr (kDA) q[k] += q1.z * p.dLd + p.dLa;
    }
#pragma unroll
    for (int k = 0; k < kIlp; ++k) {
      // T / (1 - alpha), T in [~1e-4, 1] (the forward stops before T < 1e-4)
      // and 1 - alpha in [0.01, 1]: the quotient from the correctly rounded
      // reciprocal and one remainder correction
      const float t = T * y[k], Tn = fma(fma(-(1.f - al[k]), t, T), y[k], t);
      const float d = q[k] - B;
      // alpha <= 0.99 and T finite keep both factors finite; G itself may be
      // infinite where the entry is skipped
      if constexpr (kFull)
        o[k] = make_float2(ok[k] ? G[k] * (d * Tn - tf_bg * y[k]) : 0.f, ok[k] ? al[k] * Tn : 0.f);
      T = ok[k] ? Tn : T;
      B = ok[k] ? B + al[k] * d : B;
    }
  }

  // Lane j's entry over the block's 32 pixels, and its atomics.
  static __device__ __forceinline__ void reduce(const BackwardArgs& a, const BwdWarp& s, int j, uint32_t id, float bx,
                                                float by, float hW, float hH) {
    const float4 q0 = s.rec[kRecVec * j], q1 = s.rec[kRecVec * j + 1];
    float S = 0.f, Sx = 0.f, Sy = 0.f, Sxx = 0.f, Sxy = 0.f, Syy = 0.f, c0 = 0.f, c1 = 0.f, c2 = 0.f, cd = 0.f;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float dy = q0.y - (by + float(r));
      float rs = 0.f, rx = 0.f;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float2 uw = s.uw[j][8 * r + c];
        const float4 up = s.up[8 * r + c];
        const float dx = q0.x - (bx + float(c)), t = uw.x * dx;
        rs += uw.x;
        rx += t;
        Sxx += t * dx;
        c0 += uw.y * up.x;
        c1 += uw.y * up.y;
        c2 += uw.y * up.z;
        if constexpr (kDA) cd += uw.y * up.w;
      }
      S += rs;
      Sx += rx;
      Sxy += dy * rx;
      const float t = dy * rs;
      Sy += t;
      Syy += t * dy;
    }
    // no pixel of the block took the entry
    if (S == 0.f && Sxx == 0.f && Syy == 0.f && c0 == 0.f && c1 == 0.f && c2 == 0.f && cd == 0.f) return;
    const float h = -0.5f * q1.y;
    atomicAdd(a.dL_dcolors + 3 * size_t(id), c0);
    atomicAdd(a.dL_dcolors + 3 * size_t(id) + 1, c1);
    atomicAdd(a.dL_dcolors + 3 * size_t(id) + 2, c2);
    if constexpr (kDA) atomicAdd(a.acc_depth + id, cd);
    atomicAdd(a.dL_dmean2D + 3 * size_t(id), -q1.y * hW * (q0.z * Sx + q0.w * Sy));
    atomicAdd(a.dL_dmean2D + 3 * size_t(id) + 1, -q1.y * hH * (q1.x * Sy + q0.w * Sx));
    atomicAdd(a.acc_cov + 4 * size_t(id), h * Sxx);
    atomicAdd(a.acc_cov + 4 * size_t(id) + 1, h * Sxy);
    atomicAdd(a.acc_cov + 4 * size_t(id) + 3, h * Syy);
    atomicAdd(a.dL_dopacity + id, S);
  }
};

// The forward's Gaussian value (blend.cu), split at its division so that a
// warp's divisions can run branch-free together.
__device__ __forceinline__ float gauss_num_fwd(float px, float py, float mx, float my, float cxx, float cxy,
                                               float cyy) {
  using namespace fp;
  const float dx = sub(px, mx), dy = sub(py, my);
  const float tX = d2<BL_TX>(dx, cyy, dy, cxy);
  const float tY = s2<BL_TY>(-dx, cxy, dy, cxx);
  return s2<BL_NUM>(tX, dx, tY, dy);
}

// Exact derivative of the forward blend for one pixel; slots
// (mx, my, cxx, cxy), (cyy, det, opacity, depth), (r, g, b, position).  The
// suffix sums behind the current entry (colour including the background,
// depth, weight) enter only through their upstream-weighted sum D.
struct ExactChain {
  float T, D;
  __device__ __forceinline__ ExactChain(const BackwardArgs& a, const BwdPixel& p) {
    T = p.inside ? a.T_final[p.pix] : 0.0f;
    D = T * (p.bg[0] * p.dLp0 + p.bg[1] * p.dLp1 + p.bg[2] * p.dLp2);
  }
  static __device__ __forceinline__ void gather(const BackwardArgs& a, uint32_t id, float4& r0, float4& r1, float4& r2) {
    const float4* r = reinterpret_cast<const float4*>(a.record) + 4 * size_t(id);
    const float4 m = __ldg(r), o = __ldg(r + 1), c = __ldg(r + 2), dc = __ldg(r + 3);
    r0 = make_float4(m.x, m.y, c.x, c.y);
    r1 = make_float4(c.z, c.w, o.w, dc.x);
    r2 = make_float4(dc.y, dc.z, dc.w, 0.f);
  }

  // As RefChain::step.  u = dL/dalpha g: nothing passes the 0.99 clamp (a
  // negative mahalanobis distance, mapped to 1000 by the forward, has g = 0).
  template <bool kFull>
  __device__ __forceinline__ void step(const float4* e, const BwdPixel& p, float pxf, float pyf, float2 (&o)[kIlp]) {
    float num[kIlp], det[kIlp], opac[kIlp], q[kIlp];
    bool ok[kIlp], in_range = true;
#pragma unroll
    for (int k = 0; k < kIlp; ++k) {
      const float4 q0 = e[kRecVec * k], q1 = e[kRecVec * k + 1], q2 = e[kRecVec * k + 2];
      num[k] = gauss_num_fwd(pxf, pyf, q0.x, q0.y, q0.z, q0.w, q1.x);
      det[k] = q1.y;
      opac[k] = q1.z;
      in_range = in_range && div_in_range(num[k], q1.y);
      q[k] = q2.x * p.dLp0 + q2.y * p.dLp1 + q2.z * p.dLp2 + q1.w * p.dLd + p.dLa;
      ok[k] = __float_as_uint(q2.w) < p.last;
    }
    // the forward's Gaussian values (same division as the blend)
    float m[kIlp], g[kIlp], og[kIlp], ia[kIlp];
    if (__all_sync(0xffffffffu, in_range)) {
#pragma unroll
      for (int k = 0; k < kIlp; ++k) m[k] = div_markstein(num[k], det[k]);
    } else {
#pragma unroll
      for (int k = 0; k < kIlp; ++k) m[k] = div(num[k], det[k]);
    }
#pragma unroll
    for (int k = 0; k < kIlp; ++k) {
      g[k] = expf(mul(-0.5f, m[k] < 0.0f ? 1000.0f : m[k]));
      og[k] = mul(opac[k], g[k]);
      ok[k] = ok[k] && og[k] >= 1.0f / 255.0f;
      ia[k] = rcp_markstein(1.0f - fminf(0.99f, og[k]));  // 1 - alpha in [0.01, 1]
    }
#pragma unroll
    for (int k = 0; k < kIlp; ++k) {
      const float al = fminf(0.99f, og[k]);
      const float Tn = T * ia[k];  // transmittance in front of this entry
      const float aT = al * Tn;
      if constexpr (kFull)
        o[k] = make_float2(ok[k] && og[k] < 0.99f ? (q[k] * Tn - D * ia[k]) * g[k] : 0.f, ok[k] ? aT : 0.f);
      T = ok[k] ? Tn : T;
      D = ok[k] ? D + q[k] * aT : D;
    }
  }

  // With e = cyy dx - cxy dy and f = cxx dy - cxy dx (offsets from the mean),
  // d(num / det) = 2 (e, f) / det over the offsets and -(e e, 2 e f, f f) / det^2
  // over the covariance.
  static __device__ __forceinline__ void reduce(const BackwardArgs& a, const BwdWarp& s, int j, uint32_t id, float bx,
                                                float by, float hW, float hH) {
    const float4 q0 = s.rec[kRecVec * j], q1 = s.rec[kRecVec * j + 1];
    float S = 0.f, Se = 0.f, Sf = 0.f, See = 0.f, Sef = 0.f, Sff = 0.f, c0 = 0.f, c1 = 0.f, c2 = 0.f, cd = 0.f;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float dy = (by + float(r)) - q0.y, ey = -q0.w * dy, fy = q0.z * dy;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float2 uw = s.uw[j][8 * r + c];
        const float4 up = s.up[8 * r + c];
        const float dx = (bx + float(c)) - q0.x;
        const float e = q1.x * dx + ey, f = fy - q0.w * dx;
        const float te = uw.x * e, tf = uw.x * f;
        S += uw.x;
        Se += te;
        Sf += tf;
        See += te * e;
        Sef += te * f;
        Sff += tf * f;
        c0 += uw.y * up.x;
        c1 += uw.y * up.y;
        c2 += uw.y * up.z;
        cd += uw.y * up.w;
      }
    }
    if (S == 0.f && See == 0.f && Sff == 0.f && c0 == 0.f && c1 == 0.f && c2 == 0.f && cd == 0.f) return;
    // det >= 0.09 (the forward's +0.3 low-pass on a positive semi-definite
    // covariance), where rcp_markstein is the correctly rounded 1/det
    const float idet = rcp_markstein(q1.y), k1 = q1.z * idet, k2 = k1 * idet;
    atomicAdd(a.dL_dcolors + 3 * size_t(id), c0);
    atomicAdd(a.dL_dcolors + 3 * size_t(id) + 1, c1);
    atomicAdd(a.dL_dcolors + 3 * size_t(id) + 2, c2);
    atomicAdd(a.acc_depth + id, cd);
    atomicAdd(a.dL_dmean2D + 3 * size_t(id), k1 * hW * Se);
    atomicAdd(a.dL_dmean2D + 3 * size_t(id) + 1, k1 * hH * Sf);
    atomicAdd(a.acc_cov + 4 * size_t(id), 0.5f * k2 * See);
    atomicAdd(a.acc_cov + 4 * size_t(id) + 1, k2 * Sef);
    atomicAdd(a.acc_cov + 4 * size_t(id) + 2, 0.5f * k2 * Sff);
    atomicAdd(a.dL_dopacity + id, S);
  }
};

// Pixel-loop prologue for block `block` of tile `tile`: the call's image, or
// its batch item's.
__device__ __forceinline__ BwdPixel make_bwd_pixel(const BackwardArgs& a, int tile, int block) {
  if (a.items == nullptr) return BwdPixel(a, tile, tile, block, a.W, a.H, 0, a.bg);
  const BatchItem& it = a.items[find_item_tile(a.items, a.num_items, uint32_t(tile))];
  return BwdPixel(a, tile, tile - int(it.tile_base), block, it.W, it.H, size_t(it.pix_base), it.bg);
}

// Work item b's tile and segment: the first kSplitWays * split items are the
// segments of the `split` heaviest tiles (segment 0..kSplitWays-1), the rest
// one whole tile each (segment -1), heaviest first.
template <int kSplitWays>
__device__ __forceinline__ int item_tile(const BackwardArgs& a, int b, int& seg) {
  if (b < kSplitWays * a.split) {
    seg = b % kSplitWays;
    return int(a.order_bwd[b / kSplitWays]);
  }
  seg = -1;
  return int(a.order_bwd[b - (kSplitWays - 1) * a.split]);
}

template <typename Chain, int kSplitWays>
__global__ void __launch_bounds__(32 * kBwdWarps, 16 / kBwdWarps) render_bwd_kernel(BackwardArgs a) {
  __shared__ BwdWarp s_warp[kBwdWarps];
  int seg;
  const int tile = item_tile<kSplitWays>(a, int(blockIdx.x) / kBwdParts, seg);
  const int warp = int(threadIdx.x >> 5), lane = int(threadIdx.x & 31);
  const int block = (int(blockIdx.x) % kBwdParts) * kBwdWarps + warp;
  const BwdPixel p = make_bwd_pixel(a, tile, block);
  if (p.walk <= 0) return;  // warp-uniform
  BwdWarp& s = s_warp[warp];
  s.up[lane] = make_float4(p.dLp0, p.dLp1, p.dLp2, p.dLd);
  Chain ch(a, p);
  const float pxf = float(p.tp.px), pyf = float(p.tp.py);
  const float hW = 0.5f * float(p.W), hH = 0.5f * float(p.H);
  const uint32_t* list = a.point_list + p.range.x;
  BlockWalk walk;
  // the blend's block masks, when this binning state has them
  const bool use_masks = a.masks_valid != nullptr && *a.masks_valid != 0u;
  walk.words = use_masks ? a.masks + mask_row(p.range.x, tile, int(p.range.y - p.range.x), block) : nullptr;
  walk.record = a.record;
  walk.list = list;
  walk.num_records = uint32_t(a.P);
  walk.bx = p.tp.bx;
  walk.by = p.tp.by;

  // Positions of the next group, and lane j's id in it (an id of num_records
  // or more -- a list left inconsistent by a sort whose bounded wait ran out,
  // which its error word reports -- is skipped, never read).
  auto pack = [&](uint32_t& pos, uint32_t& id) {
    __syncwarp();
    const int n = walk.next(s.slot);
    pos = lane < n ? s.slot[lane] : 0u;
    id = lane < n ? __ldg(list + pos) : ~0u;
    return n;
  };
  auto gather = [&](GroupLoad& g, uint32_t pos, uint32_t id, int n) {
    g.id = id;
    g.count = n;
    g.r0 = g.r1 = g.r2 = make_float4(0.f, 0.f, 0.f, 0.f);  // opacity 0: contributes nothing
    if (id < uint32_t(a.P)) Chain::gather(a, id, g.r0, g.r1, g.r2);
    g.r2.w = __uint_as_float(id < uint32_t(a.P) ? pos : ~0u);  // past every pixel's last contributor
  };
  auto run = [&](int lo, int top, auto full) {
    constexpr bool kFull = decltype(full)::value;
    walk.start(lo, top);
    GroupLoad g;
    uint32_t pos, id;
    int n = pack(pos, id);
    gather(g, pos, id, n);
    n = n > 0 ? pack(pos, id) : 0;
    while (g.count > 0) {
      const int count = g.count;
      const uint32_t cur = g.id;
      s.rec[kRecVec * lane] = g.r0;
      s.rec[kRecVec * lane + 1] = g.r1;
      s.rec[kRecVec * lane + 2] = g.r2;
      gather(g, pos, id, n);             // the next group's records and
      n = n > 0 ? pack(pos, id) : 0;     // the ids of the one after it are in flight below
      __syncwarp();
      for (int j = 0; j < count; j += kIlp) {
        float2 o[kIlp];
        ch.template step<kFull>(s.rec + kRecVec * j, p, pxf, pyf, o);
        if constexpr (kFull) {
#pragma unroll
          for (int k = 0; k < kIlp; ++k) s.uw[j + k][lane] = o[k];
        }
      }
      __syncwarp();
      if constexpr (kFull) {
        if (lane < count && cur < uint32_t(a.P))
          Chain::reduce(a, s, lane, cur, float(p.tp.bx), float(p.tp.by), hW, hH);
        __syncwarp();
      }
    }
  };
  if (seg < 0) {
    run(0, p.walk, std::true_type{});
  } else {
    int lo, hi;
    segment_of<kSplitWays>(p.walk, seg, lo, hi);
    run(hi, p.walk, std::false_type{});
    __syncwarp();
    run(lo, hi, std::true_type{});
  }
}

// ---------------------------------------------------------------------------
// Per-Gaussian passes: one thread per Gaussian, with the SH rows (up to 48
// floats each) moved between global and shared memory by the whole warp, so
// that global loads and stores are contiguous 128-byte runs instead of one
// 192-byte-strided row per thread.
// ---------------------------------------------------------------------------
constexpr int kGaussThreads = 128;

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

// Write the span of 32 rows of `len` floats at dst: row g's element c is
// coefficient (c + off) / 3, channel (c + off) % 3 of Gaussian g, the product of
// its basis value and colour factor in s (row g at g * 21: 16 basis, 3 factors).
__device__ __forceinline__ void store_span(float* dst, int len, const float* s, int off) {
  const int lane = threadIdx.x & 31, nf = 8 * len;
  float4* q = reinterpret_cast<float4*>(dst);
  for (int f = lane; f < nf; f += 32) {
    int g = (4 * f) / len, c = 4 * f - g * len;
    float o[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const int e = c + off, k = e / 3, ch = e - 3 * k;
      o[w] = s[g * 21 + k] * s[g * 21 + 16 + ch];
      if (++c == len) {
        c = 0;
        ++g;
      }
    }
    q[f] = make_float4(o[0], o[1], o[2], o[3]);
  }
}

// dsh rows [i0, i0 + n) ([P, M, 3]) = basis[k] * cf[ch] (k < 16; 0 beyond),
// written contiguously; each thread's factors pass through s.  Warp-collective.
__device__ __forceinline__ void sh_store_outer(float* dsh, int M, int i0, int n, float* s, const float (&basis)[16],
                                               const float (&cf)[3], bool active) {
  constexpr int kRow = 21;  // 16 basis + 3 colour factors, odd stride
  const int lane = threadIdx.x & 31, rg = 3 * M;
  __syncwarp();  // the SH rows in s have been read
#pragma unroll
  for (int k = 0; k < 16; ++k) s[lane * kRow + k] = active ? basis[k] : 0.f;
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) s[lane * kRow + 16 + ch] = active ? cf[ch] : 0.f;
  __syncwarp();
  if (M == 16 && n == 32 && aligned16(dsh)) {
    store_span(dsh + size_t(i0) * 48, 48, s, 0);
    return;
  }
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
__device__ __forceinline__ void sh_stage_in_raw(const float* dc, const float* ac, int M, int i0, int n, float* s,
                                                int stride) {
  constexpr int kInFlight = 8;
  const int rs = 3 * (M < 16 ? M : 16), ra = 3 * (M - 1), lane = threadIdx.x & 31;
  if (M == 16 && n == 32 && aligned16(dc) && aligned16(ac)) {
    stage_span(dc + size_t(i0) * 3, 3, s, stride, 0);
    stage_span(ac + size_t(i0) * 45, 45, s, stride, 3);
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
}

// sh_store_outer for the raw path: coefficient 0 to ddc, the rest to dac.
__device__ __forceinline__ void sh_store_outer_raw(float* ddc, float* dac, int M, int i0, int n, float* s,
                                                   const float (&basis)[16], const float (&cf)[3], bool active) {
  constexpr int kRow = 21;
  const int lane = threadIdx.x & 31, rg = 3 * M, ra = 3 * (M - 1);
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 16; ++k) s[lane * kRow + k] = active ? basis[k] : 0.f;
#pragma unroll
  for (int ch = 0; ch < 3; ++ch) s[lane * kRow + 16 + ch] = active ? cf[ch] : 0.f;
  __syncwarp();
  if (M == 16 && n == 32 && aligned16(ddc) && aligned16(dac)) {
    store_span(ddc + size_t(i0) * 3, 3, s, 0);
    store_span(dac + size_t(i0) * 45, 45, s, 3);
    return;
  }
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
      const float w = __ldg(&quat[4 * gi]), x = __ldg(&quat[4 * gi + 1]), y = __ldg(&quat[4 * gi + 2]),
                  z = __ldg(&quat[4 * gi + 3]);
      const float inv = __frcp_rn(fmaxf(sqrtf((w * w + y * y) + (x * x + z * z)), 1e-12f));
      return make_float4(w * inv, x * inv, y * inv, z * inv);
    }
    return make_float4(__ldg(&rotations[4 * gi]), __ldg(&rotations[4 * gi + 1]), __ldg(&rotations[4 * gi + 2]),
                       __ldg(&rotations[4 * gi + 3]));
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

// One Gaussian (radius > 0) of the reference-formula pass: every output but
// dL_dsh, plus the SH basis and masked colour gradient dL_dsh is built from.
// sh_row: this Gaussian's SH coefficients (staged in shared memory).
__device__ __forceinline__ void ref_gaussian(const BackwardArgs& a, int i, const GView& gv, const float* sh_row, float (&basis)[16],
                                             float (&cf)[3], GOut& o) {
  const int M = a.M;
  const float* mats = gv.mats;
  const float* cam = mats + 32;
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
  float dc[6];
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
  float sd[3] = {view[0] * gvx + view[1] * gvy + view[2] * gvz, view[4] * gvx + view[5] * gvy + view[6] * gvz,
                 view[8] * gvx + view[9] * gvy + view[10] * gvz};

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
    const float q0 = __ldg(&gv.quat[4 * gv.gi]), q1 = __ldg(&gv.quat[4 * gv.gi + 1]),
                q2 = __ldg(&gv.quat[4 * gv.gi + 2]), q3 = __ldg(&gv.quat[4 * gv.gi + 3]);
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

// 8 CTAs per SM (64 registers, no spills; shared memory allows 9): more
// Gaussians' loads in flight (0.452 -> 0.415 ms per 4-view step against the
// default 6 CTAs at 80 registers).
__global__ void __launch_bounds__(kGaussThreads, 8) gaussians_ref_kernel(BackwardArgs a) {
  __shared__ float s_sh[kGaussThreads / 32][32 * kShStride];
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
    if (a.sh_dc != nullptr) sh_stage_in_raw(a.sh_dc, a.sh_ac, a.M, i0, n, sw, stride);
    else sh_stage_in(a.shs, a.M, i0, n, sw, stride);
  } else {
    batch_sh_stage_in(a, i0, n, sw, stride);
  }
  float basis[16], cf[3] = {0.f, 0.f, 0.f};
  const bool active = lane < n && a.radii[i] > 0;
  if (active) {
    GOut o;
    ref_gaussian(a, i, gv, sw + lane * stride, basis, cf, o);
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
  __shared__ float s_sh[kGaussThreads / 32][32 * kShStride];
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
  __shared__ float s_sh[kGaussThreads / 32][32 * kShStride];
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
      else ref_gaussian(a, int(i), gv, sh_row, basis, cf, o);
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
  if (a.grad_mode == 1) gaussians_group_kernel<1><<<unsigned(blocks), kGaussThreads, 0, stream>>>(a);
  else gaussians_group_kernel<0><<<unsigned(blocks), kGaussThreads, 0, stream>>>(a);
  stage_end(kStBwdGaussians, stream, 1);
}

void launch_backward_render(const BackwardArgs& a, cudaStream_t stream) {
  const int tiles = a.items ? a.total_tiles : ((a.W + kTile - 1) / kTile) * ((a.H + kTile - 1) / kTile);
  if (tiles <= 0) return;
  BackwardArgs b = a;
  int sms = 148, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // the heaviest tiles by largest contributor count: knob quarters of the SM count
  b.split = min(tiles / 4, sms * tune_value(kTuneBwdSplit) / 4);
  const int ways = tune_value(kTuneBwdWays);
  stage_begin(kStBwdRender, stream);
  const int grid = (tiles + (ways - 1) * b.split) * kBwdParts;
  const bool da = a.dL_ddepth != nullptr || a.dL_dalpha != nullptr;  // a loss reaches depth or alpha
  auto launch = [&](auto kernel) { kernel<<<grid, 32 * kBwdWarps, 0, stream>>>(b); };
  if (ways == 3) {
    if (a.grad_mode == 1) launch(render_bwd_kernel<ExactChain, 3>);
    else if (da) launch(render_bwd_kernel<RefChain<true>, 3>);
    else launch(render_bwd_kernel<RefChain<false>, 3>);
  } else {
    if (a.grad_mode == 1) launch(render_bwd_kernel<ExactChain, 2>);
    else if (da) launch(render_bwd_kernel<RefChain<true>, 2>);
    else launch(render_bwd_kernel<RefChain<false>, 2>);
  }
  stage_end(kStBwdRender, stream, 1);
}

void launch_backward_gaussians(const BackwardArgs& a, cudaStream_t stream) {
  if (a.P <= 0) return;
  const int blocks = (a.P + kGaussThreads - 1) / kGaussThreads;
  stage_begin(kStBwdGaussians, stream);
  if (a.grad_mode == 1) gaussians_exact_kernel<<<blocks, kGaussThreads, 0, stream>>>(a);
  else gaussians_ref_kernel<<<blocks, kGaussThreads, 0, stream>>>(a);
  stage_end(kStBwdGaussians, stream, 1);
}

}  // namespace w2w
