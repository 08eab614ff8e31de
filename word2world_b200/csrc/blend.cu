// Per-tile front-to-back alpha blending (reference pixelGaussiansFull.cu:3-98,
// pixelGaussiansDev.cuh:5-96, gaussEval.h:7-29).
//
// One warp per 8x4 pixel block (tile_walk.cuh), one thread per pixel.  Each
// warp walks the tile's list on its own, tests every entry against its block,
// evaluates the ones that can reach it with alpha >= 1/255, 32 at a time (all
// their alphas at the block's pixels before the sequential transmittance and
// colour updates), and stops when its pixels have all terminated (the
// reference keeps loading every batch of the tile).
//
// Per pixel the arithmetic is the reference's, in its operation order: the
// Gaussian is evaluated from the 2-D covariance and its determinant
// (mahalanobis / det, negative -> 1000), alpha = min(0.99, o*g), entries with
// alpha < 1/255 are skipped, the pixel terminates before the entry that would
// take transmittance below 1e-4, colour accumulates with fma, and the
// contributor count is the 1-based index of the last blended entry.
#include "common.cuh"
#include "kernels.h"
#include "tile_walk.cuh"
#include "tma.cuh"

#include <algorithm>
#include <mutex>
#include <type_traits>

namespace w2w {
namespace {

constexpr int kBlendIlp = 4;  // list entries the queue-fed blend evaluates together per warp

struct BlendPixel {
  float C0 = 0.f, C1 = 0.f, C2 = 0.f, Wt = 0.f, D = 0.f, T = 1.0f;
  uint32_t last = 0;
  bool done;

  // Eight entries of the list in order: alphas `v` (0 where an entry is skipped
  // or the pixel has terminated), depths and colours dc[k]; `at` becomes e + k of
  // the last one blended.  Only the transmittance runs through them: it never
  // grows, so the entry that would take it below 1e-4 and all after it are the
  // ones whose product lies below, and their weight is 0.  Weight 0 keeps an entry
  // out by multiplication while its depth and colour are finite; kSelect: by
  // selection.
  template <bool kSelect>
  __device__ __forceinline__ void step(const float (&v)[8], const float4* dc, int e, int& at) {
    float t = T;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float nT = mul(t, sub(1.0f, v[k]));
      const bool alive = nT >= 0.0001f;
      const float aT = alive ? mul(v[k], t) : 0.0f;
      const float4 q = kSelect && aT == 0.0f ? make_float4(0.f, 0.f, 0.f, 0.f) : dc[k];
      C0 = fma(q.y, aT, C0);
      C1 = fma(q.z, aT, C1);
      C2 = fma(q.w, aT, C2);
      Wt = add(Wt, aT);
      D = s1<fp::BL_DEPTH>(q.x, aT, D);
      T = alive ? nT : T;
      at = aT > 0.0f ? e + k : at;
      t = nT;
    }
    done = done || t < 0.0001f;
  }

  // Entry with alpha `al` and depth and colour `dc`, 1-based list position `pos`.
  // Branch-free: the updates are selected, so a warp's lanes never diverge.
  // An entry that does not accumulate adds exactly zero: its weight aT is
  // selected to 0, colours and depth are finite (or, kSelect, selected to 0 too),
  // and C, Wt and D are never -0 (non-negative colours and weights, positive
  // depths), so x + c * 0 = x.
  template <bool kSelect>
  __device__ __forceinline__ void step(float al, float4 dc, uint32_t pos) {
    const bool blend = !done && al >= 1.0f / 255.0f;
    const float nT = mul(T, sub(1.0f, al));
    const bool term = blend && nT < 0.0001f;
    const bool acc = blend && !term;
    const float aT = acc ? mul(al, T) : 0.0f;
    if (kSelect && !acc) dc = make_float4(0.f, 0.f, 0.f, 0.f);
    C0 = fma(dc.y, aT, C0);
    C1 = fma(dc.z, aT, C1);
    C2 = fma(dc.w, aT, C2);
    Wt = add(Wt, aT);
    D = s1<fp::BL_DEPTH>(dc.x, aT, D);
    T = acc ? nT : T;
    last = acc ? pos : last;
    done = done || term;
  }
};

// kBlendIlp Gaussian values' alphas at one pixel: entry k's position and
// opacity (mx, my, opacity) and its covariance (cxx, cxy, cyy, det).
// Warp-collective: the branch-free division when every lane's operands allow it.
__device__ __forceinline__ void blend_alphas(const float4 (&m)[kBlendIlp], const float4 (&cov)[kBlendIlp], float pxf,
                                             float pyf, float (&al)[kBlendIlp]) {
  float num[kBlendIlp], d[kBlendIlp];
  bool in_range = true;
#pragma unroll
  for (int k = 0; k < kBlendIlp; ++k) {
    num[k] = gauss_num(pxf, pyf, m[k].x, m[k].y, cov[k].x, cov[k].y, cov[k].z);
    in_range = in_range && div_in_range(num[k], cov[k].w);
  }
  if (__all_sync(0xffffffffu, in_range)) {
#pragma unroll
    for (int k = 0; k < kBlendIlp; ++k) d[k] = div_markstein(num[k], cov[k].w);
  } else {
#pragma unroll
    for (int k = 0; k < kBlendIlp; ++k) d[k] = div(num[k], cov[k].w);
  }
#pragma unroll
  for (int k = 0; k < kBlendIlp; ++k) al[k] = fminf(0.99f, mul(m[k].z, gauss_from_m(d[k])));
}

constexpr int kBlendWarps = 1;      // blocks (warps) per CTA
constexpr int kBlendResident = 16;  // warps per SM the registers are sized for
constexpr int kTestChunks = 4;      // 32-entry chunks tested together
constexpr int kRing = 256;          // waiting entries: a group of 32, up to 31 after it and 128 newly tested
constexpr int kAlphaStride = 36;    // floats per pixel row of the alpha table: rows start on 16 bytes, 8 rows cover the banks

// A warp's shared memory.
struct __align__(16) BlendWarp {
  float alpha[33 * kAlphaStride];  // [pixel of the block][entry of the group], and a row of zeros
  float4 dc[32];                   // the group's depths and colours
  uint2 ring[kRing];               // entries that can reach the block: (id, 1-based list position)
};

// A lane's entry of the group to evaluate next: its record.
struct BlendEntry {
  float4 m, c, dc;  // (mx, my, opacity, _), (cxx, cxy, cyy, det), (depth, r, g, b)
};

// Alphas of a group's entries at the block's 32 pixels, into the alpha table (0
// where an entry is skipped): gauss_values' lanes and pixels.
template <int kLanes>
__device__ __forceinline__ void group_alphas(BlendWarp& s, const BlendEntry& en, float bx, float by) {
  const int e = int(threadIdx.x & 31u) % (32 / kLanes);
  gauss_values<kLanes>(en.m.x, en.m.y, en.c, bx, by, [&](int p, float g) {
    const float al = fminf(0.99f, mul(en.m.z, g));
    s.alpha[p * kAlphaStride + e] = al >= 1.0f / 255.0f ? al : 0.0f;
  });
}

// One CTA per kBlendWarps blocks of a tile; its warps never wait for one
// another.  A warp tests the tile's entries against its block 128 at a time
// (four per lane; the next 128 entries' culling sectors, and the ids of the 128
// after them, are in flight meanwhile) and queues the ones that can reach it;
// the ballots of the tests are the block's mask words for the backward.  It
// takes them from the queue 32 at a time: every lane evaluates one entry at all
// 32 pixels (group_alphas), the next group's records are requested, and then
// every lane runs its pixel through the group's alphas.
//
// What bounds it: at 500k Gaussians instruction issue (about 24 instructions
// per entry and 32 pixels for the alphas, 16 for the pixels' chains, 1.3 per
// tested entry); at small scenes, and at the end of large ones, the busiest
// warp's chain.
template <bool kWide>
__global__ void __launch_bounds__(32 * kBlendWarps, kBlendResident / kBlendWarps) blend_kernel(BlendArgs a) {
  grid_wait();
  constexpr int kParts = 8 / kBlendWarps;  // CTAs per tile
  __shared__ BlendWarp s_warp[kBlendWarps];
  const int tile = int(a.order[blockIdx.x / kParts]);
  const int warp = int(threadIdx.x >> 5);
  const int block = (int(blockIdx.x) % kParts) * kBlendWarps + warp;
  // this tile's image: the call's, or its batch item's
  int W = a.W, H = a.H, ltile = tile;
  size_t pbase = 0;
  const float* bg = a.bg;
  if (a.items != nullptr) {
    const BatchItem& it = a.items[find_item_tile(a.items, a.num_items, uint32_t(tile))];
    W = it.W;
    H = it.H;
    ltile = tile - int(it.tile_base);
    pbase = size_t(it.pix_base);
    bg = it.bg;
  }
  const TilePixel tp(ltile, (W + kTile - 1) / kTile, block);
  const int lane = tp.lane;
  const bool inside = tp.px < W && tp.py < H;
  const uint2 range = a.ranges[tile];
  const int n = int(range.y - range.x);
  const uint32_t* ids = a.point_list + range.x;
  const float4* records = reinterpret_cast<const float4*>(a.record);
  uint32_t* row = a.masks == nullptr ? nullptr : a.masks + mask_row(range.x, tile, n, block);
  BlendWarp& s = s_warp[warp];
  const uint32_t lt = lanemask_lt();
  s.alpha[32 * kAlphaStride + lane] = 0.0f;

  BlendPixel pix;
  pix.done = !inside;
  bool done = __all_sync(0xffffffffu, pix.done) != 0;
  const int chunks = done ? 0 : (n + 31) >> 5;
  // the culling sectors of the chunks to test next (lane j: entry j of each),
  // their ids and the ids of the chunks after them.  An id of num_records or
  // more (a list left inconsistent by a sort whose bounded wait ran out, which
  // its error word reports) is skipped, never read.
  uint32_t id[kTestChunks], id_next[kTestChunks];
  float4 t0[kTestChunks], t1[kTestChunks];
  auto load_ids = [&](int c) {
#pragma unroll
    for (int q = 0; q < kTestChunks; ++q) {
      const int e = 32 * (c + q) + lane;
      id_next[q] = e < n ? __ldg(ids + e) : ~0u;
    }
  };
  auto load_tests = [&]() {
#pragma unroll
    for (int q = 0; q < kTestChunks; ++q) {
      id[q] = id_next[q];
      t0[q] = make_float4(0.f, 0.f, -1.f, 0.f);  // hy < 0: reaches nothing
      t1[q] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (id[q] < a.num_records) {
        ldg32<kWide>(records + 4 * size_t(id[q]), t0[q], t1[q]);
      }
    }
  };
  int c = 0;                    // next chunk to test
  uint32_t head = 0, tail = 0;  // queue: [head, tail)
  uint32_t word = 0;            // lane l: the mask word of chunk 32 * (c / 32) + l
  // Tests chunks until 32 entries wait or the list ends.
  auto refill = [&]() {
    while (tail - head < 32u && c < chunks) {
#pragma unroll
      for (int q = 0; q < kTestChunks; ++q) {
        const bool reach = block_test(t0[q].x, t0[q].y, t0[q].z, t0[q].w, t1[q].x, t1[q].y, t1[q].z, tp.bx, tp.by);
        const uint32_t bits = __ballot_sync(0xffffffffu, reach);
        if (lane == ((c + q) & 31)) word = bits;
        if (reach) s.ring[(tail + __popc(bits & lt)) & (kRing - 1)] = make_uint2(id[q], uint32_t(32 * (c + q) + lane + 1));
        tail += __popc(bits);
      }
      c += kTestChunks;
      load_tests();
      load_ids(c + kTestChunks);
      // a full set of 32 words, or the list's last ones
      if (row != nullptr && ((c & 31) == 0 || c >= chunks)) {
        const int w = ((c - 1) & ~31) + lane;
        if (w < chunks) row[w] = word;
      }
    }
    __syncwarp();
  };
  // The lane's entry of the next group: `count` entries from `head`, spread over the lanes as group_alphas wants them.
  BlendEntry en;
  auto load_group = [&](int count) {
    const int e = count > 16 ? lane : count > 8 ? lane & 15 : lane & 7;
    // past the count: opacity 0, so alpha 0, and operands in gauss_values' range
    en.m = make_float4(-1024.f, -1024.f, 0.f, 0.f);
    en.c = make_float4(1.f, 0.f, 1.f, 1.f);
    en.dc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (e < count) {
      const float4* r = records + 4 * size_t(s.ring[(head + uint32_t(e)) & (kRing - 1)].x);
      float4 o;
      ldg32<kWide>(r, en.m, o);
      en.m.z = o.w;
      ldg32<kWide>(r + 2, en.c, en.dc);
    }
  };
  int count = 0;
  if (chunks > 0) {
    load_ids(0);
    load_tests();
    load_ids(kTestChunks);
    refill();
    count = int(min(tail - head, 32u));
    load_group(count);
  }
  auto run = [&](auto select) {
    while (count > 0 && !done) {
      if (count > 16) group_alphas<1>(s, en, float(tp.bx), float(tp.by));
      else if (count > 8) group_alphas<2>(s, en, float(tp.bx), float(tp.by));
      else group_alphas<4>(s, en, float(tp.bx), float(tp.by));
      s.dc[lane] = en.dc;
      const uint32_t first = head;
      head += uint32_t(count);
      refill();  // synchronises the warp
      const int next = int(min(tail - head, 32u));
      load_group(next);
      const float* mine = s.alpha + (pix.done ? 32 : lane) * kAlphaStride;  // a terminated pixel: zeros
      int at = -1;  // this pixel's last blended entry of the group
      for (int e = 0; e < count; e += 8) {
        const float4 a0 = *reinterpret_cast<const float4*>(mine + e), a1 = *reinterpret_cast<const float4*>(mine + e + 4);
        const float v[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        pix.template step<decltype(select)::value>(v, s.dc + e, e, at);
        if (pix.done) mine = s.alpha + 32 * kAlphaStride;
      }
      if (at >= 0) pix.last = s.ring[(first + uint32_t(at)) & (kRing - 1)].y;
      done = __all_sync(0xffffffffu, pix.done) != 0;
      __syncwarp();
      count = next;
    }
  };
  if (a.wild == nullptr || *a.wild == 0u) run(std::false_type{});
  else run(std::true_type{});
  // the mask words not yet written (the backward reads none past the last contributor)
  if (row != nullptr && (c & 31) != 0 && c < chunks && lane < (c & 31)) row[(c & ~31) + lane] = word;
  if (inside) {
    const size_t q = size_t(tp.py) * W + tp.px;
    const size_t p = pbase + q, cp = 3 * pbase + q;
    const size_t hw = size_t(W) * H;
    a.n_contrib[p] = pix.last;
    a.out_alpha[p] = pix.Wt;
    a.out_depth[p] = pix.D;
    a.T_final[p] = pix.T;
    a.out_color[cp] = fma(pix.T, bg[0], pix.C0);
    a.out_color[hw + cp] = fma(pix.T, bg[1], pix.C1);
    a.out_color[2 * hw + cp] = fma(pix.T, bg[2], pix.C2);
  }
  // largest contributor count in the tile, for inspection of the image state (the
  // backward's blocks start at their own pixels' counts); the tile's warps combine
  // theirs (tile_max is cleared before the launch)
  const uint32_t wm = __reduce_max_sync(0xffffffffu, pix.last);
  if (lane == 0 && wm != 0u) atomicMax(&a.tile_max[tile], wm);
}

// ---------------------------------------------------------------------------
// Persistent blend over a device tile queue, staged by TMA row gathers.
//
// A CTA runs kW consumer warps (the blocks of one tile half, or of the whole
// tile for kW = 8) and one producer warp, for as long as the queue (tile
// halves in the heaviest-first order; every item of a batched call in one
// queue) has items.  The producer takes the next item with an atomic, reads
// a batch's Gaussian ids from the list, writes the stage's header and the
// bit mask of its valid entries, and gathers the entries' 64-byte records into
// one of kQStages shared-memory stages with TMA (four rows per gather),
// completing on the stage's barrier.  Each consumer warp waits for that
// barrier, tests the staged entries against its own 8x4 block (block_test,
// as the backward's warps do), walks the ones that can reach it as the
// per-tile kernel does, and releases the stage.  A warp whose pixels have all
// terminated tells the producer, which skips the rest of a tile once every
// consumer warp has.  The stages run across tile boundaries, so a CTA never
// drains its pipeline between tiles, and no warp waits at a CTA barrier for
// the slowest warp of a batch: warps drift apart by up to kQStages batches.
// This blend writes no block masks: it clears the binning state's flag, and
// the backward tests each entry itself.
// Every wait is bounded; one that runs out sets kErrTimeout in `error`, and
// the CTA stops after its copies in flight land.  Results are bit-identical
// to blend_kernel's (same entries, same order).
// ---------------------------------------------------------------------------
constexpr int kQStages = 3;
constexpr int kQRec = 4;  // float4s per staged record (the whole record)

struct QueueStage {
  int tile;   // tile id (-1: the queue is empty, stop)
  int part;   // tile half (kW = 4) or 0
  int base;   // list position of the batch's first entry, from the tile's start
  int seq;    // the CTA's item number
  int first;  // 1: the item's first batch
  int pad[3];
};

template <int kW>
struct __align__(128) QueueShared {
  float4 rec[kQStages][kBatch * kQRec];  // 16 KB per stage; gathers land 256 B at a time
  uint32_t valid[kQStages][kBatch / 32];  // bit j of word c: entry 32c + j holds a valid id
  QueueStage hdr[kQStages];
  uint8_t list[kW][kBatch];
  unsigned long long full_bar[kQStages];   // header written and the stage's gathers landed
  unsigned long long empty_bar[kQStages];  // every consumer warp is done with the stage
  uint32_t done[4];                        // per item (seq mod 4): consumer warps whose pixels all terminated
  uint32_t abort;
};

template <int kW>
constexpr size_t queue_smem_bytes() {
  return sizeof(QueueShared<kW>) + 128;  // + alignment slack of the dynamic shared memory base
}

// Bounded wait on `bar`'s phase `parity`: hardware-suspended waits of at
// most kQWaitNs each, limit / 256 + 4 of them (about 0.16 s at the default
// limit).  False when it ran out (or another warp's did), after flagging the
// CTA and the call.  Warp-collective: every lane waits (so each acquires the
// phase itself) and the warp decides together, so its lanes never part ways.
constexpr uint32_t kQWaitNs = 10000;
__device__ __forceinline__ bool queue_wait(unsigned long long* bar, uint32_t parity, volatile uint32_t* abort,
                                           uint32_t limit, uint32_t* error) {
  const uint32_t tries = (limit >> 8) + 4u;
  for (uint32_t i = 0; i < tries; ++i) {
    if (__all_sync(0xffffffffu, tma::bar_try_wait(bar, parity, kQWaitNs))) return true;
    if (__any_sync(0xffffffffu, *abort != 0u)) return false;
  }
  if ((threadIdx.x & 31u) == 0u) {
    *abort = 1u;
    if (error != nullptr) atomicOr(error, kErrTimeout);
  }
  return false;
}

// The producer's position in the queue: its current item (tile part) and
// the next batch of it to stage.  Warp-uniform.
struct QueueCursor {
  int tile = -1, part = 0, n = 0, nb = 1, b = 0;
  uint32_t rx = 0;
  bool end = true;

  // Take the next item (lane 0's atomic, broadcast) as item number `seq`;
  // clears that item's slot of `done` (seen by the consumers through the
  // item's first stage).
  template <int kW>
  __device__ __forceinline__ void fetch(const BlendArgs& a, uint32_t* done, uint32_t seq, int lane) {
    constexpr int kParts = 8 / kW;
    int item = 0;
    if (lane == 0) {
      item = int(atomicAdd(a.queue, 1u));
      done[seq & 3u] = 0u;
    }
    item = __shfl_sync(0xffffffffu, item, 0);
    end = item >= a.total_tiles * kParts;
    b = 0;
    if (end) {
      tile = -1;
      part = 0;
      n = 0;
      nb = 1;
      rx = 0;
      return;
    }
    tile = int(a.order[item / kParts]);
    part = item % kParts;
    const uint2 range = a.ranges[tile];
    rx = range.x;
    n = int(range.y - range.x);
    nb = max(1, (n + kBatch - 1) / kBatch);  // an empty list still has its pixels written
  }
};

// Every consumer warp of item `seq` has terminated (lane 0 reads, the warp agrees).
template <int kW>
__device__ __forceinline__ bool queue_all_done(const uint32_t* done, uint32_t seq, int lane) {
  uint32_t d = 0;
  if (lane == 0) d = *reinterpret_cast<const volatile uint32_t*>(&done[seq & 3u]);
  return __shfl_sync(0xffffffffu, d, 0) == uint32_t(kW);
}

template <int kW>
__global__ void __launch_bounds__(32 * (kW + 1)) blend_queue_kernel(BlendArgs a, const __grid_constant__ CUtensorMap map) {
  extern __shared__ unsigned char q_raw[];
  QueueShared<kW>& s = *reinterpret_cast<QueueShared<kW>*>((reinterpret_cast<uintptr_t>(q_raw) + 127) & ~uintptr_t(127));
  const int warp = int(threadIdx.x >> 5), lane = int(threadIdx.x & 31);
  const uint32_t limit = a.spin_limit;
  const uint32_t wild = a.wild != nullptr ? *a.wild : 0u;
  volatile uint32_t* abort = &s.abort;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kQStages; ++i) {
      tma::bar_init(&s.full_bar[i], 1);
      tma::bar_init(&s.empty_bar[i], kW);
    }
    s.abort = 0u;
    tma::bar_init_fence();
    // this blend leaves no block masks for the backward passes
    if (blockIdx.x == 0 && a.masks_valid != nullptr) *a.masks_valid = 0u;
  }
  if (threadIdx.x == 32 * kW) tma::prefetch_map(&map);
  __syncthreads();

  if (warp == kW) {
    // ---------------- producer ----------------
    QueueCursor cur;
    uint32_t seq = 0, k = 0;
    cur.fetch<kW>(a, s.done, seq, lane);
    for (;; ++k) {
      if (cur.b > 0 && (cur.b >= cur.nb || queue_all_done<kW>(s.done, seq, lane))) cur.fetch<kW>(a, s.done, ++seq, lane);
      const int st = int(k % kQStages);
      if (!queue_wait(&s.empty_bar[st], ((k / kQStages) & 1u) ^ 1u, abort, limit, a.error)) goto stop;
      const int base = cur.b * kBatch;
      const int cnt = cur.end ? 0 : min(kBatch, cur.n - base);
      const int groups = (cnt + 3) >> 2;
      // lane l gathers groups l and l + 32 (entries 4g .. 4g + 3)
      const uint32_t* ids = a.point_list + cur.rx + base;
      int r[2][4];
      uint32_t vbits = 0;  // bit 4h + q: entry 4 (l + 32h) + q holds a valid id
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int g = lane + 32 * h;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int e = 4 * g + q;
          const uint32_t id = e < cnt ? ids[e] : a.num_records;
          const bool ok = id < a.num_records;
          vbits |= ok ? 1u << (4 * h + q) : 0u;
          r[h][q] = ok ? int(id) : 0;  // a stray id gathers row 0 and stays invalid
        }
      }
      // the stage's valid-entry words and header, by lane 0, before its
      // arrival (which releases them to the consumers)
#pragma unroll
      for (int c = 0; c < kBatch / 32; ++c) {
        const int j = 32 * c + lane, g = j >> 2;
        const uint32_t w = __ballot_sync(0xffffffffu, (__shfl_sync(0xffffffffu, vbits, g & 31) >> (4 * (g >> 5) + (j & 3))) & 1u);
        if (lane == 0) s.valid[st][c] = w;
      }
      if (lane == 0) {
        s.hdr[st] = QueueStage{cur.tile, cur.part, base, int(seq), cur.b == 0 ? 1 : 0, {0, 0, 0}};
        tma::bar_arrive_expect(&s.full_bar[st], uint32_t(groups) * 4u * 64u);  // an empty stage completes at once
      }
      __syncwarp();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int g = lane + 32 * h;
        if (g < groups) tma::gather4(&s.rec[st][kQRec * 4 * g], &map, &s.full_bar[st], r[h][0], r[h][1], r[h][2], r[h][3]);
      }
      ++cur.b;
      if (cur.end) break;
    }
    return;
  stop:
    // a wait ran out: let the copies of the stages issued last land before the CTA ends
    for (uint32_t kk = k > uint32_t(kQStages) ? k - kQStages : 0u; kk < k; ++kk) {
      const int st = int(kk % kQStages);
      for (uint32_t i = 0; i < (limit >> 8) + 4u && !tma::bar_try_wait(&s.full_bar[st], (kk / kQStages) & 1u, kQWaitNs);
           ++i) {
      }
    }
    return;
  }

  // ---------------- consumers ----------------
  BlendPixel pix;
  pix.done = true;
  bool have = false, reported = true;
  int tile = -1, W = 0, H = 0;
  size_t pbase = 0;
  const float* bg = a.bg;
  TilePixel tp(0, 1, warp);
  float pxf = 0.f, pyf = 0.f;
  auto finish = [&]() {
    if (!have) return;
    if (tp.px < W && tp.py < H) {
      const size_t q = size_t(tp.py) * W + tp.px;
      const size_t p = pbase + q, cp = 3 * pbase + q;
      const size_t hw = size_t(W) * H;
      a.n_contrib[p] = pix.last;
      a.out_alpha[p] = pix.Wt;
      a.out_depth[p] = pix.D;
      a.T_final[p] = pix.T;
      a.out_color[cp] = fma(pix.T, bg[0], pix.C0);
      a.out_color[hw + cp] = fma(pix.T, bg[1], pix.C1);
      a.out_color[2 * hw + cp] = fma(pix.T, bg[2], pix.C2);
    }
    const uint32_t wm = __reduce_max_sync(0xffffffffu, pix.last);
    if (lane == 0 && wm != 0u) atomicMax(&a.tile_max[tile], wm);
  };
  const uint32_t lt = (1u << lane) - 1u;
  for (uint32_t k = 0;; ++k) {
    const int st = int(k % kQStages);
    if (!queue_wait(&s.full_bar[st], (k / kQStages) & 1u, abort, limit, a.error)) return;
    const QueueStage h = s.hdr[st];
    if (h.first != 0 || h.tile < 0) {
      finish();
      if (h.tile < 0) return;
      tile = h.tile;
      int ltile = tile;
      W = a.W;
      H = a.H;
      pbase = 0;
      bg = a.bg;
      if (a.items != nullptr) {
        const BatchItem& it = a.items[find_item_tile(a.items, a.num_items, uint32_t(tile))];
        W = it.W;
        H = it.H;
        ltile = tile - int(it.tile_base);
        pbase = size_t(it.pix_base);
        bg = it.bg;
      }
      tp = TilePixel(ltile, (W + kTile - 1) / kTile, h.part * kW + warp);
      pxf = float(tp.px);
      pyf = float(tp.py);
      pix = BlendPixel();
      pix.done = !(tp.px < W && tp.py < H);
      have = true;
      reported = false;
    }
    if (!__all_sync(0xffffffffu, pix.done)) {
      const float4* sr = s.rec[st];
      // the stage's entries that can reach this warp's block, in order
      int cnt = 0;
#pragma unroll 2
      for (int c = 0; c < kBatch / 32; ++c) {
        const uint32_t vw = s.valid[st][c];
        bool reach = false;
        if ((vw >> lane) & 1u) {
          const int j = 32 * c + lane;
          const float4 r0 = sr[kQRec * j], r1 = sr[kQRec * j + 1];
          reach = block_test(r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, tp.bx, tp.by);
        }
        const uint32_t bits = __ballot_sync(0xffffffffu, reach);
        if (reach) s.list[warp][cnt + __popc(bits & lt)] = uint8_t(32 * c + lane);
        cnt += __popc(bits);
      }
      __syncwarp();
      const uint8_t* lst = s.list[warp];
      const uint32_t base = uint32_t(h.base) + 1u;
      for (int k0 = 0; k0 < cnt; k0 += kBlendIlp) {
        const uint32_t packed = *reinterpret_cast<const uint32_t*>(lst + k0);
        int j[kBlendIlp];
#pragma unroll
        for (int kk = 0; kk < kBlendIlp; ++kk) j[kk] = k0 + kk < cnt ? int((packed >> (8 * kk)) & 255u) : -1;
        float al[kBlendIlp];
        float4 m[kBlendIlp], cov[kBlendIlp];
#pragma unroll
        for (int kk = 0; kk < kBlendIlp; ++kk) {
          const int jj = j[kk] < 0 ? j[0] : j[kk];
          m[kk] = sr[kQRec * jj];
          m[kk].z = sr[kQRec * jj + 1].w;
          cov[kk] = sr[kQRec * jj + 2];
        }
        blend_alphas(m, cov, pxf, pyf, al);
#pragma unroll
        for (int kk = 0; kk < kBlendIlp; ++kk) {
          const int jj = j[kk] < 0 ? j[0] : j[kk];
          const float v = j[kk] < 0 ? 0.0f : al[kk];
          if (wild == 0u) pix.step<false>(v, sr[kQRec * jj + 3], base + uint32_t(j[kk]));
          else pix.step<true>(v, sr[kQRec * jj + 3], base + uint32_t(j[kk]));
        }
        if (__all_sync(0xffffffffu, pix.done)) break;
      }
    }
    if (!reported && __all_sync(0xffffffffu, pix.done)) {
      reported = true;
      if (lane == 0) atomicAdd(&s.done[h.seq & 3], 1u);
    }
    __syncwarp();
    if (lane == 0) tma::bar_arrive(&s.empty_bar[st]);
  }
}

}  // namespace

// The tiles' processing order from their ranges (tile_walk.cuh), with `zero` (the
// blend's per-tile maximum) and `counter` (the persistent blend's queue)
// cleared.  One block.
__global__ void __launch_bounds__(1024) tile_order_kernel(const uint2* ranges, int num_tiles, uint32_t* order,
                                                          uint32_t* zero, uint32_t* counter) {
  __shared__ uint32_t s_cnt[kTileBuckets], s_pos[kTileBuckets];
  if (counter != nullptr && threadIdx.x == 0) *counter = 0u;
  for (int i = threadIdx.x; i < kTileBuckets; i += blockDim.x) s_cnt[i] = 0u;
  __syncthreads();
  for (int t = threadIdx.x; t < num_tiles; t += blockDim.x) {
    zero[t] = 0u;
    atomicAdd(&s_cnt[tile_bucket(ranges[t].y - ranges[t].x)], 1u);
  }
  __syncthreads();
  if (threadIdx.x < 32) bucket_positions(s_cnt, s_pos);
  __syncthreads();
  for (int t = threadIdx.x; t < num_tiles; t += blockDim.x)
    order[atomicAdd(&s_pos[tile_bucket(ranges[t].y - ranges[t].x)], 1u)] = uint32_t(t);
}

namespace {

// The driver's tensor-map encoder, looked up once through the runtime (the
// library links only the runtime).
using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encoder() {
  static std::once_flag once;
  static EncodeTiled fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiled>(p);
  });
  return fn;
}

// The records as a 2-D tensor of num_records rows of 16 floats (64 bytes),
// gathered one row per index (box: one row).  False when the map cannot be
// made (no encoder, a base not 16-byte aligned, no rows).
bool record_map(const BlendArgs& a, CUtensorMap* map) {
  if (a.record == nullptr || a.num_records == 0u || (reinterpret_cast<uintptr_t>(a.record) & 15u) != 0u) return false;
  const EncodeTiled enc = encoder();
  if (enc == nullptr) return false;
  const cuuint64_t dims[2] = {16u, cuuint64_t(a.num_records)};
  const cuuint64_t strides[1] = {64u};
  const cuuint32_t box[2] = {16u, 1u};
  const cuuint32_t elem[2] = {1u, 1u};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(a.record), dims, strides, box, elem,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Persistent grid: every CTA the SMs hold at once (at most one per item).
template <int kW>
bool launch_queue(const BlendArgs& a, int tiles, cudaStream_t stream) {
  CUtensorMap map;
  if (a.queue == nullptr || !record_map(a, &map)) return false;
  constexpr int threads = 32 * (kW + 1);
  constexpr size_t smem = queue_smem_bytes<kW>();
  static std::once_flag once;
  static int per_sm = 0;
  std::call_once(once, [] {
    if (cudaFuncSetAttribute(blend_queue_kernel<kW>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) ==
        cudaSuccess)
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, blend_queue_kernel<kW>, threads, smem);
  });
  if (per_sm <= 0) return false;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int items = tiles * (8 / kW);
  const int grid = std::min(items, sms * per_sm);
  BlendArgs b = a;
  b.total_tiles = tiles;  // the queue's length (a single-view call leaves it unset)
  blend_queue_kernel<kW><<<grid, threads, smem, stream>>>(b, map);
  return true;
}

}  // namespace

void launch_blend(const BlendArgs& a, cudaStream_t stream) {
  const int tiles = a.items ? a.total_tiles : ((a.W + kTile - 1) / kTile) * ((a.H + kTile - 1) / kTile);
  if (tiles <= 0) return;
  const int warps = tune_value(kTuneBlendWarps);
  const bool queue = tune_value(kTuneBlendQueue) == 1 && a.queue != nullptr;
  // a tile's warps combine their contributor counts in its maximum, cleared
  // first; the queue counter starts at zero
  if (!a.ordered) {
    stage_begin(kStOther, stream);
    tile_order_kernel<<<1, 1024, 0, stream>>>(a.ranges, tiles, a.order, a.tile_max, a.queue);
    stage_end(kStOther, stream, 1);
  }
  stage_begin(kStBlend, stream);
  const bool queued = queue && (warps == 4 ? launch_queue<4>(a, tiles, stream) : launch_queue<8>(a, tiles, stream));
  if (!queued) {
    auto launch = [&](auto kernel) {
      launch_after(kernel, unsigned(tiles * (8 / kBlendWarps)), 32 * kBlendWarps, 0, stream, a);
    };
    if ((reinterpret_cast<uintptr_t>(a.record) & 31u) == 0u) launch(blend_kernel<true>);
    else launch(blend_kernel<false>);
  }
  stage_end(kStBlend, stream, 1);
}

}  // namespace w2w
