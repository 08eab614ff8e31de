// Key emission: one (tile | depth) key and one Gaussian id per covered tile
// (reference prepareSort.cu:239-301).
//
// Gaussian i owns slots [max(start_i, prev_reach_i), min(start_i + emit_i, R)),
// where start_i is its allocation offset and prev_reach_i the largest end slot
// of any earlier Gaussian (both from the preprocess scan).  With the
// reference's emission rectangle (compat mode) a Gaussian may emit more keys
// than it allocated; those keys land in its successors' slots, and each slot
// is written exactly once, by the lowest-index Gaussian whose emission covers
// it.  Entries are written in row-major order of the rectangle
// (prepareSort.cu:191-204).
//
// Batched calls: every view's Gaussians emit into its own slot range, with its
// own tile grid, and tile ids offset by the view's first global tile.
//
// The kernel also writes the binning state's header (a planned render's: the
// caller's key plan, checked against the view's own count and depth range; one
// that does not fit emits nothing and makes the sort process nothing) and clears
// the sort's histograms and status words: a one-thread kernel and a memset of
// their own cost about 5 us a view in launches and gaps.
//
// Load balance: each warp expands 32 consecutive Gaussians; every lane emits
// one entry per round, so large and small Gaussians cost the same per entry
// and stores to consecutive slots are coalesced.
//
// Bound by the rounds' instructions and by latency (order -> gathers -> lookback
// -> rounds), not by the bytes written.  A round finds its owners in five
// shuffles and takes six or seven words from them, and the row of a cell comes
// from a multiplication where that is exact.  In depth order, per view: 100k
// Gaussians, 2.4M instances, 25 -> 22.6 us; 500k, 5.9M, 47 -> 44.6; 1M, 36M, 141
// -> 120-128, against eleven words and a division.
#include "common.cuh"
#include "kernels.h"

namespace w2w {
namespace {

constexpr uint32_t kScanAgg = 1u << 30, kScanInc = 2u << 30, kScanMask = (1u << 30) - 1u;

// The sum of the blocks before `tile`, by warp 0 (decoupled lookback, 32 status
// words a step; a status word carries its flag and count together).  Bounded.
__device__ __forceinline__ uint32_t lookback_sum(const uint32_t* status, int tile, uint32_t spin_limit,
                                                 uint32_t* error) {
  const int lane = threadIdx.x & 31;
  uint32_t sum = 0, spins = 0;
  int t = tile - 1;
  while (t >= 0) {
    const int q = t - lane;
    const uint32_t w = q >= 0 ? ld_relaxed(status + q) : kScanInc;
    const uint32_t inc = __ballot_sync(0xffffffffu, (w & ~kScanMask) == kScanInc);
    const uint32_t ready = __ballot_sync(0xffffffffu, (w & ~kScanMask) != 0u);
    const uint32_t need = inc ? ((inc & (0u - inc)) << 1) - 1u : 0xffffffffu;
    if ((ready & need) != need) {
      if (++spins > spin_limit) {
        if (lane == 0) atomicOr(error, kErrTimeout);
        break;
      }
      continue;
    }
    sum += __reduce_add_sync(0xffffffffu, (need >> lane) & 1u ? w & kScanMask : 0u);
    if (inc) break;
    t -= 32;
  }
  return sum;
}

// kOrdered: thread j takes the j-th Gaussian by depth, and the entries follow
// one another in that order (their count scanned here), instead of Gaussian j
// and the slots it owns: the list is then sorted by depth already, and the sort
// has only the tile digits left.
template <bool kKey64, bool kOrdered>
__global__ void __launch_bounds__(kDupThreads) duplicate_kernel(DuplicateArgs a) {
  grid_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int block = blockIdx.x;
  if constexpr (kOrdered) {  // blocks in the order they start, so that lookback waits on running ones
    __shared__ int s_block;
    if (threadIdx.x == 0) s_block = int(atomicAdd(a.scan_counter, 1u));
    __syncthreads();
    block = s_block;
  }
  const int j = block * kDupThreads + int(threadIdx.x);
  uint32_t g = uint32_t(j);
  if constexpr (kOrdered) g = j < a.P ? a.order[j] : ~0u;
  uint32_t p0 = 0, cnt = 0, start = 0, x0 = 0, y0 = 0, w = 1, dlow = 0, gwv = uint32_t(a.gw), tbase = 0;
  uint32_t R = a.R, prefix = a.depth_prefix;
  bool fits = true;
  if (a.plan != nullptr) {  // a.R is the capacity
    R = a.plan->num_rendered;
    const uint32_t dmin = ~a.plan->depth_min, x = dmin ^ a.plan->depth_max;
    const uint32_t need = x == 0u ? 0u : 32u - uint32_t(__clz(x));
    fits = R <= a.R && need <= a.depth_bits && (a.plan->error & (kErrTimeout | kErrCapacity)) == 0u;
    prefix = a.depth_bits >= 32 ? 0u : (dmin & ~((1u << a.depth_bits) - 1u));
  }
  const uint32_t Rlim = fits ? R : 0u;
  if (block == 0 && threadIdx.x == 0) {
    BinHeader* h = a.header;
    if constexpr (!kOrdered) h->error = 0u;  // else cleared before the depth sort, which reports there too
    h->masks_valid = 1u;  // the blend that follows writes the block masks
    h->key64 = kKey64 ? 1u : 0u;
    h->depth_bits = a.depth_bits;
    h->depth_prefix = prefix;
    h->tile_bits = a.tile_bits;
    h->passes = a.passes;
    h->num_rendered = R;
    h->n_sort = Rlim;
    h->replan = fits ? 0u : 1u;
    for (int i = 0; i <= kMaxPasses; ++i) h->tile_counter[i] = 0u;
  }
  for (uint32_t i = blockIdx.x * kDupThreads + threadIdx.x; i < a.clear_vecs; i += gridDim.x * kDupThreads)
    a.clear[i] = make_uint4(0u, 0u, 0u, 0u);
  if (block * kDupThreads >= a.P) return;  // a block that only clears
  if (g < uint32_t(a.P)) {  // Gaussians that emit nothing have an empty rectangle
    uint32_t end = Rlim;
    if (a.items != nullptr) {  // batched: this view's tile grid, first tile id and end slot
      const int item = find_item_elem(a.items, a.num_items, g);
      gwv = uint32_t(a.items[item].gw);
      tbase = a.items[item].tile_base;
      end = a.item_end[item];
    }
    start = a.offsets[g] - a.tiles[g];
    const uint2 rc = reinterpret_cast<const uint2*>(a.rect)[g];
    x0 = rc.x & 0xffffu;
    y0 = rc.x >> 16;
    const uint32_t x1 = rc.y & 0xffffu, y1 = rc.y >> 16;
    w = x1 > x0 ? x1 - x0 : 1u;
    const uint32_t n = (x1 > x0 && y1 > y0) ? (x1 - x0) * (y1 - y0) : 0u;
    const uint32_t reach = start + n;
    p0 = max(start, a.prev_reach[g]);
    const uint32_t p1 = min(reach, end);
    cnt = p1 > p0 ? p1 - p0 : 0u;
    const uint32_t db = __float_as_uint(a.depth[g]);
    dlow = a.depth_bits >= 32 ? db : (db & ((1u << a.depth_bits) - 1u));
  }
  // warp inclusive scan of the entry counts
  uint32_t incl = cnt;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += o;
  }
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
  const uint32_t excl = incl - cnt;
  uint32_t before = 0;  // kOrdered: entries before this warp's
  if constexpr (kOrdered) {
    __shared__ uint32_t s_warp[kDupThreads / 32], s_before;
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t mine = 0, all = 0;
#pragma unroll
    for (int w2 = 0; w2 < kDupThreads / 32; ++w2) {
      if (w2 < warp) mine += s_warp[w2];
      all += s_warp[w2];
    }
    if (warp == 0) {
      const bool publish = block != a.unpublished_tile;
      if (lane == 0 && block > 0 && publish) st_relaxed(a.scan_status + block, kScanAgg | all);
      const uint32_t b = lookback_sum(a.scan_status, block, a.spin_limit, &a.header->error);
      if (lane == 0) {
        if (publish) st_relaxed(a.scan_status + block, kScanInc | ((b + all) & kScanMask));
        s_before = b;
      }
    }
    __syncthreads();
    before = s_before + mine;
  }
  // what an entry's lane needs of its owner, in as few words as it takes: entry
  // e is rectangle cell e + cell; the row by a multiplication where that is
  // exact (cell numbers and widths below 2^16)
  const uint32_t cell = p0 - excl - start, slot = p0 - excl, corner = x0 | (y0 << 16);
  const uint32_t inv = w > 1u ? 0xffffffffu / w + 1u : 0u;
  const bool batched = a.items != nullptr;
  const bool small = __all_sync(0xffffffffu, w < 65536u && p0 - start + cnt <= 65536u);
  for (uint32_t base = 0; base < total; base += 32) {
    const uint32_t e = base + lane;
    // owner lane: number of lanes whose inclusive count is <= e
    int o = 0;
#pragma unroll
    for (int b = 16; b > 0; b >>= 1) {
      const uint32_t t = __shfl_sync(0xffffffffu, incl, o + b - 1);
      if (t <= e) o += b;
    }
    o = min(o, 31);
    const uint32_t k = e + __shfl_sync(0xffffffffu, cell, o);
    const uint32_t oc = __shfl_sync(0xffffffffu, corner, o);
    const uint32_t ow = __shfl_sync(0xffffffffu, w, o);
    const uint32_t oi = __shfl_sync(0xffffffffu, inv, o);
    const uint32_t odl = __shfl_sync(0xffffffffu, dlow, o);
    const uint32_t og = __shfl_sync(0xffffffffu, g, o);
    const uint32_t at = kOrdered ? before + e : e + __shfl_sync(0xffffffffu, slot, o);
    uint32_t ogw = uint32_t(a.gw), otb = 0;
    if (batched) {
      ogw = __shfl_sync(0xffffffffu, gwv, o);
      otb = __shfl_sync(0xffffffffu, tbase, o);
    }
    if (e < total && at < Rlim) {
      const uint32_t row = small ? (ow > 1u ? __umulhi(k, oi) : k) : k / ow;
      const uint32_t tile = otb + ((oc >> 16) + row) * ogw + (oc & 0xffffu) + (k - row * ow);
      if constexpr (kKey64) {
        reinterpret_cast<uint64_t*>(a.keys)[at] = (uint64_t(tile) << a.depth_bits) | odl;
      } else {
        reinterpret_cast<uint32_t*>(a.keys)[at] = (a.depth_bits >= 32 ? 0u : (tile << a.depth_bits)) | odl;
      }
      a.vals[at] = og;
    }
  }
}

}  // namespace

void launch_duplicate(const DuplicateArgs& a, cudaStream_t stream) {
  if (a.P <= 0 || a.R == 0) return;
  // enough blocks to clear 16 KB each when the Gaussians need fewer
  const int blocks = max((a.P + kDupThreads - 1) / kDupThreads, min(296, int(a.clear_vecs / 1024u)));
  stage_begin(kStDuplicate, stream);
  if (a.order != nullptr) {
    if (a.key64) launch_after(duplicate_kernel<true, true>, unsigned(blocks), kDupThreads, 0, stream, a);
    else launch_after(duplicate_kernel<false, true>, unsigned(blocks), kDupThreads, 0, stream, a);
  } else {
    if (a.key64) launch_after(duplicate_kernel<true, false>, unsigned(blocks), kDupThreads, 0, stream, a);
    else launch_after(duplicate_kernel<false, false>, unsigned(blocks), kDupThreads, 0, stream, a);
  }
  stage_end(kStDuplicate, stream, 1);
}

}  // namespace w2w
