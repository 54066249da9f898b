// Batched segmented sort: thousands of uint32 arrays of uneven size, each
// sorted independently (stable, ascending), through a captured CUDA graph.
//
// Public plans with 8-bit digits sort by buckets (launch_seg_buckets,
// pa_buckets.cu); only the segments that declines go through the digit passes
// here (declined_*_kernel, over lists made on the device).  A run that waits, by
// four digit passes alone -> now (us): 4096 arrays of 1 K to 4 M uniform keys, 2.0 G
// keys, 36060 -> 15800; 300 of 1 K to 1 M 898 -> 381; 64 of 1 K to 50 K 90 -> 60.
// Skewed keys pay for the maps and counts they are declined on: 1000 arrays of 1 M
// 16430 -> 17100, 2000 of 20 K 863 -> 890, 300 of 1 K to 1 M 906 -> 919; 64 of 1 K to
// 50 K 84 -> 84, 64 of 3000 42 -> 41.
//
// 11-bit plans, and the plans other sorts build for their groups, run ONE
// persistent kernel fed by a device work queue (8-bit ones then a launch per
// digit pass):
//
// No reference counterpart: the reference sorts one array per call
// (SortRadixPar, RadixSortLsdParallel.h:367); its nearest idea is bundling
// small work items (BundleSmallWorkItems.cpp:36).  Per segment the result is
// exactly SortRadixPar's.
//
// Work items, in queue order (a CTA takes the next item with one atomicAdd):
//   HIST  one chunk of a large segment: its four byte-digit counts, added
//         into the segment's histogram;
//   SCAN  one large segment: bin starts of its four digits;
//   PASS  (11-bit plans) one tile of one large segment for digit pass p: the
//         onesweep tile of the plain sort (pa_onesweep_tile.cuh), look-back
//         within the segment.  8-bit plans run each pass as its own launch
//         after the persistent kernel instead (seg_pass_kernel: the plain
//         sort's pass geometry over all large segments' tiles at once, no
//         work-queue round trips per tile);
//   SMALL one small segment (<= the small/large cutoff) sorted entirely in
//         shared memory by eight stable 4-bit counting passes, read once and
//         written once.
// Small items are spread between the large-segment stages so that CTAs
// waiting on a stage have work.  An item waits only on earlier items of the
// same segment (per-segment completion counters: HIST chunks before SCAN,
// SCAN before pass 0, all tiles of pass p before pass p + 1); items are taken
// in queue order by running CTAs, so the earliest unfinished item can always
// proceed.  Every wait is bounded and reports through the plan's error word.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <vector>

#include "pa_common.cuh"
#include "pa_gpu.h"
#include "pa_kernels.cuh"
#include "pa_onesweep_tile.cuh"
#include "pa_segmented.cuh"

namespace pa {
namespace seg {

using namespace os;

// Bounded wait until *ctr >= need (acquire).  Thread 0 only.
__device__ __forceinline__ void wait_count(const uint32_t* ctr, uint32_t need, uint32_t* err) {
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    if (ld_acquire_gpu(ctr) >= need) return;
    __nanosleep(64);
  }
  raise_error(err, DEVERR_LOOKBACK_TIMEOUT);
}

// Lane copies of each HIST counter: the 8-bit table (4 x 256) keeps 8, the
// 11-bit one (3 x 2048) 2, so that both fit shared memory.
template <int RB>
__host__ __device__ constexpr int hist_lanes() { return RB == 11 ? 2 : kHistLanes; }

template <int RB>
__device__ __forceinline__ void hist_item(const PlanDev& P, const Item& it, unsigned char* smem) {
  constexpr uint32_t D = RB == 11 ? 3u : 4u, R = 1u << RB;
  constexpr uint32_t L = hist_lanes<RB>();
  const LargeSeg L_ = P.large[it.seg];
  uint32_t* h = reinterpret_cast<uint32_t*>(smem);
  constexpr uint32_t kWords = D * R * L;
  for (uint32_t i = threadIdx.x; i < kWords; i += kBlock) h[i] = 0;
  __syncthreads();
  const uint32_t lo = it.idx * kHistChunk;
  const uint32_t len = min(kHistChunk, L_.len - lo);
  const uint32_t* src = P.keys + L_.base + lo;
  uint32_t* my = h + (threadIdx.x % L);
  for (uint32_t i = threadIdx.x; i < len; i += kBlock) {
    const uint32_t k = src[i];
#pragma unroll
    for (uint32_t d = 0; d < D; ++d) atomicAdd(my + (d * R + ((k >> (RB * d)) & (R - 1))) * L, 1u);
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < D * R; e += kBlock) {
    uint32_t sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < L; ++j) sum += h[e * L + ((j + e) % L)];
    if (sum) atomicAdd(&P.hist[(size_t)it.seg * D * R + e], sum);
  }
}

template <int RB>
__device__ __forceinline__ void scan_item(const PlanDev& P, const Item& it, unsigned char* smem) {
  constexpr uint32_t D = RB == 11 ? 3u : 4u, R = 1u << RB;
  constexpr uint32_t PER = R >= kBlock ? R / kBlock : 1;  // bins per thread
  uint32_t* s_warp = reinterpret_cast<uint32_t*>(smem);
  const uint32_t tid = threadIdx.x;
  for (uint32_t d = 0; d < D; ++d) {
    const uint32_t* hd = P.hist + (size_t)it.seg * D * R + d * R;
    uint32_t c[PER];
    uint32_t local = 0;
#pragma unroll
    for (uint32_t i = 0; i < PER; ++i) {
      const uint32_t b = tid * PER + i;
      c[i] = b < R ? hd[b] : 0u;
      local += c[i];
    }
    uint32_t run = block_exclusive_scan<kBlock>(local, s_warp);
#pragma unroll
    for (uint32_t i = 0; i < PER; ++i) {
      const uint32_t b = tid * PER + i;
      if (b < R) P.bin_start[(size_t)it.seg * D * R + d * R + b] = run;
      run += c[i];
    }
    __syncthreads();  // s_warp is reused by the next digit's scan
  }
}

template <int PASS_ITEMS, int RB>
__device__ __forceinline__ void pass_item(const PlanDev& P, const Item& it, unsigned char* smem, uint64_t* bar,
                                          uint32_t& parity) {
  constexpr uint32_t D = RB == 11 ? 3u : 4u, R = 1u << RB;
  const LargeSeg L = P.large[it.seg];
  const bool even = (it.pass & 1u) == 0;
  TileJob<uint32_t, uint32_t> job;
  job.in = (even ? P.keys : P.tmp) + L.base;
  job.out = (even ? P.tmp : P.keys) + L.base;
  job.vin = nullptr;
  job.vout = nullptr;
  job.n = L.len;
  job.out_n = L.len;
  job.tile = it.idx;
  job.shift = RB * it.pass;
  job.tin = false;
  job.tout = false;
  job.bin_start = P.bin_start + (size_t)it.seg * D * R + it.pass * R;
  job.status = P.status + ((size_t)it.pass * P.total_tiles + L.tile_base) * R;
  job.err = P.err;
  job.spin_limit = kSpinLimit;
  if constexpr (RB == 11)
    onesweep_tile_wide<uint32_t, false, kBlock, PASS_ITEMS, 11, uint32_t>(job, smem, bar, parity);
  else
    onesweep_tile_multisplit<uint32_t, false, kBlock, PASS_ITEMS, uint32_t>(job, smem, bar, parity);
}

template <int SMALL_ITEMS>
__device__ __forceinline__ void small_item(const PlanDev& P, const Item& it, unsigned char* smem) {
  using GS = Geometry<uint32_t, false, kBlock, SMALL_ITEMS>;
  constexpr uint32_t TILE = GS::kTile;
  uint32_t* s_keys = reinterpret_cast<uint32_t*>(smem + GS::kKeysOff);
  uint32_t* s_cnt = reinterpret_cast<uint32_t*>(smem + GS::kCntOff);
  uint32_t* s_warp = reinterpret_cast<uint32_t*>(smem + GS::kWarpTotOff);
  const unsigned long long base = P.seg_off[it.seg];
  const uint32_t len = (uint32_t)(P.seg_off[it.seg + 1] - base);
  const uint32_t* keys = P.keys + base;
  uint32_t* out = result_buffer(P) + base;
  for (uint32_t i = threadIdx.x; i < TILE; i += kBlock) s_keys[i] = i < len ? keys[i] : 0xFFFFFFFFu;
  __syncthreads();
  uint32_t k[SMALL_ITEMS];
  uint32_t v[1];
#pragma unroll 1
  for (uint32_t sh = 0; sh < 32; sh += 4) {
    load_run<uint32_t, false, SMALL_ITEMS>(k, v, s_keys, nullptr);
    nibble_pass<uint32_t, false, kBlock, SMALL_ITEMS>(k, v, sh, s_keys, nullptr, s_cnt, s_warp);
  }
  for (uint32_t i = threadIdx.x; i < len; i += kBlock) out[i] = s_keys[i];
}

template <int PASS_ITEMS, int SMALL_ITEMS, int RB>
__global__ void __launch_bounds__(kBlock, 2) segsort_kernel(const PlanDev P) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ Item s_item;
  __shared__ uint32_t s_index;
  // The bulk-copy barrier lives outside the dynamic area, which every item
  // kind lays out differently.
  __shared__ __align__(8) uint64_t s_bar_storage;
  uint64_t* s_bar = &s_bar_storage;
  if (threadIdx.x == 0) {
    mbar_init(s_bar, 1);
    mbar_fence_init();
  }
  uint32_t parity = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      const uint32_t i = atomicAdd(P.head, 1u);
      s_index = i;
      if (i < P.num_items) s_item = P.items[i];
    }
    __syncthreads();
    if (s_index >= P.num_items) break;
    const Item it = s_item;
    if (it.kind == ITEM_SCAN || it.kind == ITEM_PASS) {
      if (threadIdx.x == 0) {
        const LargeSeg L = P.large[it.seg];
        const uint32_t* d = P.done + (size_t)it.seg * kStages;
        if (it.kind == ITEM_SCAN)
          wait_count(d + ST_HIST, L.hist_chunks, P.err);
        else if (it.pass == 0)
          wait_count(d + ST_SCAN, 1, P.err);
        else
          wait_count(d + ST_PASS0 + it.pass - 1, L.tiles, P.err);
        fence_proxy_async();
      }
      __syncthreads();
    }
    if (it.kind == ITEM_SMALL)
      small_item<SMALL_ITEMS>(P, it, smem);
    else if (it.kind == ITEM_HIST)
      hist_item<RB>(P, it, smem);
    else if (it.kind == ITEM_SCAN)
      scan_item<RB>(P, it, smem);
    else
      pass_item<PASS_ITEMS, RB>(P, it, smem, s_bar, parity);
    __syncthreads();
    if (it.kind != ITEM_SMALL && threadIdx.x == 0) {
      __threadfence();
      const uint32_t st = it.kind == ITEM_HIST ? ST_HIST : it.kind == ITEM_SCAN ? ST_SCAN : ST_PASS0 + it.pass;
      atomicAdd(P.done + (size_t)it.seg * kStages + st, 1u);
    }
  }
}

// One digit pass over every large segment of an 8-bit plan: tiles taken in
// launch order (ticket), each mapped to its segment through the plan's tile
// table; the onesweep tile of the plain sort with the segment as the array,
// so the look-back stays inside the segment (its first tile publishes an
// INCLUSIVE word).  Runs after the persistent kernel has finished every
// HIST and SCAN item, so no item waits.
using PassGeometry = Geometry<uint32_t, false, kPassBlock, kPassItems>;

__device__ __forceinline__ void seg_pass_tile(const PlanDev& P, uint32_t pass, const DeclinedTile& t, uint32_t tile,
                                              size_t words, unsigned char* smem, uint64_t* s_bar, uint32_t& parity) {
  const bool even = (pass & 1u) == 0;
  TileJob<uint32_t, uint32_t> job;
  job.in = (even ? P.keys : P.tmp) + t.base;
  job.out = (even ? P.tmp : P.keys) + t.base;
  job.vin = nullptr;
  job.vout = nullptr;
  job.n = t.len;
  job.out_n = t.len;
  job.tile = tile;
  job.shift = 8u * pass;
  job.tin = false;
  job.tout = false;
  job.bin_start = P.bin_start + (size_t)t.seg * 4 * 256 + pass * 256;
  job.status = P.pass_status + words * 256;
  job.err = P.err;
  job.spin_limit = kSpinLimit;
  onesweep_tile_multisplit<uint32_t, false, kPassBlock, kPassItems, uint32_t>(job, smem, s_bar, parity);
}

__global__ void __launch_bounds__(kPassBlock, 3) seg_pass_kernel(const PlanDev P, uint32_t pass) {
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + PassGeometry::kBarOff);
  uint32_t* s_tile = reinterpret_cast<uint32_t*>(smem + PassGeometry::kTileIdOff);
  if (threadIdx.x == 0) {
    *s_tile = atomicAdd(P.pass_ticket + pass, 1u);
    mbar_init(s_bar, 1);
    mbar_fence_init();
  }
  __syncthreads();
  const uint32_t g = *s_tile;
  if (g >= P.pass_tiles) {  // a ticket counter that was not cleared
    if (threadIdx.x == 0) raise_error(P.err, DEVERR_BAD_STATE);
    return;
  }
  const uint32_t seg = P.tile_seg[g];
  const LargeSeg L = P.large[seg];
  uint32_t parity = 0;
  seg_pass_tile(P, pass, {L.base, L.len, seg, L.ptile_base, {}}, g - L.ptile_base, L.ptile_base, smem, s_bar, parity);
}

// The same over the segments the bucket sort declined.  How many tiles they have
// is known on the device alone, so resident CTAs take tickets until the tiles are
// used up: a CTA for each tile there might be would cost evenly spread keys, which
// leave nothing to the passes, 50 us a pass of 33 K tiles.  (The loop costs tiles
// of long segments 3 %: 300 of 1M keys 1123 to 1185 us a pass against 1088 to 1148;
// a tile's code called instead of inlined 1165 to 1240.)
__global__ void __launch_bounds__(kPassBlock, 3) declined_pass_kernel(const PlanDev P, uint32_t pass) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ DeclinedTile s_job;
  uint64_t* s_bar = reinterpret_cast<uint64_t*>(smem + PassGeometry::kBarOff);
  uint32_t* s_tile = reinterpret_cast<uint32_t*>(smem + PassGeometry::kTileIdOff);
  const uint32_t tiles = P.declined[kDeclinedTiles];
  if (tiles == 0) return;
  if (threadIdx.x == 0) {
    mbar_init(s_bar, 1);
    mbar_fence_init();
  }
  uint32_t parity = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      const uint32_t g = atomicAdd(P.pass_ticket + pass, 1u);
      *s_tile = g;
      if (g < tiles) s_job = P.declined_tile[g];
    }
    __syncthreads();
    const uint32_t g = *s_tile;
    if (g >= tiles) {
      if (g >= tiles + gridDim.x && threadIdx.x == 0) raise_error(P.err, DEVERR_BAD_STATE);  // a counter not cleared
      return;
    }
    seg_pass_tile(P, pass, s_job, g - s_job.first, (size_t)s_job.first + (P.status_sets > 1 ? (size_t)pass * P.pass_tiles : 0),
                  smem, s_bar, parity);
    __syncthreads();
    // (a tile that gave up ends its CTA, as in the plain pass)
    if (*reinterpret_cast<uint32_t*>(smem + PassGeometry::kAbortOff)) return;
  }
}

// The segments the bucket sort declined: their tiles' look-back words cleared
// (sets: passes to clear for), their digit counts and bin starts.  The chunks to
// be counted are one list over all of them: 2000 segments of 20 K keys, each
// walked by every CTA, cost 0.6 ms of waiting for two loads a segment.
__device__ __forceinline__ void clear_status(const PlanDev& P, uint32_t sets) {
  const size_t words = (size_t)P.declined[kDeclinedTiles] * 64;  // 16-byte words: 256 counters a tile
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (uint32_t p = 0; p < sets; ++p) {
    uint4* q = reinterpret_cast<uint4*>(P.pass_status + (size_t)p * P.pass_tiles * 256);
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < words; i += stride) q[i] = make_uint4(0u, 0u, 0u, 0u);
  }
}

__global__ void __launch_bounds__(kBlock, 2) declined_counts_kernel(const PlanDev P) {
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t num = P.declined[kDeclinedChunks];
  if (num == 0) return;
  clear_status(P, P.status_sets);
  for (uint32_t d = blockIdx.x; d < num; d += gridDim.x) {
    const uint2 c = P.declined_chunk[d];
    hist_item<8>(P, Item{ITEM_HIST, 0, c.x, c.y}, smem);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kBlock) declined_scan_kernel(const PlanDev P) {
  __shared__ __align__(16) unsigned char s_scan[kBlock / 32 * 4];
  const uint32_t num = P.declined[kDeclinedSegs];
  for (uint32_t d = blockIdx.x; d < num; d += gridDim.x)
    scan_item<8>(P, Item{ITEM_SCAN, 0, P.declined[kDeclinedHead + d], 0}, s_scan);
}

__global__ void __launch_bounds__(256) declined_clear_kernel(const PlanDev P) { clear_status(P, 1); }

// ---- host side ---------------------------------------------------------------
template <int PI, int SI, int RB>
constexpr size_t smem_bytes_for() {
  using GS = Geometry<uint32_t, false, kBlock, SI>;
  size_t b = RB == 11 ? WideGeometry<uint32_t, false, kBlock, PI, 11>::kBytes : Geometry<uint32_t, false, kBlock, PI>::kBytes;
  if (GS::kBytes > b) b = GS::kBytes;
  const size_t hist = (size_t)(RB == 11 ? 3 : 4) * (1u << RB) * hist_lanes<RB>() * 4;
  if (hist > b) b = hist;
  return b;
}


template <int PI, int SI, int RB>
KernelChoice choice() {
  return {segsort_kernel<PI, SI, RB>, smem_bytes_for<PI, SI, RB>(), (uint32_t)kBlock * PI, (uint32_t)kBlock * SI};
}

template <int RB>
bool pick_kernel_rb(int pi, int si, KernelChoice* out) {
  if (pi == 8 && si == 4) *out = choice<8, 4, RB>();
  if (pi == 8 && si == 8) *out = choice<8, 8, RB>();
  if (pi == 8 && si == 16) *out = choice<8, 16, RB>();
  if (pi == 16 && si == 4) *out = choice<16, 4, RB>();
  if (pi == 16 && si == 8) *out = choice<16, 8, RB>();
  if (pi == 16 && si == 16) *out = choice<16, 16, RB>();
  return true;
}

bool pick_kernel(int tile_keys, int small_cutoff, int radix_bits, KernelChoice* out) {
  const int pi = tile_keys == 4096 ? 8 : tile_keys == 8192 ? 16 : 0;
  const int si = small_cutoff == 2048 ? 4 : small_cutoff == 4096 ? 8 : small_cutoff == 8192 ? 16 : 0;
  if (!pi || !si) return false;
  return radix_bits == 11 ? pick_kernel_rb<11>(pi, si, out) : pick_kernel_rb<8>(pi, si, out);
}

// ---- host-side planning --------------------------------------------------------
constexpr uint32_t kStatusSetTiles = 16384;  // 64 MB of look-back words for four passes

int build_host_plan(const uint64_t* off_host, size_t num_segments, const pa_segsort_config* cfg, HostPlan* hp,
                    int passes, bool by_buckets) {
  if (passes < 1 || passes > kPasses) return record_error(PA_ERR_ARG, "a batched plan runs 1 to 4 digit passes");
  pa_segsort_config c{};
  if (cfg) c = *cfg;
  for (int r : c.reserved)
    if (r) return record_error(PA_ERR_ARG, "pa_segsort_config.reserved must be zero");
  if (c.small_cutoff == 0) c.small_cutoff = 4096;
  if (c.tile_keys == 0) c.tile_keys = 8192;
  if (c.digit_bits == 0) c.digit_bits = 8;
  if (c.digit_bits != 8 && c.digit_bits != 11)
    return record_error(PA_ERR_ARG, "digit_bits must be 8 or 11 for the batched sort");
  if (c.digit_bits == 11) passes = 3;
  KernelChoice kc{};
  if (!pick_kernel(c.tile_keys, c.small_cutoff, c.digit_bits, &kc))
    return record_error(PA_ERR_ARG, "tile_keys must be 4096 or 8192 and small_cutoff 2048, 4096 or 8192");
  const uint64_t* off = off_host;
  for (size_t i = 0; i < num_segments; ++i) {
    if (off[i + 1] < off[i]) return record_error(PA_ERR_ARG, "seg_offsets must be non-decreasing");
    if (off[i + 1] - off[i] > kMaxSegmentKeys)
      return record_error(PA_ERR_ARG, "a segment exceeds 2^30 - 1 keys (the batched sort's limit)");
  }
  hp->cfg = c;
  hp->kc = kc;
  hp->passes = (uint32_t)passes;
  hp->radix_bits = (uint32_t)c.digit_bits;
  hp->split = c.digit_bits == 8;
  hp->tile_seg.clear();
  hp->pass_tiles = 0;
  hp->by_buckets = by_buckets && hp->split && passes == kPasses;
  hp->bsegs.clear();
  hp->of_large.clear();
  hp->bjobs.clear();
  hp->buckets = hp->part_tiles = 0;
  hp->off.assign(off, off + num_segments + 1);
  hp->items.clear();
  hp->large.clear();
  std::vector<uint32_t> small_ids;
  uint32_t total_tiles = 0;
  for (size_t i = 0; i < num_segments; ++i) {
    const uint64_t len = off[i + 1] - off[i];
    if (len == 0 || (len == 1 && (passes % 2) == 0)) continue;  // (an odd pass count moves even single keys to tmp)
    const bool small = hp->by_buckets ? len <= (uint64_t)kBucketSegKeys
                                      : len <= (uint64_t)kc.small_tile && len <= (uint64_t)c.small_cutoff;
    if (small) {
      small_ids.push_back((uint32_t)i);
    } else {
      LargeSeg L{};
      L.base = off[i];
      L.len = (uint32_t)len;
      L.tiles = (uint32_t)((len + kc.pass_tile - 1) / kc.pass_tile);
      L.hist_chunks = (uint32_t)((len + kHistChunk - 1) / kHistChunk);
      L.tile_base = total_tiles;
      total_tiles += L.tiles;
      if (hp->by_buckets) {
        uint32_t bits = 1;  // about 1500 to 3072 keys a bucket
        while (bits < kSegBinsLog2 && (len >> bits) > 3072) ++bits;
        if (len > kBucketSegMax) {
          hp->of_large.push_back(0xFFFFFFFFu);
        } else {
          hp->of_large.push_back((uint32_t)hp->bsegs.size());
          hp->bsegs.push_back({off[i], (uint32_t)len, bits, hp->buckets, hp->part_tiles, (uint32_t)hp->large.size(), 0});
          hp->buckets += 1u << bits;
          hp->part_tiles += (uint32_t)((len + 3 + kSegTile - 1) / kSegTile);
        }
      }
      if (hp->split) {
        const uint32_t pt = (uint32_t)((len + kPassTile - 1) / kPassTile);
        L.ptile_base = hp->pass_tiles;
        hp->pass_tiles += pt;
        hp->tile_seg.insert(hp->tile_seg.end(), pt, (uint32_t)hp->large.size());
      }
      hp->large.push_back(L);
    }
  }
  // largest small segments first (they take longest)
  std::stable_sort(small_ids.begin(), small_ids.end(),
                   [&](uint32_t a, uint32_t b) { return off[a + 1] - off[a] > off[b + 1] - off[b]; });
  auto& items = hp->items;
  size_t next_small = 0;
  // small items go after HIST, after SCAN and (PASS items) after each pass but the last
  const size_t gaps = hp->split ? 2 : 1 + 1 + (size_t)passes;
  auto add_small = [&](size_t share_of) {
    const size_t upto = std::min(small_ids.size(), (small_ids.size() * share_of + gaps - 1) / gaps);
    for (; next_small < upto; ++next_small) items.push_back({ITEM_SMALL, 0, small_ids[next_small], 0});
  };
  const uint32_t nlarge = (uint32_t)hp->large.size();
  for (uint32_t l = 0; l < nlarge; ++l)
    for (uint32_t ch = 0; ch < hp->large[l].hist_chunks; ++ch) items.push_back({ITEM_HIST, 0, l, ch});
  hp->hist_items = (uint32_t)items.size();
  if (hp->by_buckets) {  // a small segment is one bucket, sorted in place
    for (uint32_t i : small_ids)
      hp->bjobs.push_back({off[i], (uint32_t)(off[i + 1] - off[i]), 0u, 1u, 1u, 0u, 0u});
    hp->buckets += (uint32_t)hp->bjobs.size();
  }
  add_small(1);
  for (uint32_t l = 0; l < nlarge; ++l) items.push_back({ITEM_SCAN, 0, l, 0});
  add_small(2);
  if (!hp->split) {
    for (uint32_t p = 0; p < (uint32_t)passes; ++p) {
      for (uint32_t l = 0; l < nlarge; ++l)
        for (uint32_t t = 0; t < hp->large[l].tiles; ++t) items.push_back({ITEM_PASS, p, l, t});
      add_small(3 + p);
    }
  }
  add_small(gaps);
  hp->total_tiles = total_tiles;
  hp->num_small = (uint32_t)small_ids.size();
  hp->num_large = nlarge;
  // device layout
  const size_t nl = std::max<size_t>(nlarge, 1);
  size_t o = 0;
  auto take = [&](size_t bytes) {
    o = (o + 255) & ~(size_t)255;
    const size_t at = o;
    o += bytes;
    return at;
  };
  hp->o_items = take(std::max<size_t>(items.size(), 1) * sizeof(Item));
  hp->o_off = take(hp->off.size() * 8);
  hp->o_large = take(nl * sizeof(LargeSeg));
  hp->o_tile_seg = take(std::max<size_t>(hp->tile_seg.size(), 1) * 4);  // (the uploaded image ends here)
  const size_t per_seg = (size_t)seg_digits(hp->radix_bits) * seg_bins(hp->radix_bits);
  hp->o_bins = take(nl * per_seg * 8);
  hp->o_err = take(256);
  hp->o_head = take(256);  // everything from here on is cleared per run
  hp->o_done = take(nl * kStages * 4);
  hp->o_hist = take(nl * per_seg * 4);
  if (hp->by_buckets) {
    hp->o_count = take((size_t)std::max<uint32_t>(hp->buckets, 1) * 4);
    hp->o_decl = take((kDeclinedHead + nl) * 4);
    hp->o_rare = take(((size_t)hp->buckets + 1) * 4);
  }
  hp->o_status = take(hp->split ? 0 : (size_t)passes * std::max<uint32_t>(total_tiles, 1) * seg_bins(hp->radix_bits) * 4);
  hp->o_pticket = take(256);
  // (a plan by buckets: the passes' words all at once where that is little memory)
  hp->status_sets = hp->by_buckets && hp->pass_tiles <= kStatusSetTiles ? (uint32_t)passes : 1u;
  hp->o_pstatus = take((size_t)std::max<uint32_t>(hp->pass_tiles, 1) * 256 * 4 * hp->status_sets);
  if (hp->by_buckets) {  // (not cleared)
    hp->o_bseg = take(std::max<size_t>(hp->bsegs.size(), 1) * sizeof(BucketSeg));
    hp->o_of_large = take(nl * 4);
    hp->o_map = take(std::max<size_t>(hp->bsegs.size(), 1) * sizeof(SegMap));
    hp->o_bjob = take((size_t)std::max<uint32_t>(hp->buckets, 1) * sizeof(SegBucketJob));
    hp->o_tjob = take((size_t)std::max<uint32_t>(hp->part_tiles, 1) * sizeof(SegTileJob));
    hp->o_dtile = take((size_t)std::max<uint32_t>(hp->pass_tiles, 1) * sizeof(DeclinedTile));
    hp->o_dchunk = take((size_t)std::max<uint32_t>(hp->hist_items, 1) * sizeof(uint2));
  }
  hp->bytes = o;
  return PA_OK;
}

PlanDev device_view(const HostPlan& hp, char* dev, uint32_t* keys, uint32_t* tmp) {
  PlanDev d{};
  d.keys = keys;
  d.tmp = tmp;
  d.passes = hp.passes;
  d.items = reinterpret_cast<const Item*>(dev + hp.o_items);
  d.num_items = (uint32_t)hp.items.size();
  d.total_tiles = hp.total_tiles;
  d.seg_off = reinterpret_cast<const unsigned long long*>(dev + hp.o_off);
  d.large = reinterpret_cast<const LargeSeg*>(dev + hp.o_large);
  d.head = reinterpret_cast<uint32_t*>(dev + hp.o_head);
  d.done = reinterpret_cast<uint32_t*>(dev + hp.o_done);
  d.hist = reinterpret_cast<uint32_t*>(dev + hp.o_hist);
  d.status = reinterpret_cast<uint32_t*>(dev + hp.o_status);
  d.bin_start = reinterpret_cast<unsigned long long*>(dev + hp.o_bins);
  d.err = reinterpret_cast<uint32_t*>(dev + hp.o_err);
  d.radix_bits = hp.radix_bits;
  d.tile_seg = reinterpret_cast<const uint32_t*>(dev + hp.o_tile_seg);
  d.pass_tiles = hp.pass_tiles;
  d.pass_ticket = reinterpret_cast<uint32_t*>(dev + hp.o_pticket);
  d.pass_status = reinterpret_cast<uint32_t*>(dev + hp.o_pstatus);
  d.by_buckets = hp.by_buckets ? 1u : 0u;
  d.num_large = hp.num_large;
  if (hp.by_buckets) {
    d.status_sets = hp.status_sets;
    d.sb.whole = (uint32_t)hp.bjobs.size();
    d.declined = reinterpret_cast<uint32_t*>(dev + hp.o_decl);
    d.declined_tile = reinterpret_cast<DeclinedTile*>(dev + hp.o_dtile);
    d.declined_chunk = reinterpret_cast<uint2*>(dev + hp.o_dchunk);
    d.sb.rare = reinterpret_cast<uint32_t*>(dev + hp.o_rare);
    d.sb.num = (uint32_t)hp.bsegs.size();
    d.sb.buckets = hp.buckets;
    d.sb.tiles = hp.part_tiles;
    d.sb.chunks = hp.hist_items;
    d.sb.seg = reinterpret_cast<const BucketSeg*>(dev + hp.o_bseg);
    d.sb.of_large = reinterpret_cast<const uint32_t*>(dev + hp.o_of_large);
    d.sb.map = reinterpret_cast<SegMap*>(dev + hp.o_map);
    d.sb.count = reinterpret_cast<uint32_t*>(dev + hp.o_count);
    d.sb.tile_job = reinterpret_cast<SegTileJob*>(dev + hp.o_tjob);
    d.sb.bucket_job = reinterpret_cast<SegBucketJob*>(dev + hp.o_bjob);
  }
  return d;
}

size_t plan_image_bytes(const HostPlan& hp) { return hp.o_tile_seg + std::max<size_t>(hp.tile_seg.size(), 1) * 4; }

cudaError_t upload_plan(const HostPlan& hp, char* dev, cudaStream_t s, void* pinned_staging) {
  cudaError_t e = cudaSuccess;
  if (pinned_staging && hp.by_buckets) return cudaErrorInvalidValue;  // (its tables are not in the image)
  if (pinned_staging) {
    char* img = static_cast<char*>(pinned_staging);
    const size_t bytes = plan_image_bytes(hp);
    std::memset(img, 0, bytes);
    if (!hp.items.empty()) std::memcpy(img + hp.o_items, hp.items.data(), hp.items.size() * sizeof(Item));
    std::memcpy(img + hp.o_off, hp.off.data(), hp.off.size() * 8);
    if (!hp.large.empty()) std::memcpy(img + hp.o_large, hp.large.data(), hp.large.size() * sizeof(LargeSeg));
    if (!hp.tile_seg.empty()) std::memcpy(img + hp.o_tile_seg, hp.tile_seg.data(), hp.tile_seg.size() * 4);
    e = cudaMemcpyAsync(dev, img, bytes, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(dev + hp.o_err, 0, 256, s);
    return e;
  }
  if (!hp.items.empty())
    e = cudaMemcpyAsync(dev + hp.o_items, hp.items.data(), hp.items.size() * sizeof(Item), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(dev + hp.o_off, hp.off.data(), hp.off.size() * 8, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && !hp.large.empty())
    e = cudaMemcpyAsync(dev + hp.o_large, hp.large.data(), hp.large.size() * sizeof(LargeSeg),
                        cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && !hp.tile_seg.empty())
    e = cudaMemcpyAsync(dev + hp.o_tile_seg, hp.tile_seg.data(), hp.tile_seg.size() * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && !hp.bsegs.empty())
    e = cudaMemcpyAsync(dev + hp.o_bseg, hp.bsegs.data(), hp.bsegs.size() * sizeof(BucketSeg), cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && !hp.of_large.empty())
    e = cudaMemcpyAsync(dev + hp.o_of_large, hp.of_large.data(), hp.of_large.size() * 4, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && !hp.bjobs.empty())  // (the partitioned segments' jobs, behind them, are written by each run)
    e = cudaMemcpyAsync(dev + hp.o_bjob, hp.bjobs.data(), hp.bjobs.size() * sizeof(SegBucketJob),
                        cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(dev + hp.o_err, 0, 256, s);
  return e;
}

unsigned plan_grid(const HostPlan& hp) {
  if (ensure_dynamic_smem(hp.kc.fn, hp.kc.smem) != cudaSuccess) cudaGetLastError();  // the launch reports it
  if (hp.split && ensure_dynamic_smem(hp.by_buckets ? declined_pass_kernel : seg_pass_kernel, PassGeometry::kBytes) != cudaSuccess)
    cudaGetLastError();
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, hp.kc.fn, kBlock, hp.kc.smem) != cudaSuccess) {
    cudaGetLastError();
    per_sm = 1;
  }
  unsigned grid = (unsigned)std::max(1, per_sm) * (unsigned)device_info().sm_count;
  const uint32_t items = (uint32_t)hp.items.size();
  if (items < grid) grid = std::max<uint32_t>(items, 1);
  return grid;
}

namespace {

// Keys of a batch whose declined segments get a stream of their own: above,
// launches are long and nothing is gained.
constexpr size_t kForkMostKeys = (size_t)1 << 27;

// The declined segments' digit passes (launches that return at once when there
// are none).
cudaError_t launch_declined(const HostPlan& hp, const PlanDev& pd, cudaStream_t s) {
  const unsigned sms = (unsigned)device_info().sm_count;
  const size_t hist_smem = (size_t)4 * 256 * hist_lanes<8>() * 4;
  declined_counts_kernel<<<sms * 2, kBlock, hist_smem, s>>>(pd);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  declined_scan_kernel<<<std::min<unsigned>(hp.num_large, sms * 4), kBlock, 0, s>>>(pd);
  e = cudaGetLastError();
  for (uint32_t p = 0; p < hp.passes && e == cudaSuccess; ++p) {
    if (p > 0 && hp.status_sets == 1) declined_clear_kernel<<<sms * 4, 256, 0, s>>>(pd);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    declined_pass_kernel<<<std::min<unsigned>(hp.pass_tiles, sms * 3), kPassBlock, PassGeometry::kBytes, s>>>(pd, p);
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace

cudaError_t launch_plan(const HostPlan& hp, const PlanDev& pd, char* dev, unsigned grid, cudaStream_t s,
                        const PlanFork* fork) {
  cudaError_t e = cudaMemsetAsync(dev + hp.o_head, 0, hp.o_pticket + 256 - hp.o_head, s);
  if (e != cudaSuccess) return e;
  if (hp.by_buckets) {
    const size_t total = hp.off.empty() ? 0 : (size_t)hp.off.back();
    if ((e = launch_seg_plan(pd, s)) != cudaSuccess) return e;
    if (hp.pass_tiles == 0) return launch_seg_buckets(pd, total, s);
    if (!fork || total > kForkMostKeys) {
      e = launch_seg_buckets(pd, total, s);
      return e != cudaSuccess ? e : launch_declined(hp, pd, s);
    }
    // From here on the two kinds of segments share neither keys nor tables, and in
    // small batches each launch is mostly latency: side by side.  (us a run, one
    // behind the other -> beside, both before crowding was looked at: 64 arrays of 1 K
    // to 50 K skewed keys 122 -> 94, 300 of 1 K to 1 M 950 -> 925, uniform 379 -> 379;
    // 1000 of 1 M 17.1 ms both ways.)
    if ((e = cudaEventRecord(fork->leave, s)) != cudaSuccess) return e;
    if ((e = cudaStreamWaitEvent(fork->side, fork->leave, 0)) != cudaSuccess) return e;
    e = launch_declined(hp, pd, fork->side);
    const cudaError_t e2 = launch_seg_buckets(pd, total, s);
    // (always back, so that nothing outlives the call's place in its stream)
    const cudaError_t e3 = cudaEventRecord(fork->back, fork->side), e4 = cudaStreamWaitEvent(s, fork->back, 0);
    for (const cudaError_t x : {e2, e3, e4})
      if (e == cudaSuccess) e = x;
    return e;
  }
  if (!hp.items.empty()) {
    hp.kc.fn<<<grid, kBlock, hp.kc.smem, s>>>(pd);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (!hp.split || hp.pass_tiles == 0) return cudaSuccess;
  for (uint32_t p = 0; p < hp.passes && e == cudaSuccess; ++p) {
    e = cudaMemsetAsync(dev + hp.o_pstatus, 0, (size_t)hp.pass_tiles * 256 * 4, s);
    if (e == cudaSuccess) {
      seg_pass_kernel<<<hp.pass_tiles, kPassBlock, PassGeometry::kBytes, s>>>(pd, p);
      e = cudaGetLastError();
    }
  }
  return e;
}

}  // namespace seg
}  // namespace pa

using namespace pa;
using namespace pa::seg;

struct pa_segsort_plan {
  int device = -1;
  size_t num_segments = 0;
  unsigned long long total_keys = 0;
  HostPlan hp;
  unsigned grid = 0;
  char* dev = nullptr;
  PlanDev pd{};
  uint32_t* err_host = nullptr;  // page-locked, the device's error word: read without a copy when the stream is done
  cudaStream_t cap_stream = nullptr;
  PlanFork fork;  // (plans by buckets with segments that may be declined)
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  uint32_t* g_keys = nullptr;
  uint32_t* g_tmp = nullptr;
};

namespace {

int cfail(cudaError_t e, const char* what) {
  char buf[256];
  snprintf(buf, sizeof(buf), "%s: %s", what, cudaGetErrorString(e));
  cudaGetLastError();
  return record_error(e == cudaErrorMemoryAllocation ? PA_ERR_OOM : PA_ERR_CUDA, buf);
}

#define PA_SEG_CUDA(call)                                 \
  do {                                                    \
    cudaError_t e_ = (call);                              \
    if (e_ != cudaSuccess) return cfail(e_, #call);       \
  } while (0)

bool dev_ptr(const void* p) {
  cudaPointerAttributes at;
  if (!p || cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  int d = 0;
  cudaGetDevice(&d);
  return (at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged) && at.device == d;
}

void destroy_graph(pa_segsort_plan* p) {
  if (p->exec) cudaGraphExecDestroy(p->exec);
  if (p->graph) cudaGraphDestroy(p->graph);
  p->exec = nullptr;
  p->graph = nullptr;
  p->g_keys = p->g_tmp = nullptr;
}

int enqueue(pa_segsort_plan* p, cudaStream_t s) {
  PA_SEG_CUDA(launch_plan(p->hp, p->pd, p->dev, p->grid, s, p->fork.back ? &p->fork : nullptr));
  // an odd number of passes (11-bit digits: three) leaves every segment in tmp
  if (p->hp.passes & 1u)
    PA_SEG_CUDA(cudaMemcpyAsync(p->pd.keys, p->pd.tmp, (size_t)p->total_keys * 4, cudaMemcpyDeviceToDevice, s));
  return PA_OK;
}

}  // namespace

extern "C" {

int pa_segsort_plan_create(const uint64_t* seg_offsets, size_t num_segments, const pa_segsort_config* cfg,
                           pa_segsort_plan** out) {
  if (!out) return record_error(PA_ERR_ARG, "out is NULL");
  *out = nullptr;
  if (!seg_offsets) return record_error(PA_ERR_ARG, "seg_offsets is NULL");
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) {
    cudaGetLastError();
    return record_error(PA_ERR_NO_DEVICE, "no CUDA device");
  }
  // The offsets must be readable on the host to plan the work.
  std::vector<uint64_t> off(num_segments + 1);
  if (dev_ptr(seg_offsets)) {
    PA_SEG_CUDA(cudaMemcpy(off.data(), seg_offsets, off.size() * 8, cudaMemcpyDeviceToHost));
  } else {
    std::memcpy(off.data(), seg_offsets, off.size() * 8);
  }
  auto* p = new pa_segsort_plan();
  if (int rc = build_host_plan(off.data(), num_segments, cfg, &p->hp, kPasses, true)) {
    delete p;
    return rc;
  }
  cudaGetDevice(&p->device);
  p->num_segments = num_segments;
  p->total_keys = num_segments ? off[num_segments] : 0;
  cudaError_t e = cudaMalloc(&p->dev, p->hp.bytes);
  if (e != cudaSuccess) {
    delete p;
    return cfail(e, "cudaMalloc(plan)");
  }
  e = cudaMallocHost(&p->err_host, sizeof(uint32_t));
  if (e == cudaSuccess) e = upload_plan(p->hp, p->dev, (cudaStream_t)0);
  if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)0);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&p->cap_stream, cudaStreamNonBlocking);
  if (p->hp.by_buckets && p->hp.pass_tiles) {
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&p->fork.side, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&p->fork.leave, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&p->fork.back, cudaEventDisableTiming);
  }
  if (e != cudaSuccess) {
    pa_segsort_plan_destroy(p);
    return cfail(e, "plan set-up");
  }
  p->grid = plan_grid(p->hp);
  p->pd = device_view(p->hp, p->dev, nullptr, nullptr);
  *p->err_host = 0;
  p->pd.err = p->err_host;
  *out = p;
  return PA_OK;
}

int pa_segsort_plan_info(const pa_segsort_plan* p, uint32_t* num_small, uint32_t* num_large, uint32_t* num_items) {
  if (!p) return record_error(PA_ERR_ARG, "plan is NULL");
  if (num_small) *num_small = p->hp.num_small;
  if (num_large) *num_large = p->hp.num_large;
  if (num_items) *num_items = (uint32_t)p->hp.items.size();
  return PA_OK;
}

int pa_segsort_plan_run(pa_segsort_plan* p, uint32_t* keys, uint32_t* tmp, const pa_opts* opts) {
  if (!p) return record_error(PA_ERR_ARG, "plan is NULL");
  if (p->total_keys == 0) return PA_OK;
  if (!dev_ptr(keys) || !dev_ptr(tmp))
    return record_error(PA_ERR_ARG, "keys and tmp must be device memory holding the plan's total key count");
  cudaStream_t s = opts ? static_cast<cudaStream_t>(opts->stream) : (cudaStream_t)0;
  p->pd.keys = keys;
  p->pd.tmp = tmp;
  if (p->hp.cfg.use_graph) {
    if (!p->exec || p->g_keys != keys || p->g_tmp != tmp) {
      destroy_graph(p);
      PA_SEG_CUDA(cudaStreamBeginCapture(p->cap_stream, cudaStreamCaptureModeThreadLocal));
      const int rc = enqueue(p, p->cap_stream);
      cudaGraph_t g = nullptr;
      const cudaError_t ec = cudaStreamEndCapture(p->cap_stream, &g);
      if (rc != PA_OK) {
        if (g) cudaGraphDestroy(g);
        return rc;
      }
      if (ec != cudaSuccess) return cfail(ec, "cudaStreamEndCapture");
      p->graph = g;
      PA_SEG_CUDA(cudaGraphInstantiate(&p->exec, p->graph, 0));
      p->g_keys = keys;
      p->g_tmp = tmp;
    }
    PA_SEG_CUDA(cudaGraphLaunch(p->exec, s));
  } else {
    if (int rc = enqueue(p, s)) return rc;
  }
  if (opts && opts->async_device) return PA_OK;
  return pa_segsort_plan_sync(p, opts ? opts->stream : nullptr);
}

int pa_segsort_plan_sync(pa_segsort_plan* p, void* stream) {
  if (!p) return record_error(PA_ERR_ARG, "plan is NULL");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  PA_SEG_CUDA(cudaStreamSynchronize(s));
  if (*const_cast<volatile uint32_t*>(p->err_host)) {
    *const_cast<volatile uint32_t*>(p->err_host) = 0;
    return record_error(PA_ERR_TIMEOUT, "a bounded device-side wait of the batched sort gave up");
  }
  return PA_OK;
}

int pa_segsort_plan_destroy(pa_segsort_plan* p) {
  if (!p) return PA_OK;
  destroy_graph(p);
  if (p->cap_stream) cudaStreamDestroy(p->cap_stream);
  if (p->fork.side) cudaStreamDestroy(p->fork.side);
  if (p->fork.leave) cudaEventDestroy(p->fork.leave);
  if (p->fork.back) cudaEventDestroy(p->fork.back);
  if (p->dev) cudaFree(p->dev);
  if (p->err_host) cudaFreeHost(p->err_host);
  delete p;
  return PA_OK;
}

int pa_segmented_sort_u32(uint32_t* keys, const uint64_t* seg_offsets, size_t num_segments,
                          const pa_segsort_config* cfg, const pa_opts* opts) {
  if (num_segments == 0) return PA_OK;
  if (!keys || !seg_offsets) return record_error(PA_ERR_ARG, "NULL buffer");
  pa_segsort_plan* p = nullptr;
  pa_segsort_config c{};
  if (cfg) c = *cfg;
  c.use_graph = 0;  // one-shot: nothing to replay
  if (int rc = pa_segsort_plan_create(seg_offsets, num_segments, &c, &p)) return rc;
  const size_t n = (size_t)p->total_keys;
  cudaStream_t s = opts ? static_cast<cudaStream_t>(opts->stream) : (cudaStream_t)0;
  uint32_t* d_keys = keys;
  uint32_t* d_tmp = nullptr;
  const bool host = !dev_ptr(keys);
  cudaError_t e = cudaSuccess;
  if (n && host) e = cudaMalloc(&d_keys, n * 4);
  if (e == cudaSuccess && n) e = cudaMalloc(&d_tmp, n * 4);
  if (e == cudaSuccess && n && host) e = cudaMemcpyAsync(d_keys, keys, n * 4, cudaMemcpyHostToDevice, s);
  int rc = PA_OK;
  if (e != cudaSuccess) {
    rc = cfail(e, "batched sort buffers");
  } else if (n) {
    pa_opts o{};
    if (opts) o = *opts;
    o.async_device = 0;
    rc = pa_segsort_plan_run(p, d_keys, d_tmp, &o);
    if (rc == PA_OK && host) {
      e = cudaMemcpyAsync(keys, d_keys, n * 4, cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) rc = cfail(e, "copy back");
    }
  }
  if (d_tmp) cudaFree(d_tmp);
  if (host && d_keys && d_keys != keys) cudaFree(d_keys);
  pa_segsort_plan_destroy(p);
  return rc;
}

}  // extern "C"
