// Keys-only sorts by buckets (MSD): two partition passes, then one pass that
// sorts every bucket in shared memory.
//
// A sort of keys alone has one result whatever the order equal keys were
// moved in, so its passes need not be stable, and an unstable partition is
// much cheaper than the stable digit pass of pa_onesweep.cu: a key's place in
// its tile is the value a shared-memory atomic returns (no lane matching, no
// per-warp counters), and a tile's place in a bin is one global atomic per bin
// (no look-back).  Keys cross memory 1 + 2 + 2 + 2 times (count, partition,
// partition, bucket sort) against 1 + 2 * 4 (1 + 2 * 8 for 64-bit keys).
//
//   bucket_plan_kernel     one cluster of 8 CTAs reads 16384 keys, one at a
//                          random place of each stride, takes the range they
//                          span, and lays nb equal buckets over it (BucketMap);
//                          counts the sample per bucket to judge the fit: a
//                          sample that crowds into few buckets leaves the sort
//                          to the LSD passes, which do not mind how keys are
//                          spread;
//   bucket_count_kernel    one read: exact keys per bucket, and the cells of a few
//                          buckets; the last CTA turns the counts into bucket
//                          starts and cursors, or the sort away;
//   bucket_scatter_kernel  one tile at a time: rank, reserve, stage by bin,
//                          write out in bin-contiguous runs.  First on the
//                          bucket's high bits (keys -> tmp), then, bucket
//                          group by bucket group, on its low bits (tmp ->
//                          keys).  At most 256 buckets: one pass (keys -> tmp);
//   bucket_finish_kernel   one CTA per bucket: the keys set bits of a bitmap of
//                          their range, and a key's place is the number of bits
//                          set below its own.
//
// The map is monotone in the key whatever the sample was, so the sample
// decides only how evenly the buckets fill, never the result.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "pa_common.cuh"
#include "pa_kernels.cuh"
#include "pa_onesweep_tile.cuh"
#include "pa_segmented.cuh"

namespace pa {
namespace {

namespace cg = cooperative_groups;

constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr int kPlanCtas = 8;
constexpr int kPlanBlock = 1024;
constexpr int kPlanPer = 2;  // sample keys per thread
constexpr int kSampleLog2 = 14;
constexpr uint32_t kSample = 1u << kSampleLog2;
static_assert(kSample == (uint32_t)kPlanCtas * kPlanBlock * kPlanPer, "a key per thread and round");
constexpr uint32_t kGroups = 256;         // bins of a partition pass, at most
constexpr uint32_t kPlanParts = 64;       // parts of the buckets whose shares of the sample the plan looks at
// Keys in buckets beyond the finish kernel, which go through bucket_rare_kernel at
// about 27 us a million (100M keys, all of them in such buckets: 3.6 ms against
// 1.66 by digits and 0.93 without): up to an eighth of the keys, what a bucket sort
// gains over the digit passes (8.6 us a million) pays for several times over.
constexpr uint32_t kOverShare = 8;
constexpr uint32_t kBucketsMax = 32768;   // counters of the count kernel: 128 KB of shared memory
constexpr uint32_t kBucketTarget = 3072;  // keys per bucket, at most, while more buckets can be had
static_assert(kBucketMostKeys == (size_t)kBucketsMax * kBucketTarget, "the declared limit");
constexpr uint32_t kFinishCap = 4096;     // keys of a bucket the finish kernel holds
constexpr int kCellBits = 16, kBinBits = 12;
constexpr uint32_t kCells = 1u << kCellBits;      // cells of the finish kernel's bitmap
constexpr uint32_t kCountSpan = 1u << (kCellBits - 3);  // values a counted bucket may span
constexpr uint32_t kBucketBins = 1u << kBinBits;  // values a crowded bucket may span to be counted instead
constexpr int kFinishBlock = 256;
constexpr uint32_t kEntryHits = 6;  // keys of one entry of the bitmap that found their cell taken, at most
// Keys may crowd into few cells of every bucket however evenly these fill (multiples
// of some number, few prefixes with small numbers behind them, clusters): the finish
// kernel then leaves nearly all of them to bucket_rare_kernel.  So the count kernel
// lays out half of the cells of kCrowdBuckets buckets (an entry: 32 cells' bits,
// and its keys, as the finish kernel has them), and turns the sort away where those
// with too many keys in taken cells hold more than 3/8 of their keys.
constexpr int kCrowdLog2 = 3;
constexpr uint32_t kCrowdBuckets = 1u << kCrowdLog2;
constexpr uint32_t kCrowdEntries = kCells / 32 / 2;
constexpr uint32_t kCrowdHits = kFinishBlock / 2;  // keys in taken cells of half of a bucket's, at most

struct BucketArgs {
  BucketMap* map;
  SortCtrl* ctrl;
  uint32_t* count;
  uint32_t* start;
  uint32_t* cursor;
  uint32_t* group_cursor;
  uint32_t* tile_first;
  uint32_t* rare;
  uint32_t nb;
  uint32_t nb_bits;     // nb = 1 << nb_bits
  uint32_t low_bits;
  uint32_t tile;        // keys per partition tile
  uint32_t tmp_align;   // scratch address modulo 16
  size_t keys;          // of the sort
  uint32_t hot_above;   // sample keys above which a bucket looks too full
  uint32_t max_sample;  // sample keys no bucket may exceed
  uint32_t* err;
  SortWords* words;     // where plan and count tell a host that waits (may be null)
};

// What plan and count turn a sort away for, besides.  (Not in BucketArgs: words
// more there cost the partition passes 1 % at 100M keys.)
struct BucketLimits {
  uint32_t dense_above;  // sample keys above which a 64th of the buckets looks too full
  uint32_t most_keys;   // keys no bucket may exceed
  uint32_t most_over;   // keys that may lie in buckets beyond the finish kernel
  uint2* crowd;         // [kCrowdBuckets][kCrowdEntries] in the scratch array, not yet in use (may be null)
};

// t: the key's distance from the bottom of the map, in 32 bits.
template <typename K>
__device__ __forceinline__ uint32_t map_t(K key, K lo, uint32_t s) {
  if constexpr (sizeof(K) == 4) {
    (void)s;
    return key > lo ? key - lo : 0u;
  } else {
    const K t = (key > lo ? key - lo : (K)0) >> s;
    return t > (K)0xFFFFFFFFu ? 0xFFFFFFFFu : (uint32_t)t;
  }
}
__device__ __forceinline__ uint32_t map_bucket(uint32_t t, uint32_t mult, uint32_t last) {
  return min(__umulhi(t, mult), last);
}

// The key's top 32 bits: its distance from the bottom of a plain map.
__device__ __forceinline__ uint32_t top_word(uint32_t key) { return key; }
__device__ __forceinline__ uint32_t top_word(unsigned long long key) { return (uint32_t)(key >> 32); }

// Adds a key's cell to a bucket's laid out half: one entry in two, by the parity of
// all bits of its number and the bucket's (`part`), so that multiples of a power of
// two do not all miss it.
__device__ __forceinline__ void crowd_add(uint2* crowd, uint32_t cell, uint32_t part) {
  const uint32_t entry = (cell / 32) & (2 * kCrowdEntries - 1);
  if ((__popc(entry) ^ part) & 1u) return;
  atomicOr(&crowd[entry / 2].x, 1u << (cell & 31u));
  atomicAdd(&crowd[entry / 2].y, 1u);
}
// Whether the finish kernel would leave the bucket (its keys: cnt) to the rare launch,
// as far as its half tells: too many keys in taken cells, an entry with too many of
// them, or the half's share of the keys missing, which are then crowded elsewhere.
__device__ __forceinline__ bool crowd_listed(uint32_t cnt, uint32_t hits, uint32_t full, uint32_t seen) {
  return hits > kCrowdHits || full != 0 || (cnt > 256 && seen < cnt / 4);
}

// Elements from the 16-byte boundary at or below p to p.
template <typename K>
__device__ __forceinline__ uint32_t skew_of(const K* p) {
  return (uint32_t)(reinterpret_cast<uintptr_t>(p) & 15u) / (uint32_t)sizeof(K);
}

template <typename K>
__device__ __forceinline__ void warp_minmax(K& lo, K& hi) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const K a = __shfl_xor_sync(kFull, lo, o), b = __shfl_xor_sync(kFull, hi, o);
    lo = a < lo ? a : lo;
    hi = b > hi ? b : hi;
  }
}

// ---------------------------------------------------------------------------
// Plan.
// ---------------------------------------------------------------------------
// Latency only (about 16 K scattered sectors): one cluster instead of one CTA,
// so that the sample's loads and its per-bucket counts (each CTA holds 1/8 of
// them, reached through distributed shared memory) are spread over 8 SMs, and
// cluster barriers instead of global tickets, so that nothing has to be zeroed
// first.
template <typename K>
__global__ void __cluster_dims__(kPlanCtas, 1, 1) __launch_bounds__(kPlanBlock)
    bucket_plan_kernel(const K* __restrict__ keys, size_t n, BucketArgs a, BucketLimits most) {
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ uint32_t s_hist[kBucketsMax / kPlanCtas];
  __shared__ K s_lo[32], s_hi[32];
  __shared__ K s_cta_lo[kPlanCtas], s_cta_hi[kPlanCtas];
  __shared__ uint32_t s_mult, s_s;
  __shared__ K s_base;
  __shared__ uint32_t s_max[kPlanCtas], s_hot[kPlanCtas], s_dense;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const uint32_t rank = cluster.block_rank();
  K k[kPlanPer];
  K lo = ~(K)0, hi = 0;
#pragma unroll
  for (int j = 0; j < kPlanPer; ++j) {
    const uint32_t i = ((uint32_t)j * kPlanCtas + rank) * kPlanBlock + tid;
    k[j] = keys[sample_place(i, kSampleLog2, n)];
    lo = min(lo, k[j]);
    hi = max(hi, k[j]);
  }
  for (uint32_t i = tid; i < a.nb / kPlanCtas; i += kPlanBlock) s_hist[i] = 0;
  if (tid == 0) s_dense = 0;
  warp_minmax(lo, hi);
  if (lane == 0) {
    s_lo[warp] = lo;
    s_hi[warp] = hi;
  }
  cluster.sync();  // (every CTA of the cluster runs before its memory is written from another)
  chain_next();
  if (warp == 0) {
    lo = s_lo[lane];
    hi = s_hi[lane];
    warp_minmax(lo, hi);
    if (lane < (uint32_t)kPlanCtas) {
      cluster.map_shared_rank(s_cta_lo, lane)[rank] = lo;
      cluster.map_shared_rank(s_cta_hi, lane)[rank] = hi;
    }
  }
  cluster.sync();
  K raw = 0;  // (thread 0) the sample's range
  if (tid == 0) {
    for (int c = 0; c < kPlanCtas; ++c) {
      lo = min(lo, s_cta_lo[c]);
      hi = max(hi, s_cta_hi[c]);
    }
    // widen by 1/1024 each way: about 16 keys of the sample's spacing, so that
    // few keys of an even spread fall outside and crowd into the end buckets
    // (unless that made the buckets too wide to be counted)
    raw = hi - lo;
    K pad = raw >> 10;
    const K most = (K)kCountSpan * a.nb;
    if (raw < most && raw + 2 * pad >= most) pad = 0;
    lo -= min(lo, pad);
    hi += min((K)(~(K)0 - hi), pad);
    // keys over most of their type's range: the map is their top bits, which
    // costs the partition passes a shift instead of a subtract and a multiply
    if (hi - lo >= (~(K)0 >> 3) * 7) {
      lo = 0;
      hi = ~(K)0;
    }
    uint32_t s = 0;
    if constexpr (sizeof(K) == 8) s = (uint32_t)max(0, 32 - __clzll((long long)(hi - lo)));
    const unsigned long long range = (unsigned long long)((hi - lo) >> s) + 1;
    const unsigned long long mult = ((unsigned long long)a.nb << 32) / range;
    s_mult = mult > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)mult;
    s_s = s;
    s_base = lo;
  }
  __syncthreads();
  const uint32_t mult = s_mult, s = s_s, last = a.nb - 1;
  const K base = s_base;
  const uint32_t per = a.nb / kPlanCtas;
#pragma unroll
  for (int j = 0; j < kPlanPer; ++j) {
    const uint32_t b = map_bucket(map_t<K>(k[j], base, s), mult, last);
    uint32_t* c = cluster.map_shared_rank(s_hist, b / per) + b % per;
    if (__all_sync(kFull, b == __shfl_sync(kFull, b, 0))) {  // (constant keys: one add, not 32 in turn)
      if (lane == 0) atomicAdd(c, 32u);
    } else {
      atomicAdd(c, 1u);
    }
  }
  cluster.sync();
  // the keys of the sample in 64ths of the buckets that look fuller than the
  // finish kernel holds on average: the sample tells a 64th's keys to a sixteenth,
  // a bucket's not at all where there are more buckets than sample keys
  if (warp < kPlanParts / kPlanCtas) {
    const uint32_t part = a.nb / kPlanParts;
    uint32_t c = 0;
    for (uint32_t i = lane; i < part; i += 32) c += s_hist[warp * part + i];
    c = __reduce_add_sync(kFull, c);
    if (lane == 0 && c > most.dense_above) atomicAdd(cluster.map_shared_rank(&s_dense, 0), c);
  }
  // the fullest bucket, and the keys of the sample in buckets that look fuller
  // than the finish kernel holds
  uint32_t mx = 0, hot = 0;
  for (uint32_t i = tid; i < per; i += kPlanBlock) {
    const uint32_t c = s_hist[i];
    mx = max(mx, c);
    hot += c > a.hot_above ? c : 0u;
  }
  mx = __reduce_max_sync(kFull, mx);
  hot = __reduce_add_sync(kFull, hot);
  __syncthreads();  // s_lo is free
  uint32_t* w = reinterpret_cast<uint32_t*>(s_lo);
  uint32_t* w2 = reinterpret_cast<uint32_t*>(s_hi);
  if (lane == 0) {
    w[warp] = mx;
    w2[warp] = hot;
  }
  __syncthreads();
  if (warp == 0) {
    mx = __reduce_max_sync(kFull, w[lane]);
    hot = __reduce_add_sync(kFull, w2[lane]);
    if (lane == 0) {
      cluster.map_shared_rank(s_max, 0)[rank] = mx;
      cluster.map_shared_rank(s_hot, 0)[rank] = hot;
    }
  }
  cluster.sync();
  if (rank == 0 && tid == 0) {
    for (int c = 1; c < kPlanCtas; ++c) {
      mx = max(mx, s_max[c]);
      hot += s_hot[c];
    }
    bool fits = mx <= a.max_sample && hot <= kSample / 64 && s_dense <= kSample / kOverShare;
    BucketMap m{};
    m.plain = base == 0 && mult == a.nb && s == 8 * sizeof(K) - 32 ? 1u : 0u;
    m.mult = mult;
    m.inv = (1ull << 63) / mult;
    m.s = s;
    m.lo = base;
    // cells of the finish kernel: the widest bucket spans ceil(2^32 / mult)
    // values of t, 2^s keys each
    const unsigned long long width = ((1ull << 32) + mult - 1) / mult;
    uint32_t sh = 0;
    while (((width - 1) >> sh) >= kCells) ++sh;
    m.cell_shift = sh + s;
    m.counts = s == 0 && width <= kCountSpan ? 1u : 0u;
    // Buckets of few values are counted.  Where they span too many for that and too
    // few for the bitmap (200 of m keys meet another), the LSD passes run, as they
    // do for ranges of two digits whose counters would see every value hundreds of
    // times (100M keys of 16 bits: 922 us by digits, 1275 by buckets).
    const unsigned long long per = a.keys / a.nb;
    if (!m.counts && s < 16 && per * per > (400 * width) << s) fits = false;
    if (m.counts && raw < 65536 && a.keys / ((unsigned long long)raw + 1) > 512) fits = false;
    m.on = fits ? 1u : 0u;
    *a.map = m;
    a.rare[0] = 0;
    if (fits) {  // the LSD passes enqueued behind this sort do nothing
      for (int p = 0; p < kMaxPasses; ++p) a.ctrl->pass[p].skip = 1;
      a.ctrl->final_in_tmp = 0;
    }
    if (a.words) {  // (the caller polls it)
      __threadfence_system();
      *reinterpret_cast<volatile uint32_t*>(&a.words->decided) = fits ? 1u : 0u;
    }
  }
  // (last, so that no cluster barrier waits for these stores)
  for (uint32_t i = rank * kPlanBlock + tid; i < a.nb; i += kPlanCtas * kPlanBlock) a.count[i] = 0;
  if (most.crowd)
    for (uint32_t i = rank * kPlanBlock + tid; i < kCrowdBuckets * kCrowdEntries; i += kPlanCtas * kPlanBlock)
      most.crowd[i] = make_uint2(0u, 0u);
}

// ---------------------------------------------------------------------------
// Count.
// ---------------------------------------------------------------------------
// One read against a shared counter per bucket (up to 128 KB, so one CTA per
// SM).  A thread's next four 16-byte loads are issued before the current ones
// are counted: 32 warps alone left the SM waiting for loads half of the time.
// 100M 32-bit keys: 0.105 ms, 3.8 TB/s (the digit histogram it replaces, with
// its tile tables: 0.113 ms).
constexpr int kCountBlock = 1024;

template <typename K, bool CROWD>
__global__ void __launch_bounds__(kCountBlock, 1) bucket_count_kernel(const K* __restrict__ keys, size_t n,
                                                                      BucketArgs a, BucketLimits most) {
  extern __shared__ __align__(16) uint32_t s_cnt[];
  __shared__ uint32_t s_warp[kCountBlock / 32];
  __shared__ uint32_t s_last, s_over;
  __shared__ uint32_t s_hits[kCrowdBuckets], s_full[kCrowdBuckets], s_seen[kCrowdBuckets];
  constexpr int V = 16 / (int)sizeof(K);
  const uint32_t tid = threadIdx.x;
  for (uint32_t i = tid; i < a.nb; i += kCountBlock) s_cnt[i] = 0;
  if (tid == 0) s_over = 0;
  if (tid < kCrowdBuckets) s_hits[tid] = s_full[tid] = s_seen[tid] = 0;
  chain_wait();
  chain_next();
  const BucketMap m = *a.map;
  if (!m.on) return;
  __syncthreads();
  const uint32_t last = a.nb - 1;
  // the buckets whose cells are laid out: one in nb / kCrowdBuckets, none of them at
  // the map's ends (pick beyond every bucket: none at all)
  const bool crowd = CROWD && !m.counts;
  const uint32_t crowd_mask = a.nb / kCrowdBuckets - 1;
  const uint32_t pick = crowd ? (crowd_mask * 5) >> 3 : 0xFFFFFFFFu;
  auto count = [&](auto plainc) {
    constexpr bool PLAIN = decltype(plainc)::value;
    const K lo = (K)m.lo;
    const uint32_t shift = 32u - a.nb_bits;
    auto bucket = [&](K key) {
      if constexpr (PLAIN) return top_word(key) >> shift;
      else return map_bucket(map_t<K>(key, lo, m.s), m.mult, last);
    };
    auto look = [&](const K* k) {  // a vector's keys (few have one that is looked at)
      if constexpr (CROWD) {
        bool any = false;
#pragma unroll
        for (int e = 0; e < V; ++e) any = any || (bucket(k[e]) & crowd_mask) == pick;
        if (!any) return;
        for (int e = 0; e < V; ++e) {
          const uint32_t b = bucket(k[e]), j = b >> (a.nb_bits - kCrowdLog2);
          if ((b & crowd_mask) == pick)
            crowd_add(most.crowd + j * kCrowdEntries, (uint32_t)((PLAIN ? k[e] : k[e] - lo) >> m.cell_shift), j);
        }
      }
    };
    const uintptr_t addr = reinterpret_cast<uintptr_t>(keys);
    size_t head = ((16u - (addr & 15u)) & 15u) / sizeof(K);
    if (head > n) head = n;
    const size_t nvec = (n - head) / V;
    const size_t tail = head + nvec * V;
    const uint4* vec = reinterpret_cast<const uint4*>(keys + head) + tid;
    const size_t stride = (size_t)gridDim.x * kCountBlock;
    constexpr int U = 4;
    // whole rounds of U vectors per thread (every lane of a warp takes part),
    // the next round's loads issued before this one's keys are counted
    size_t i = (size_t)blockIdx.x * kCountBlock;
    auto whole = [&](size_t at) { return at + (U - 1) * stride + kCountBlock <= nvec; };
    uint4 q[U];
    if (whole(i)) {
#pragma unroll
      for (int u = 0; u < U; ++u) q[u] = ld_stream_v4(vec + i + u * stride);
    }
    while (whole(i)) {
      const size_t nx = i + U * stride;
      const bool more = whole(nx);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint4 w = q[u];
        if (more) q[u] = ld_stream_v4(vec + nx + u * stride);
        const K* k = reinterpret_cast<const K*>(&w);
        const uint32_t d0 = bucket(k[0]);
        bool one = d0 == __shfl_sync(kFull, d0, 0);
        if (__all_sync(kFull, one)) {
          // sorted or constant runs: one add for a warp that agrees, where its
          // atomics would queue on one word
#pragma unroll
          for (int e = 1; e < V; ++e) one = one && bucket(k[e]) == d0;
          if (__all_sync(kFull, one)) {
            if ((tid & 31u) == 0) atomicAdd(s_cnt + d0, 32u * V);
            if ((d0 & crowd_mask) == pick) look(k);
            continue;
          }
        }
#pragma unroll
        for (int e = 0; e < V; ++e) atomicAdd(s_cnt + bucket(k[e]), 1u);
        look(k);
      }
      i = nx;
    }
    for (; i < nvec; i += stride) {
      if (i + tid < nvec) {
        const uint4 w = ld_stream_v4(vec + i);
        const K* k = reinterpret_cast<const K*>(&w);
#pragma unroll
        for (int e = 0; e < V; ++e) atomicAdd(s_cnt + bucket(k[e]), 1u);
        look(k);
      }
    }
    if (blockIdx.x == 0) {  // head and tail: fewer than 2 * V keys
      const size_t rest = head + (n - tail);
      for (size_t r = tid; r < rest; r += kCountBlock) atomicAdd(s_cnt + bucket(keys[r < head ? r : tail + (r - head)]), 1u);
    }
  };
  if (m.plain) count(std::true_type{});
  else count(std::false_type{});
  __syncthreads();
  // each CTA adds its counts starting at another place, so that CTAs that end
  // together do not queue on the same words
  const uint32_t off = (uint32_t)(((unsigned long long)blockIdx.x * a.nb) / gridDim.x);
  for (uint32_t j = tid; j < a.nb; j += kCountBlock) {
    const uint32_t b = (j + off) & last;
    const uint32_t c = s_cnt[b];
    if (c) atomicAdd(a.count + b, c);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(&a.map->ticket, 1u) == gridDim.x - 1u ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // The last CTA: whether the buckets fit after all, their starts, cursors of both
  // passes, and the second pass's tiles per group (tile_first).
  const uint32_t per = max(1u, a.nb / kCountBlock);  // buckets per thread
  if (crowd) {  // four warps a laid out bucket: its keys in taken cells, entries with too many of them
    constexpr uint32_t kWarps = kCountBlock / 32 / kCrowdBuckets;
    constexpr uint32_t kPer = kCrowdEntries / 2 / kWarps;  // 16-byte words, two entries, per warp
    const uint32_t j = (tid >> 5) / kWarps;
    const uint4* e = reinterpret_cast<const uint4*>(most.crowd + j * kCrowdEntries) + ((tid >> 5) % kWarps) * kPer;
    uint32_t hits = 0, full = 0, seen = 0;
#pragma unroll
    for (uint32_t q = 0; q < kPer / 32; ++q) {
      const uint4 x = __ldcg(e + q * 32 + (tid & 31u));
      const uint32_t h0 = x.y - __popc(x.x), h1 = x.w - __popc(x.z);
      hits += h0 + h1;
      seen += x.y + x.w;
      full |= max(h0, h1) > kEntryHits ? 1u : 0u;
    }
    hits = __reduce_add_sync(kFull, hits);
    full = __reduce_or_sync(kFull, full);
    seen = __reduce_add_sync(kFull, seen);
    if ((tid & 31u) == 0) {
      atomicAdd(&s_hits[j], hits);
      atomicOr(&s_full[j], full);
      atomicAdd(&s_seen[j], seen);
    }
  }
  if (a.nb >= (uint32_t)kCountBlock) {
    for (uint32_t j = tid * 4; j < a.nb; j += kCountBlock * 4)
      *reinterpret_cast<uint4*>(s_cnt + j) = __ldcg(reinterpret_cast<const uint4*>(a.count + j));
  } else if (tid < a.nb) {
    s_cnt[tid] = __ldcg(a.count + tid);
  }
  __syncthreads();
  uint32_t local = 0, over = 0;
  bool large = false;
  if (tid * per < a.nb)
    for (uint32_t j = 0; j < per; ++j) {
      const uint32_t c = s_cnt[tid * per + ((j + tid) & (per - 1))];
      local += c;
      over += c > kFinishCap ? c : 0u;
      large |= c > most.most_keys;
    }
  if (over) atomicAdd(&s_over, over);
  if (crowd && tid < 32) {
    uint32_t c = 0, listed = 0;
    if (tid < kCrowdBuckets) {
      c = s_cnt[tid * (crowd_mask + 1) + pick];
      listed = crowd_listed(c, s_hits[tid], s_full[tid], s_seen[tid]) ? c : 0u;
    }
    large |= __reduce_add_sync(kFull, listed) > __reduce_add_sync(kFull, c) / 8 * 3;
  }
  if (__syncthreads_or(large) || s_over > most.most_over) {
    if (tid == 0) {
      a.map->on = 0;  // (every other CTA is past its look at it; the launches behind find nothing to do)
      if (a.words) *reinterpret_cast<volatile uint32_t*>(&a.words->again) = kAgainByDigits;
    }
    return;
  }
  uint32_t run = os::block_exclusive_scan<kCountBlock>(local, s_warp);
  if (tid * per < a.nb) {
    for (uint32_t j = 0; j < per; ++j) {
      const uint32_t c = s_cnt[tid * per + j];
      s_cnt[tid * per + j] = run;
      run += c;
    }
  }
  __syncthreads();
  for (uint32_t j = tid; j < a.nb; j += kCountBlock) {
    const uint32_t v = s_cnt[j];
    a.start[j] = v;
    a.cursor[j] = v;
  }
  if (tid == 0) a.start[a.nb] = (uint32_t)n;
  const uint32_t groups = a.nb >> a.low_bits;
  uint32_t tiles = 0;
  if (tid < groups) {
    const uint32_t g0 = s_cnt[tid << a.low_bits];
    const uint32_t g1 = tid + 1 < groups ? s_cnt[(tid + 1) << a.low_bits] : (uint32_t)n;
    a.group_cursor[tid] = g0;
    // tiles start at 16-byte boundaries of the input (bucket_scatter_kernel)
    const uint32_t head2 = (uint32_t)(((a.tmp_align + (size_t)g0 * sizeof(K)) & 15u) / sizeof(K));
    tiles = g1 > g0 ? (g1 - g0 + head2 + a.tile - 1) / a.tile : 0;
  }
  __syncthreads();  // s_warp is reused
  const uint32_t before = os::block_exclusive_scan<kCountBlock>(tiles, s_warp);
  if (tid < groups) a.tile_first[tid] = before;
  if (tid == groups - 1) a.tile_first[groups] = before + tiles;
}

// ---------------------------------------------------------------------------
// Partition pass.
// ---------------------------------------------------------------------------
// Bound by the shared-memory / L1 data pipe (84 % of its cycles at 100M
// uniform keys): per 32 keys one atomic, one look-up of the bin's start and one
// store at random places (about 3 cycles each), the sequential read back, the
// look-up of the bin's destination and the stores to global memory.  So what
// counts is the number of shared accesses per key, not registers or occupancy
// (two CTAs per SM measured as three).  A tile's next loads are issued before
// it is written out, and a bin's reservation (a round trip to L2) passes while
// the tile is staged.  100M uniform 32-bit keys: 0.214 ms for the first pass,
// 0.235 ms for the grouped one (sorted keys 0.179 and 0.305; 0.241 and 0.365 while
// tiles of one bin were shuffled like the others and a warp's vectors added one
// after the other), against 0.326 and 0.385 ms for a stable digit
// pass with and without prepared offsets.
constexpr int kScatterBlock = 512;
constexpr int kScatterPerSm = 3;
template <typename K>
constexpr int kScatterItems = sizeof(K) == 4 ? 16 : 8;
template <typename K>
constexpr uint32_t kScatterTile = (uint32_t)kScatterBlock * kScatterItems<K>;

// PLAIN: the map is the key's top bits (BucketMap::plain).
template <typename K, bool GROUPED, bool PLAIN>
__device__ __forceinline__ void scatter_tiles(const K* in, K* out, uint32_t n, const BucketArgs& a, const BucketMap& m,
                                              K* s_keys, uint32_t* s_cnt, uint32_t* s_start, uint32_t* s_base,
                                              uint32_t* s_warp, uint32_t* s_one, const uint32_t* s_first) {
  constexpr int ITEMS = kScatterItems<K>;
  constexpr uint32_t T = kScatterTile<K>;
  constexpr int V = 16 / (int)sizeof(K);
  constexpr int Q = ITEMS / V;  // 16-byte vectors per thread
  const uint32_t tid = threadIdx.x, lane = tid & 31u;
  const uint32_t groups = GROUPED ? a.nb >> a.low_bits : 1u;
  const uint32_t bins = GROUPED ? 1u << a.low_bits : a.nb >> a.low_bits;
  const uint32_t tiles = GROUPED ? s_first[groups] : (n + skew_of(in) + T - 1) / T;
  const K lo = (K)m.lo;
  const uint32_t last = a.nb - 1, mask = bins - 1, shift = GROUPED ? 32u - a.nb_bits : 32u - a.nb_bits + a.low_bits;
  auto digit = [&](K key) {
    if constexpr (PLAIN) {
      const uint32_t d = top_word(key) >> shift;
      return GROUPED ? d & mask : d;
    } else {
      const uint32_t b = map_bucket(map_t<K>(key, lo, m.s), m.mult, last);
      return GROUPED ? b & mask : b >> a.low_bits;
    }
  };
  uint32_t* cursor0 = GROUPED ? a.cursor : (a.low_bits ? a.group_cursor : a.cursor);
  // The tile in hand: keys [g0, g1) of group g; the group's tiles start at the
  // 16-byte boundary at or below g0.
  uint32_t g = 0, g0 = 0, g1 = n;
  long long tlo = 0;
  bool full = false;
  K k[ITEMS];
  uint32_t valid = 0;  // bit j: item j is a key of the tile (not kept for a full tile)
  auto load = [&](uint32_t tile) {
    uint32_t t = tile;
    if constexpr (GROUPED) {
      uint32_t h = groups;  // g: the last group whose first tile is <= tile
      g = 0;
      while (h - g > 1) {
        const uint32_t mid = (g + h) >> 1;
        if (s_first[mid] <= tile) g = mid;
        else h = mid;
      }
      t = tile - s_first[g];
      g0 = a.start[g << a.low_bits];
      g1 = a.start[(g + 1) << a.low_bits];
    }
    tlo = (long long)g0 - skew_of(in + g0) + (long long)t * T;
    full = tlo >= (long long)g0 && tlo + (long long)T <= (long long)g1;
    if (full) {
      const uint4* src = reinterpret_cast<const uint4*>(in + tlo) + tid;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const uint4 v = src[q * kScatterBlock];
        const K* e = reinterpret_cast<const K*>(&v);
#pragma unroll
        for (int i = 0; i < V; ++i) k[q * V + i] = e[i];
      }
    } else {
      valid = 0;
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const long long x = tlo + (long long)j * kScatterBlock + tid;
        const bool ok = x >= (long long)g0 && x < (long long)g1;
        k[j] = ok ? in[x] : (K)0;
        valid |= ok ? 1u << j : 0u;
      }
    }
  };
  if (blockIdx.x < tiles) load(blockIdx.x);
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    if (tid < kGroups) s_cnt[tid] = 0;
    if (tid == 0) *s_one = 0;
    __syncthreads();
    uint32_t r[(ITEMS + 1) / 2];  // ranks in the tile's bins, two 16-bit halves per word
#pragma unroll
    for (int j = 0; j < (ITEMS + 1) / 2; ++j) r[j] = 0;
    if (full) {
      const uint32_t d0 = digit(k[0]);
      if (__all_sync(kFull, d0 == __shfl_sync(kFull, d0, 0))) {
        // Sorted or constant runs: the atomics of a warp that agrees would queue
        // on one word, so where all of a vector's keys agree the warp adds once.
        uint32_t ones = 0, dl = 0;  // bit q: vector q agrees; lane q: its digit
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const uint32_t dq = digit(k[q * V]);
          bool one = dq == __shfl_sync(kFull, dq, 0);
#pragma unroll
          for (int i = 1; i < V; ++i) one = one && digit(k[q * V + i]) == dq;
          ones |= __all_sync(kFull, one) ? 1u << q : 0u;
          if (lane == (uint32_t)q) dl = dq;
        }
        uint32_t x = 0;
        if ((ones >> lane) & 1u) x = atomicAdd(s_cnt + dl, 32u * V);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const uint32_t y = __shfl_sync(kFull, x, q) + lane;
          if ((ones >> q) & 1u) {
#pragma unroll
            for (int i = 0; i < V; ++i) r[(q * V + i) / 2] |= (y + 32u * i) << (16 * ((q * V + i) % 2));
          } else {
#pragma unroll
            for (int j = q * V; j < q * V + V; ++j) r[j / 2] |= atomicAdd(s_cnt + digit(k[j]), 1u) << (16 * (j % 2));
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) r[j / 2] |= atomicAdd(s_cnt + digit(k[j]), 1u) << (16 * (j % 2));
      }
    } else {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if ((valid >> j) & 1u) r[j / 2] |= atomicAdd(s_cnt + digit(k[j]), 1u) << (16 * (j % 2));
    }
    __syncthreads();
    uint32_t c = 0, at = 0;
    if (tid < bins) {
      c = s_cnt[tid];
      if (c) at = atomicAdd(cursor0 + (size_t)g * bins + tid, c);
      if (c == T) *s_one = 1;
    }
    const uint32_t excl = os::block_exclusive_scan<kScatterBlock>(c, s_warp);
    if (tid < bins) s_start[tid] = excl;
    __syncthreads();
    if (*s_one) {
      // One bin takes the whole tile (sorted keys): in their order, so that the
      // second pass finds sorted runs again and not this pass's shuffled ones.
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        uint4 v;
        K* e = reinterpret_cast<K*>(&v);
#pragma unroll
        for (int x = 0; x < V; ++x) e[x] = k[q * V + x];
        reinterpret_cast<uint4*>(s_keys)[q * kScatterBlock + tid] = v;
      }
    } else {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if (full || ((valid >> j) & 1u)) s_keys[s_start[digit(k[j])] + ((r[j / 2] >> (16 * (j % 2))) & 0xFFFFu)] = k[j];
    }
    const bool was_full = full;
    const uint32_t cnt = was_full ? T : (uint32_t)(min(tlo + (long long)T, (long long)g1) - max(tlo, (long long)g0));
    if (tid < bins) s_base[tid] = at - excl;  // (the reservation's round trip passes during the staging)
    // the next tile's keys are on their way while this one is written out
    if (tile + gridDim.x < tiles) load(tile + gridDim.x);
    __syncthreads();
    if (was_full) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const uint32_t i = (uint32_t)j * kScatterBlock + tid;
        const K key = s_keys[i];
        const uint32_t o = s_base[digit(key)] + i;
        if (o < n) out[o] = key;
      }
    } else {
      for (uint32_t i = tid; i < cnt; i += kScatterBlock) {
        const K key = s_keys[i];
        const uint32_t o = s_base[digit(key)] + i;
        if (o < n) out[o] = key;
      }
    }
    // no barrier here: the next tile's writes to s_cnt, s_start / s_base and
    // s_keys each come after a barrier that every thread reaches only past
    // its last read of them
  }
}

template <typename K, bool GROUPED>
__global__ void __launch_bounds__(kScatterBlock, kScatterPerSm) bucket_scatter_kernel(const K* in, K* out, size_t n, BucketArgs a) {
  __shared__ __align__(16) K s_keys[kScatterTile<K>];
  __shared__ uint32_t s_cnt[kGroups], s_start[kGroups], s_base[kGroups];
  __shared__ uint32_t s_warp[kScatterBlock / 32];
  __shared__ uint32_t s_one;
  __shared__ uint32_t s_first[kGroups + 1];
  chain_wait();
  chain_next();
  const BucketMap m = *a.map;
  if (!m.on) return;
  if constexpr (GROUPED) {
    for (uint32_t i = threadIdx.x; i <= (a.nb >> a.low_bits); i += kScatterBlock) s_first[i] = a.tile_first[i];
    __syncthreads();
  }
  if (m.plain)
    scatter_tiles<K, GROUPED, true>(in, out, (uint32_t)n, a, m, s_keys, s_cnt, s_start, s_base, s_warp, &s_one, s_first);
  else
    scatter_tiles<K, GROUPED, false>(in, out, (uint32_t)n, a, m, s_keys, s_cnt, s_start, s_base, s_warp, &s_one, s_first);
}

// ---------------------------------------------------------------------------
// Finish: sort each bucket.
// ---------------------------------------------------------------------------
// A bucket's keys are spread over kCells cells of equal width, about twenty
// cells per key, kept as a bitmap: one entry per 32 cells holds their bits and,
// once scanned, the number of keys before them.  A key's place is that number
// plus the set bits below its own: one atomic OR, one shared read, one popcount,
// no comparing.  The few keys that find their cell taken (about m^2 / (2 kCells)
// of m) are listed and counted beside the bits; they follow the entry's other
// keys, and the thread of the entry's first such key sorts the entry's few keys
// by comparing.  Buckets where that would be many (equal keys, clusters), and
// buckets larger than shared memory, are listed for a launch of their own.
//
// Bound by instruction issue and the shared-memory pipe together (about 60 %
// of each): 100M uniform 32-bit keys in 0.353 ms.  On the way there (same
// input): bins of one key on average and each key compared with its bin 0.80
// ms; the bitmap with 512 threads and a branch per key 0.59; 256 threads and
// more keys in flight 0.45; collisions listed instead of handled where they are
// found 0.41; no branch per key, and the next bucket's job left to one thread,
// 0.33.  Four CTAs per SM of 64 registers: five (48 registers) spill and lose
// more than they hide; 512 threads with the keys re-read from shared memory
// 0.41.  64-bit keys need 88 KB a CTA: two per SM.
template <typename K>
constexpr int kFinishPerSm = sizeof(K) == 4 ? 4 : 2;

// The least t with umulhi(t, mult) >= b (b < nb), from the rounded-down
// reciprocal inv = 2^63 / mult: the estimate is at most two short.
__device__ __forceinline__ uint32_t bucket_first_t(uint32_t b, uint32_t mult, unsigned long long inv) {
  uint32_t t = (uint32_t)__umul64hi((unsigned long long)b << 33, inv);
  while (__umulhi(t, mult) < b) ++t;
  return t;
}


// What thread 0 prepares of the next bucket while the CTA works on one.
enum : uint32_t {
  kJobSkip = 0,   // nothing to do
  kJobBulk = 1,   // cells, keys bulk-copied in
  kJobLoads = 2,  // cells, plain loads (a copy would reach past the array's ends)
  kJobLarge = 3   // more keys than shared memory holds
};
template <typename K>
struct FinishJob {
  K* src;         // its keys, sorted into dst; other: scratch of as many keys beside src (dst, unless in place)
  K* dst;
  K* other;
  K first;        // no key of the bucket is below it
  uint32_t cnt;
  uint32_t kind;
  uint32_t edge;  // 1: the bucket's range is not known (it holds keys outside the map): found here
  uint32_t cell_shift;  // cells of (key - first)
  uint32_t number;      // listed if the bucket is left to rare_buckets
  const K *lo, *hi;     // the array src lies in
};

// The shift that leaves at most `keep` bits of distances up to `range`.
template <typename K>
__device__ __forceinline__ uint32_t spread_of(K range, int keep) {
  const int bits = 8 * (int)sizeof(K) - (sizeof(K) == 4 ? __clz((int)(uint32_t)range) : __clzll((long long)range));
  return (uint32_t)max(0, bits - keep);
}

// Sorts buckets blockIdx.x, blockIdx.x + gridDim.x, ... below nb.  next(b, job)
// (thread 0) fills all of a bucket's job but its kind.  Buckets that this is not
// for are listed (rare[0]: how many, rare[1...]: which) and sorted by
// rare_buckets: their code here would cost the main path its registers (0.51 ms
// against 0.35 at 100M keys).
// RAW: float keys are read as they are stored, not in ordered form.
// COUNTS: for buckets that span at most kCountSpan values (keys that repeat, as
// floats of one octave do: 2^23 values): a 16-bit counter per value in place of
// the bitmap.  The atomic add gives a key's place among its equals, and the
// scanned counters its value's place: no key meets another.  100M 32-bit keys of
// 20 to 26 bits: 0.99 ms for the sort (by digits 1.48 to 1.66); 28 bits, whose
// bitmaps are full of keys that meet and left nearly all buckets to rare_buckets,
// 2.17 -> 1.04.  Sorted 64-bit keys, one value each: 0.223 -> 0.183 ms for this
// kernel at 33M; 32-bit 0.304 -> 0.321 at 100M.
template <typename K, bool FLT, int BLOCK = kFinishBlock, uint32_t CAP = kFinishCap, int CELL_BITS = kCellBits,
          bool RAW = false, bool COUNTS = false, typename Next>
__device__ __forceinline__ void finish_buckets(uint32_t nb, uint32_t* rare, uint32_t* err, Next&& next) {
  constexpr uint32_t B = BLOCK;
  constexpr int ITEMS = (int)CAP / BLOCK;
  constexpr uint32_t kEntries = 1u << (CELL_BITS - 5);
  constexpr uint32_t kHits = B;  // one listed key per thread
  constexpr size_t kAux = kEntries * 8;
  constexpr int C = 4;  // items handled together: their atomics in flight at once
  constexpr int W = B / 32;
  constexpr int U = (int)kEntries / (W * 64);  // 16-byte reads (two entries) per lane in the scan
  constexpr uint32_t V = 16 / sizeof(K);
  static_assert(U == 2 || U == 4, "runs of 64 entries per warp, scanned in pairs as 16-bit halves of one word");
  static_assert((CAP & (CAP - 1)) == 0 && ITEMS <= 16 && ITEMS % C == 0, "whole groups of items; places are masked");
  extern __shared__ __align__(128) unsigned char smem[];
  K* s_keys = reinterpret_cast<K*>(smem);                                           // [CAP + V]
  uint2* s_entry = reinterpret_cast<uint2*>(smem + (CAP + V) * sizeof(K));          // [kEntries]
  K* s_in = reinterpret_cast<K*>(smem + (CAP + V) * sizeof(K) + kAux);              // [CAP + 2 * V]
  K* s_hit = s_in + CAP + 2 * V;                                                    // [kHits]
  __shared__ FinishJob<K> s_job[2];
  __shared__ K s_edge[2 * W];
  __shared__ uint32_t s_warp[W];
  __shared__ uint32_t s_nhit, s_over;
  __shared__ __align__(8) uint64_t s_bar;
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  uint32_t cs = 0;
  auto entry_of = [&](K x) {  // (byte offset: the entry's number times 8)
    return reinterpret_cast<uint2*>(reinterpret_cast<char*>(s_entry) + ((uint32_t)(x >> (cs + 2)) & ((kEntries - 1) * 8)));
  };
  auto cell_of = [&](K x) { return (uint32_t)(x >> cs) & 31u; };
  // thread 0: bucket b's job, and its keys' bulk copy into s_in, from the
  // 16-byte boundary at or below the first key to the one at or above the end
  auto prepare = [&](uint32_t b, FinishJob<K>* job) {
    FinishJob<K> j;
    next(b, j);
    j.kind = j.cnt == 0 ? kJobSkip : kJobLarge;
    if (j.cnt != 0 && j.cnt <= CAP) {
      const uint32_t skew = skew_of(j.src);
      const uint32_t len = (skew + j.cnt + V - 1) / V * V;
      j.kind = kJobLoads;
      if (j.src - skew >= j.lo && j.src - skew + len <= j.hi) {
        j.kind = kJobBulk;
        fence_proxy_async();
        mbar_arrive_expect_tx(&s_bar, len * (uint32_t)sizeof(K));
        bulk_load_g2s(s_in, j.src - skew, len * (uint32_t)sizeof(K), &s_bar);
      }
    }
    *job = j;
  };
  if (tid == 0) {
    mbar_init(&s_bar, 1);
    mbar_fence_init();
    if (blockIdx.x < nb) prepare(blockIdx.x, &s_job[0]);
  }
  uint32_t parity = 0, slot = 0;
  for (uint32_t b = blockIdx.x; b < nb; b += gridDim.x, slot ^= 1u) {
    if (tid == 0) {
      s_nhit = 0;
      s_over = 0;
    }
    for (uint32_t q = tid; q < kEntries / 2; q += B) reinterpret_cast<uint4*>(s_entry)[q] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();  // the job is there; everything of the last bucket is done with
    const FinishJob<K>& job = s_job[slot];  // (read where needed: its pointers need no registers meanwhile)
    const uint32_t cnt = job.cnt;
    K first = 0;
    [[maybe_unused]] K edge_hi = 0;  // greatest key of a job of unknown range
    // thread 0, once s_in has been read: the next bucket
    auto go_on = [&]() {
      if (tid == 0 && b + gridDim.x < nb) prepare(b + gridDim.x, &s_job[slot ^ 1u]);
    };
    bool done = job.kind == kJobSkip;
    if (job.kind == kJobSkip || job.kind == kJobLarge) go_on();
    if (job.kind == kJobBulk || job.kind == kJobLoads) {
      const uint32_t skew_in = skew_of(job.src);
      const K* src = s_in + skew_in + tid;
      bool ok = true;
      if (job.kind == kJobBulk) {
        ok = mbar_wait_bounded(&s_bar, parity, err);
        parity ^= 1u;
      } else {
        for (uint32_t i = tid; i < cnt; i += B) s_in[skew_in + i] = job.src[i];  // (read by the same thread)
      }
      first = job.first;
      cs = job.cell_shift;
      if (job.edge) {  // the bucket's own range
        K lo = ~(K)0, hi = 0;
        for (uint32_t i = 0; i + tid < cnt; i += B) {
          const K x = to_ordered(src[i], RAW);
          lo = min(lo, x);
          hi = max(hi, x);
        }
        warp_minmax(lo, hi);
        if (lane == 0) {
          s_edge[warp] = lo;
          s_edge[W + warp] = hi;
        }
        __syncthreads();
#pragma unroll
        for (int w = 0; w < W; ++w) {
          lo = min(lo, s_edge[w]);
          hi = max(hi, s_edge[W + w]);
        }
        first = lo;
        edge_hi = hi;
        cs = spread_of<K>((K)(hi - lo), CELL_BITS);
      }
      // out of s_keys, where the keys lie with the destination's own offset from a
      // 16-byte boundary: whole 16-byte units in one bulk copy, the keys before
      // the first and after the last boundary singly
      auto write_out = [&](K* dst) {
        const uint32_t skew = skew_of(dst);
        K* stage = s_keys + skew;
        fence_proxy_async();
        __syncthreads();
        const uint32_t head = min(cnt, (V - skew) & (V - 1));
        const uint32_t body = (cnt - head) / V * V;
        if (tid == 0 && body) bulk_store_s2g(dst + head, stage + head, body * (uint32_t)sizeof(K));
        if (tid >= 32 && tid < 32 + V) {  // (V - 1 keys at most each)
          const uint32_t i = tid - 32;
          if (i < head) dst[i] = stage[i];
          if (head + body + i < cnt) dst[head + body + i] = stage[head + body + i];
        }
        done = true;
      };
      if constexpr (COUNTS) {
        uint32_t* s_half = reinterpret_cast<uint32_t*>(s_entry);
        constexpr uint32_t kWords = kEntries * 2;
        // (an end bucket's range is known only now, and to every thread)
        const bool wide = job.edge && (K)(edge_hi - first) > (K)(kCountSpan - 1);
        K k[ITEMS];
        uint32_t r[ITEMS / 2];
#pragma unroll
        for (int c = 0; c < ITEMS / 2; ++c) r[c] = 0;
#pragma unroll
        for (int c = 0; c < ITEMS; c += C) {
          if ((uint32_t)c * B >= cnt) break;
#pragma unroll
          for (int j = c; j < c + C; ++j) {
            const bool has = (uint32_t)j * B + tid < cnt;
            k[j] = to_ordered(src[(uint32_t)j * B], RAW) - first;
            const uint32_t sh = ((uint32_t)k[j] & 1u) * 16u;
            const uint32_t old = atomicAdd(s_half + ((uint32_t)(k[j] >> 1) & (kWords - 1)), has ? 1u << sh : 0u);
            r[j / 2] |= ((old >> sh) & 0xFFFFu) << (16 * (j % 2));
          }
        }
        if (!ok) s_over = 2;
        __syncthreads();
        if (s_over == 2) {  // (as below)
          mbar_wait_bounded(&s_bar, parity ^ 1u, err);
          if (tid == 0) bulk_store_wait_all();
          return;
        }
        go_on();
        if (!wide) {
          uint4 q[U];
          uint32_t c2[U];
          auto both = [](uint32_t w) { return (w & 0xFFFFu) + (w >> 16); };
#pragma unroll
          for (int u = 0; u < U; ++u) {
            q[u] = reinterpret_cast<uint4*>(s_half)[(warp * U + u) * 32 + lane];
            c2[u] = both(q[u].x) + both(q[u].y) + both(q[u].z) + both(q[u].w);
          }
          uint32_t p2[U / 2], t2[U / 2];
#pragma unroll
          for (int u = 0; u < U / 2; ++u) p2[u] = c2[2 * u] | (c2[2 * u + 1] << 16);
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
            for (int u = 0; u < U / 2; ++u) {
              const uint32_t x = __shfl_up_sync(kFull, p2[u], o);
              if (lane >= (uint32_t)o) p2[u] += x;
            }
          }
          uint32_t total = 0;
#pragma unroll
          for (int u = 0; u < U / 2; ++u) {
            t2[u] = __shfl_sync(kFull, p2[u], 31);
            total += (t2[u] & 0xFFFFu) + (t2[u] >> 16);
          }
          if (lane == 0) s_warp[warp] = total;
          // (the last bucket's copy out of s_keys must have read it)
          if (tid == 0) bulk_store_wait_read();
          __syncthreads();
          uint32_t before = __reduce_add_sync(kFull, lane < warp ? s_warp[lane & (W - 1)] : 0u);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            uint32_t run = before + (u & 1 ? p2[u / 2] >> 16 : p2[u / 2] & 0xFFFFu) - c2[u];
            before += u & 1 ? t2[u / 2] >> 16 : t2[u / 2] & 0xFFFFu;
            auto start = [&](uint32_t w) {
              const uint32_t at = run | ((run + (w & 0xFFFFu)) << 16);
              run += both(w);
              return at;
            };
            uint4 p;
            p.x = start(q[u].x);
            p.y = start(q[u].y);
            p.z = start(q[u].z);
            p.w = start(q[u].w);
            reinterpret_cast<uint4*>(s_half)[(warp * U + u) * 32 + lane] = p;
          }
          __syncthreads();
          K* stage = s_keys + skew_of(job.dst);
#pragma unroll
          for (int c = 0; c < ITEMS; c += C) {
            if ((uint32_t)c * B >= cnt) break;
#pragma unroll
            for (int j = c; j < c + C; ++j) {
              const uint32_t w = s_half[(uint32_t)(k[j] >> 1) & (kWords - 1)];
              const uint32_t p = ((w >> (((uint32_t)k[j] & 1u) * 16u)) & 0xFFFFu) + ((r[j / 2] >> (16 * (j % 2))) & 0xFFFFu);
              if ((uint32_t)j * B + tid < cnt) stage[p & (CAP - 1)] = from_ordered((K)(k[j] + first), FLT);
            }
          }
          write_out(job.dst);
        }
      } else {
        K k[ITEMS];  // distances from `first`; past the end, whatever s_in holds
        uint32_t hit = 0;   // bit j: key j found its cell taken
        uint32_t skip = 0;  // bit j: that, or there is no key j
#pragma unroll
        for (int c = 0; c < ITEMS; c += C) {
          if ((uint32_t)c * B >= cnt) break;
          uint32_t old[C];
          if ((uint32_t)(c + C) * B <= cnt) {
#pragma unroll
            for (int j = 0; j < C; ++j) {
              k[c + j] = to_ordered(src[(uint32_t)(c + j) * B], RAW) - first;
              old[j] = atomicOr(&entry_of(k[c + j])->x, 1u << cell_of(k[c + j]));
            }
          } else {
#pragma unroll
            for (int j = 0; j < C; ++j) {
              const bool has = (uint32_t)(c + j) * B + tid < cnt;
              k[c + j] = to_ordered(src[(uint32_t)(c + j) * B], RAW) - first;
              old[j] = atomicOr(&entry_of(k[c + j])->x, has ? 1u << cell_of(k[c + j]) : 0u);
              skip |= has ? 0u : 1u << (c + j);
            }
          }
#pragma unroll
          for (int j = 0; j < C; ++j) hit |= ((old[j] >> cell_of(k[c + j])) & 1u) << (c + j);
        }
        hit &= ~skip;
        skip |= hit;
        if (hit) {
          uint32_t p = atomicAdd(&s_nhit, (uint32_t)__popc(hit));
          for (uint32_t h = hit; h; h &= h - 1u, ++p)
            if (p < kHits) s_hit[p] = to_ordered(src[((uint32_t)__ffs((int)h) - 1u) * B], RAW) - first;
        }
        if (!ok) s_over = 2;
        __syncthreads();
        const uint32_t nhit = s_nhit;
        if (s_over == 2) {  // the copy never came: wait it out once more, sort nothing further
          mbar_wait_bounded(&s_bar, parity ^ 1u, err);
          if (tid == 0) bulk_store_wait_all();
          return;
        }
        go_on();
        bool crowded = nhit > kHits;
        K hx = 0;               // this thread's listed key
        uint32_t turn = 0;      // its number among its entry's listed keys
        uint32_t listed = 0, span = 0;  // how many those are; all of the entry's keys
        if (nhit && !crowded) {
          if (tid < nhit) {
            hx = s_hit[tid];
            turn = atomicAdd(&entry_of(hx)->y, 1u);
            if (turn >= kEntryHits) s_over = 1;
          }
          __syncthreads();
          crowded = s_over != 0;
        }
        if (!crowded) {
          // Scan: warp w owns kEntries / W entries, lane l entries 2 l and 2 l + 1
          // of each run of 64.  An entry's keys: its set bits and its listed keys.
          uint4 q[U];
          uint32_t c2[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            q[u] = reinterpret_cast<uint4*>(s_entry)[(warp * U + u) * 32 + lane];
            q[u].y += __popc(q[u].x);
            c2[u] = q[u].y + q[u].w + __popc(q[u].z);
          }
          if (tid < nhit) {
            const uint2 e = *entry_of(hx);
            listed = e.y;
            span = e.y + __popc(e.x);
          }
          uint32_t p2[U / 2], t2[U / 2];
#pragma unroll
          for (int u = 0; u < U / 2; ++u) p2[u] = c2[2 * u] | (c2[2 * u + 1] << 16);
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
            for (int u = 0; u < U / 2; ++u) {
              const uint32_t x = __shfl_up_sync(kFull, p2[u], o);
              if (lane >= (uint32_t)o) p2[u] += x;
            }
          }
          uint32_t total = 0;
#pragma unroll
          for (int u = 0; u < U / 2; ++u) {
            t2[u] = __shfl_sync(kFull, p2[u], 31);
            total += (t2[u] & 0xFFFFu) + (t2[u] >> 16);
          }
          if (lane == 0) s_warp[warp] = total;
          // (the last bucket's copy out of s_keys must have read it)
          if (tid == 0) bulk_store_wait_read();
          __syncthreads();
          uint32_t before = __reduce_add_sync(kFull, lane < warp ? s_warp[lane & (W - 1)] : 0u);
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const uint32_t run = before + (u & 1 ? p2[u / 2] >> 16 : p2[u / 2] & 0xFFFFu) - c2[u];
            before += u & 1 ? t2[u / 2] >> 16 : t2[u / 2] & 0xFFFFu;
            q[u].w = run + q[u].y;
            q[u].y = run;
            reinterpret_cast<uint4*>(s_entry)[(warp * U + u) * 32 + lane] = q[u];
          }
          __syncthreads();
          // staged with the destination's own offset from a 16-byte boundary
          K* dst = job.dst;
          const uint32_t skew = skew_of(dst);
          K* stage = s_keys + skew;
#pragma unroll
          for (int c = 0; c < ITEMS; c += C) {
            if ((uint32_t)c * B >= cnt) break;
#pragma unroll
            for (int j = c; j < c + C; ++j) {
              const uint2 e = *entry_of(k[j]);
              const uint32_t p = e.y + __popc(e.x & ((1u << cell_of(k[j])) - 1u));
              if (!((skip >> j) & 1u)) stage[p & (CAP - 1)] = from_ordered((K)(k[j] + first), FLT);
            }
          }
          if (nhit) {
            uint32_t lo = 0, bits = 0;
            if (tid < nhit) {
              const uint2 e = *entry_of(hx);
              lo = e.y;
              bits = e.x;
              if (listed > 1) stage[(lo + __popc(bits) + turn) & (CAP - 1)] = from_ordered((K)(hx + first), FLT);
            }
            __syncthreads();
            if (listed == 1) {  // between the key it met and the next: those above move up by one
              const uint32_t r = lo + __popc(bits & ((1u << cell_of(hx)) - 1u));
              const uint32_t top = min(CAP, lo + span) - 1u;
              for (uint32_t j = top; j > r + 1; --j) stage[j] = stage[j - 1];
              const K x = from_ordered((K)(hx + first), FLT), y = stage[r];
              const bool below = hx + first < to_ordered(y, FLT);
              stage[r] = below ? x : y;
              if (r < top) stage[r + 1] = below ? y : x;
            } else if (listed > 1 && turn == 0) {  // several: the entry's keys are sorted
              const uint32_t hi = min(CAP, lo + span);
              for (uint32_t j = lo + 1; j < hi; ++j) {
                const K x = stage[j];
                uint32_t p = j;
                while (p > lo) {
                  const K y = stage[p - 1];
                  if (to_ordered(y, FLT) <= to_ordered(x, FLT)) break;
                  stage[p] = y;
                  --p;
                }
                stage[p] = x;
              }
            }
          }
          write_out(dst);
        }
      }
    }
    if (!done) {
      if (tid == 0) rare[1 + atomicAdd(rare, 1u)] = job.number;
      // every thread has read s_nhit and s_over, which say which barriers it
      // takes part in, before thread 0 clears them (write_out has a barrier too;
      // counted buckets are listed without a look at either)
      if constexpr (!COUNTS) __syncthreads();
    }
  }
  if (tid == 0) bulk_store_wait_all();
}

// ---------------------------------------------------------------------------
// The listed buckets: equal keys, clusters, more keys than shared memory holds.
// ---------------------------------------------------------------------------
constexpr int kRareBlock = 512;
// Bin counters are padded by 4 words per 16, so that a thread's 16-byte reads
// of its own run of bins in the scan touch every bank once per quarter warp.
__device__ __forceinline__ uint32_t bin_at(uint32_t bin) { return bin + ((bin >> 4) << 2); }
constexpr uint32_t kBinWords = kBucketBins + kBucketBins / 4;
// bytes of the bins, or of the 4-bit passes' counters
constexpr size_t kRareAux = std::max<size_t>((size_t)(kBinWords + 4) * 4, (size_t)os::kNibbleBins * (kRareBlock + 32) * 4);

// The least and greatest of a[0, m) (in ordered form; raw: a holds floats as
// stored), in every thread.  s_ends: two words a warp.
template <typename K, int B>
__device__ __forceinline__ void block_minmax(const K* a, uint32_t m, bool raw, K* s_ends, K& lo, K& hi) {
  lo = ~(K)0;
  hi = 0;
  for (uint32_t i = threadIdx.x; i < m; i += B) {
    const K x = to_ordered(a[i], raw);
    lo = min(lo, x);
    hi = max(hi, x);
  }
  warp_minmax(lo, hi);
  if ((threadIdx.x & 31u) == 0) {
    s_ends[threadIdx.x >> 5] = lo;
    s_ends[B / 32 + (threadIdx.x >> 5)] = hi;
  }
  __syncthreads();
  for (int w = 0; w < B / 32; ++w) {
    lo = min(lo, s_ends[w]);
    hi = max(hi, s_ends[B / 32 + w]);
  }
}

// A bucket too large for shared memory, or with many keys in one bin: stable
// 8-bit LSD passes by the one CTA, a[0, m) and b[0, m) in turn; the result is
// left in `a` when `into_a`, else in `b`.  Slow (a few hundred cycles per 512
// keys and pass) and rare: the plan's sample bounds how large such a bucket
// is likely to be, and the bits all its keys share are skipped.
template <typename K>
__device__ void finish_slow(K* a, K* b, uint32_t m, bool into_a, unsigned char* smem) {
  constexpr int B = kRareBlock, W = B / 32;
  uint32_t* s_cur = reinterpret_cast<uint32_t*>(smem);                // [256]
  uint32_t* s_wc = s_cur + 256;                                       // [W][256]
  uint32_t* s_warp = s_wc + W * 256;                                  // [W]
  K* s_mm = reinterpret_cast<K*>(s_warp + W);                         // [2 * W]
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  K lo, hi;
  __syncthreads();
  block_minmax<K, B>(a, m, false, s_mm, lo, hi);
  const K diff = lo ^ hi;  // keys agree above its highest bit
  K *src = a, *dst = b;
  for (uint32_t sh = 0; sh < 8 * sizeof(K) && (diff >> sh) != 0; sh += 8) {
    __syncthreads();
    for (uint32_t i = tid; i < 256; i += B) s_cur[i] = 0;
    __syncthreads();
    for (uint32_t i = tid; i < m; i += B) atomicAdd(s_cur + ((uint32_t)(src[i] >> sh) & 255u), 1u);
    __syncthreads();
    const uint32_t c = tid < 256 ? s_cur[tid] : 0u;
    const uint32_t e = os::block_exclusive_scan<B>(c, s_warp);
    if (tid < 256) s_cur[tid] = e;
    for (uint32_t base = 0; base < m; base += B) {
      for (uint32_t i = tid; i < (uint32_t)W * 256; i += B) s_wc[i] = 0;
      __syncthreads();
      const uint32_t i = base + tid;
      const bool ok = i < m;
      const K x = ok ? src[i] : (K)0;
      const uint32_t d = ok ? (uint32_t)(x >> sh) & 255u : 256u;
      const uint32_t peers = __match_any_sync(kFull, d);
      const uint32_t below = __popc(peers & lanemask_lt());
      if (ok && below == 0) s_wc[warp * 256 + d] = __popc(peers);
      __syncthreads();
      if (tid < 256) {
        uint32_t run = s_cur[tid];
#pragma unroll
        for (int w = 0; w < W; ++w) {
          const uint32_t y = s_wc[w * 256 + tid];
          s_wc[w * 256 + tid] = run;
          run += y;
        }
        s_cur[tid] = run;
      }
      __syncthreads();
      if (ok) {
        const uint32_t o = s_wc[warp * 256 + d] + below;
        if (o < m) dst[o] = x;
      }
      __syncthreads();
    }
    K* sw = src;
    src = dst;
    dst = sw;
  }
  __syncthreads();  // (this CTA's global writes are visible to its own threads after a barrier)
  K* want = into_a ? a : b;
  if (src != want)
    for (uint32_t i = tid; i < m; i += B) want[i] = src[i];
  __syncthreads();
}

// A bucket of at most CAP keys that span fewer than kBucketBins values from
// `first` on: counted per value, and placed from each value's end down.
template <typename K>
__device__ void finish_counted(const K* in, K* out, uint32_t cnt, K first, unsigned char* smem, uint32_t* s_warp) {
  constexpr int B = kRareBlock;
  constexpr int PER = (int)kBucketBins / B;  // values per thread in the scan
  static_assert(PER % 4 == 0, "a thread's counters are read as 16-byte vectors");
  K* s_keys = reinterpret_cast<K*>(smem);
  uint32_t* s_bin = reinterpret_cast<uint32_t*>(smem + (size_t)kFinishCap * sizeof(K));
  const uint32_t tid = threadIdx.x;
  for (uint32_t i = tid * 4; i < kBinWords; i += B * 4)
    *reinterpret_cast<uint4*>(s_bin + i) = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  auto bin_of = [&](K key) { return min((uint32_t)(key - first), kBucketBins - 1); };
  for (uint32_t i = tid; i < cnt; i += B) atomicAdd(s_bin + bin_at(bin_of(in[i])), 1u);
  __syncthreads();
  uint32_t c[PER];
  uint32_t local = 0;
#pragma unroll
  for (int q = 0; q < PER / 4; ++q) {
    const uint4 x = *reinterpret_cast<const uint4*>(s_bin + bin_at(tid * PER) + 4 * q);
    c[4 * q] = x.x;
    c[4 * q + 1] = x.y;
    c[4 * q + 2] = x.z;
    c[4 * q + 3] = x.w;
  }
#pragma unroll
  for (int i = 0; i < PER; ++i) local += c[i];
  uint32_t run = os::block_exclusive_scan<B>(local, s_warp);
#pragma unroll
  for (int i = 0; i < PER; ++i) {  // the values' ends, counted down below
    run += c[i];
    c[i] = run;
  }
#pragma unroll
  for (int q = 0; q < PER / 4; ++q)
    *reinterpret_cast<uint4*>(s_bin + bin_at(tid * PER) + 4 * q) =
        make_uint4(c[4 * q], c[4 * q + 1], c[4 * q + 2], c[4 * q + 3]);
  __syncthreads();
  for (uint32_t i = tid; i < cnt; i += B) {
    const K key = in[i];
    s_keys[(atomicSub(s_bin + bin_at(bin_of(key)), 1u) - 1u) & (kFinishCap - 1)] = key;
  }
  __syncthreads();  // (every key of `in` has been read)
  for (uint32_t i = tid; i < cnt; i += B) out[i] = s_keys[i];
}

// A bucket of at most CAP keys, crowded (many keys equal or nearly so): stable
// 4-bit counting passes over the bits its keys differ in (diff: the least and
// greatest key's), in shared memory.
template <typename K, bool FLT, int B = kRareBlock, uint32_t CAP = kFinishCap, bool RAW = false>
__device__ void finish_nibbles(const K* in, K* out, uint32_t cnt, K diff, unsigned char* smem, uint32_t* s_warp) {
  constexpr int ITEMS = (int)CAP / B;
  K* s_keys = reinterpret_cast<K*>(smem);
  uint32_t* s_cnt = reinterpret_cast<uint32_t*>(smem + (size_t)CAP * sizeof(K));
  const uint32_t tid = threadIdx.x;
  for (uint32_t i = tid; i < CAP; i += B) s_keys[i] = i < cnt ? to_ordered(in[i], RAW) : ~(K)0;  // (padding sorts behind every key)
  __syncthreads();
  K k[ITEMS];
  uint32_t unused[1];
  for (uint32_t sh = 0; sh < 8 * sizeof(K) && (diff >> sh) != 0; sh += 4) {
    os::load_run<K, false, ITEMS>(k, unused, s_keys, nullptr);
    os::nibble_pass<K, false, B, ITEMS>(k, unused, sh, s_keys, nullptr, s_cnt, s_warp);  // ends with a barrier
  }
  for (uint32_t i = tid; i < cnt; i += B) out[i] = from_ordered(s_keys[i], FLT);
}

// job_of(b): bucket b's job.
template <typename K, typename JobOf>
__device__ __forceinline__ void rare_buckets(const uint32_t* rare, JobOf&& job_of) {
  constexpr int W = kRareBlock / 32;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint32_t s_warp[W];
  __shared__ K s_edge[2 * W];
  const uint32_t num = rare[0];
  for (uint32_t i = blockIdx.x; i < num; i += gridDim.x) {
    FinishJob<K> job{};
    job_of(rare[1 + i], job);
    if (job.cnt <= kFinishCap) {
      K lo, hi;
      block_minmax<K, kRareBlock>(job.src, job.cnt, false, s_edge, lo, hi);
      if (hi - lo < (K)kBucketBins)
        finish_counted<K>(job.src, job.dst, job.cnt, lo, smem, s_warp);
      else if (job.cnt <= kFinishCap / 2)  // (every pass takes the places there are, not the keys)
        finish_nibbles<K, false, kRareBlock, kFinishCap / 2>(job.src, job.dst, job.cnt, lo ^ hi, smem, s_warp);
      else
        finish_nibbles<K, false>(job.src, job.dst, job.cnt, lo ^ hi, smem, s_warp);
    } else {
      finish_slow<K>(job.src, job.other, job.cnt, job.src == job.dst, smem);
    }
    __syncthreads();
  }
}

template <typename K>
constexpr size_t rare_smem() {
  static_assert((256 + (kRareBlock / 32) * 257) * 4 + 2 * (kRareBlock / 32) * sizeof(K) <= kFinishCap * sizeof(K) + kRareAux,
                "finish_slow fits");
  return (size_t)kFinishCap * sizeof(K) + kRareAux;
}

// in == out: buckets are sorted in place and `other` is scratch; else in is
// the scratch array and other == out.
template <typename K>
__device__ __forceinline__ void plain_job(const BucketArgs& a, const BucketMap& m, uint32_t b, uint32_t at, uint32_t end,
                                          K* in, K* out, K* other, size_t n, FinishJob<K>& job) {
  job.src = in + at;
  job.dst = out + at;
  job.other = other + at;
  job.lo = in;
  job.hi = in + n;
  job.first = (K)m.lo + ((K)bucket_first_t(b, m.mult, m.inv) << m.s);
  job.cnt = (size_t)end <= n ? end - at : 0u;
  // the first and last bucket also hold the keys outside the map
  job.edge = b == 0 || b == a.nb - 1 ? 1u : 0u;
  job.cell_shift = m.cell_shift;
  job.number = b;
}

template <typename K>
__global__ void __launch_bounds__(kFinishBlock, kFinishPerSm<K>)
    bucket_finish_kernel(K* in, K* out, K* other, size_t n, BucketArgs a) {
  chain_wait();
  chain_next();
  const BucketMap m = *a.map;
  if (!m.on) return;
  // (thread 0) start[b] and start[b + 1] of the next bucket, read a bucket ahead
  uint32_t at = 0, end = 0;
  if (threadIdx.x == 0 && blockIdx.x < a.nb) {
    at = a.start[blockIdx.x];
    end = a.start[blockIdx.x + 1];
  }
  auto next = [&](uint32_t b, FinishJob<K>& job) {
    plain_job<K>(a, m, b, at, end, in, out, other, n, job);
    if (b + gridDim.x < a.nb) {
      at = a.start[b + gridDim.x];
      end = a.start[b + gridDim.x + 1];
    }
  };
  if (m.counts)
    finish_buckets<K, false, kFinishBlock, kFinishCap, kCellBits, false, true>(a.nb, a.rare, a.err, next);
  else
    finish_buckets<K, false>(a.nb, a.rare, a.err, next);
}

template <typename K>
__global__ void __launch_bounds__(kRareBlock) bucket_rare_kernel(K* in, K* out, K* other, size_t n, BucketArgs a) {
  chain_wait();
  const BucketMap m = *a.map;
  if (!m.on) return;
  rare_buckets<K>(a.rare, [&](uint32_t b, FinishJob<K>& job) {
    plain_job<K>(a, m, b, a.start[b], a.start[b + 1], in, out, other, n, job);
  });
}

template <typename K>
constexpr size_t finish_smem(int block = kFinishBlock, size_t cap = kFinishCap, int cell_bits = kCellBits) {
  return (2 * cap + (size_t)block + 3 * (16 / sizeof(K))) * sizeof(K) + ((size_t)8 << (cell_bits - 5));
}

// ---------------------------------------------------------------------------
// A few keys: the whole sort by one CTA.
// ---------------------------------------------------------------------------
// The array is one bucket of unknown range.  Latency only: about ten barriers
// and a dozen shared accesses per key, where eight (64-bit keys: sixteen) 4-bit
// passes take three barriers and about eight accesses each; those still sort
// keys that crowd, and payloads.  In a stream of them 4096 uniform 32-bit keys
// take 8 us against 27, 8192 8 us against 23; between events 4096 keys 13 us
// against 29 (Zipf, which crowds: 22 against 29), 64-bit 14 against 33.
template <typename K, bool FLT, int BLOCK, uint32_t CAP, int CELL_BITS>
__global__ void __launch_bounds__(BLOCK, 1) small_cells_kernel(K* keys, uint32_t n, uint32_t* err) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint32_t s_rare[2];
  __shared__ uint32_t s_warp[BLOCK / 32];
  __shared__ K s_ends[2 * BLOCK / 32];
  if (threadIdx.x == 0) s_rare[0] = 0;
  finish_buckets<K, FLT, BLOCK, CAP, CELL_BITS, FLT>(1, s_rare, err, [&](uint32_t, FinishJob<K>& job) {
    job.src = job.dst = job.other = keys;
    job.lo = keys;
    job.hi = keys + n;
    job.first = 0;
    job.cnt = n;
    job.edge = 1;
    job.cell_shift = 0;
    job.number = 0;
  });
  __syncthreads();
  if (s_rare[0]) {
    K lo, hi;
    block_minmax<K, BLOCK>(keys, n, FLT, s_ends, lo, hi);
    finish_nibbles<K, FLT, BLOCK, CAP, FLT>(keys, keys, n, lo ^ hi, smem, s_warp);
  }
}

template <typename K, bool FLT, int BLOCK, uint32_t CAP, int CELL_BITS>
cudaError_t small_cells_t(K* keys, size_t n, uint32_t* err, cudaStream_t stream) {
  constexpr size_t nibbles = (size_t)CAP * sizeof(K) + (size_t)os::kNibbleBins * (BLOCK + 32) * 4;
  const size_t smem = std::max(finish_smem<K>(BLOCK, CAP, CELL_BITS), nibbles);
  auto kern = small_cells_kernel<K, FLT, BLOCK, CAP, CELL_BITS>;
  cudaError_t e = ensure_dynamic_smem(kern, smem);
  if (e != cudaSuccess) return e;
  kern<<<1, BLOCK, smem, stream>>>(keys, (uint32_t)n, err);
  return cudaGetLastError();
}

// Fewer than 2048 keys leave most of 512 threads' items empty; 8192 need twice
// the cells for the same share of collisions.
template <typename K, bool FLT>
cudaError_t small_cells_k(K* keys, size_t n, uint32_t* err, cudaStream_t stream) {
  if (n <= 4096) return small_cells_t<K, FLT, 512, 4096, 16>(keys, n, err, stream);
  if constexpr (sizeof(K) == 4) return small_cells_t<K, FLT, 512, 8192, 17>(keys, n, err, stream);
  return cudaErrorInvalidValue;
}

template <typename K>
BucketArgs make_args(const BucketScratch& s, const K* tmp, size_t n, SortCtrl* ctrl, uint32_t* err) {
  BucketArgs a{};
  a.map = s.map;
  a.ctrl = ctrl;
  a.err = err;
  a.count = s.count;
  a.start = s.start;
  a.cursor = s.cursor;
  a.group_cursor = s.group_cursor;
  a.tile_first = s.tile_first;
  a.rare = s.rare;
  a.nb = s.nb;
  while ((1u << a.nb_bits) < s.nb) ++a.nb_bits;
  a.low_bits = s.low_bits;
  a.keys = n;
  a.tile = kScatterTile<K>;
  a.tmp_align = (uint32_t)(reinterpret_cast<uintptr_t>(tmp) & 15u);
  // sample keys a bucket may hold: one that would be full, with room for chance
  const double mean = (double)kSample / s.nb;
  const double cap = (double)kFinishCap * (double)kSample / (double)n;
  const double high = std::max(cap, mean + 6.0 * std::max(1.0, std::sqrt(mean)));
  a.hot_above = (uint32_t)high;
  a.max_sample = (uint32_t)(high + 4.0 + 2.0 * mean);
  return a;
}

// Least keys from which the buckets' crowding is looked at, at about 1 us a call
// (below, the launch for listed buckets is as fast as the digit passes).  Keys of
// which a tenth come 20 times each, by digit passes alone / left to that launch / turned
// away (us a call): 32-bit 2M 135 / 138 / 122, 4M 181 / 203 / 177; 100M multiples of 64
// 1803 / 2363 / 1848; 64-bit 1M 195 / 185 / 155, 5M 372 / 502 / 264; 67M of 2^20 prefixes
// 3010 / 6798 / 2090, of 2^24 values 1564 / 7430 / 1600.
template <typename K>
constexpr size_t kCrowdLeast = (size_t)1 << (sizeof(K) == 4 ? 21 : 20);

template <typename K>
BucketLimits make_limits(uint32_t nb, size_t n, const K* tmp) {
  BucketLimits m{};
  if (n >= kCrowdLeast<K>)
    m.crowd = reinterpret_cast<uint2*>((reinterpret_cast<uintptr_t>(tmp) + 15) & ~(uintptr_t)15);
  static_assert(kCrowdLeast<K> * sizeof(K) >= kCrowdBuckets * kCrowdEntries * sizeof(uint2) + 16, "fits the scratch array");
  m.dense_above = (uint32_t)((double)kFinishCap * (nb / kPlanParts) * (double)kSample / (double)n);
  // One CTA sorts such a bucket, at about 2 ns a key and byte; by then the count
  // has been paid for, a fifteenth of the digit passes: n / 1024 keys, 0.6 ms at
  // 100M, are still the shorter way, and where calls are short, 8192.
  m.most_keys = (uint32_t)std::max<size_t>(2 * kFinishCap, n / 1024);
  m.most_over = (uint32_t)(n / kOverShare);
  return m;
}

template <typename K>
cudaError_t plan_t(const BucketArgs& a, const BucketLimits& most, const K* keys, size_t n, cudaStream_t stream) {
  bucket_plan_kernel<K><<<kPlanCtas, kPlanBlock, 0, stream>>>(keys, n, a, most);
  return cudaGetLastError();
}

template <typename K>
cudaError_t count_t(const BucketArgs& a, const BucketLimits& most, const K* keys, size_t n, cudaStream_t stream) {
  auto kern = most.crowd ? bucket_count_kernel<K, true> : bucket_count_kernel<K, false>;
  const size_t smem = (size_t)std::max<uint32_t>(a.nb, 1024) * 4;
  cudaError_t e = ensure_dynamic_smem(kern, (size_t)kBucketsMax * 4);
  if (e != cudaSuccess) return e;
  const size_t work = ceil_div(n, (size_t)kCountBlock * (16 / sizeof(K)) * 2);
  const size_t grid = std::min<size_t>(std::max<size_t>(work, 1), (size_t)device_info().sm_count);
  return launch_chained(kern, (unsigned)grid, kCountBlock, smem, stream, keys, n, a, most);
}

template <typename K>
cudaError_t sort_t(const BucketArgs& a, K* keys, K* tmp, size_t n, cudaStream_t stream,
                   const std::function<cudaError_t()>& mark) {
  const unsigned sms = (unsigned)device_info().sm_count;
  auto m = [&]() { return mark ? mark() : cudaSuccess; };
  cudaError_t e = cudaSuccess;
  if ((e = m()) != cudaSuccess) return e;
  if ((e = m()) != cudaSuccess) return e;
  const size_t tiles = ceil_div(n, (size_t)kScatterTile<K>) + 1;
  e = launch_chained(bucket_scatter_kernel<K, false>, (unsigned)std::min<size_t>(tiles, sms * kScatterPerSm),
                     kScatterBlock, 0, stream, keys, tmp, n, a);
  if (e != cudaSuccess) return e;
  if ((e = m()) != cudaSuccess) return e;
  K* in = tmp;
  if (a.low_bits) {
    e = launch_chained(bucket_scatter_kernel<K, true>,
                       (unsigned)std::min<size_t>(tiles + kGroups, sms * kScatterPerSm), kScatterBlock, 0, stream, tmp, keys, n,
                       a);
    if (e != cudaSuccess) return e;
    in = keys;
  }
  if ((e = m()) != cudaSuccess) return e;
  auto kern = bucket_finish_kernel<K>;
  if ((e = ensure_dynamic_smem(kern, finish_smem<K>())) != cudaSuccess) return e;
  e = launch_chained(kern, std::min<unsigned>(a.nb, sms * kFinishPerSm<K>), kFinishBlock, finish_smem<K>(), stream, in, keys,
                     a.low_bits ? tmp : keys, n, a);
  if (e != cudaSuccess) return e;
  auto rare = bucket_rare_kernel<K>;
  if ((e = ensure_dynamic_smem(rare, rare_smem<K>())) != cudaSuccess) return e;
  e = launch_chained(rare, std::min<unsigned>(a.nb, sms * 2), kRareBlock, rare_smem<K>(), stream, in, keys,
                     a.low_bits ? tmp : keys, n, a);
  if (e != cudaSuccess) return e;
  return m();
}

// ---------------------------------------------------------------------------
// Many segments at once (the batched sort's plans, 32-bit keys).
// ---------------------------------------------------------------------------
// The same steps per segment: a map from a sample, counts, one partition pass
// (up to 2048 bins, so that every segment needs one only: a second pass would
// cross memory once more, while short runs cost the stores about a third of a
// pass), and all segments' buckets through the finish kernel.
using seg::BucketSeg;
using seg::PlanDev;
using seg::SegBucketJob;
using seg::SegBucketsDev;
using seg::SegMap;
using seg::SegTileJob;
using seg::kSegBinsLog2;
using seg::kSegTile;
constexpr uint32_t kSegBins = 1u << kSegBinsLog2;

__device__ __forceinline__ uint32_t seg_bucket(uint32_t key, uint32_t lo, uint32_t mult, uint32_t nb_bits) {
  return mult == 0 ? key >> (32u - nb_bits) : map_bucket(map_t<uint32_t>(key, lo, 0u), mult, (1u << nb_bits) - 1u);
}

// Crowding in a segment (as in bucket_count_kernel): where it is long enough to pay
// for it, half of the cells of one bucket, in the scratch array at the segment's
// own place; in shorter ones, by the sample's keys that share a cell.  (us a run by
// digit passes alone / left to the launch for listed buckets / declined, a tenth of a
// segment's keys 20 times each: 2000 of 20 K keys 854 / 1439 / 885, 300 of 100 K 573 / 1459 /
// 613, 30 of 1 M 585 / 1071 / 623; evenly spread 300 of 1 K to 1 M 376 -> 383, 1000 of 1 M
// 7.36 -> 7.40 ms, shorter ones 1 to 2 % more.  A bucket's cells for 100 K keys too: 4 %
// more for evenly spread ones.)
constexpr uint32_t kSegCrowdLeast = 1u << 17;
__device__ __forceinline__ uint2* seg_crowd(const PlanDev& P, const BucketSeg& g) {
  return reinterpret_cast<uint2*>((reinterpret_cast<uintptr_t>(P.tmp + g.base) + 7) & ~(uintptr_t)7);
}
constexpr int kSegCellLog2 = 11;  // slots for the sample's cells
// Whether its buckets are counted: they span at most ceil(2^32 / mult) values.
__device__ __forceinline__ bool seg_counted(const SegMap& m) { return ((1ull << 32) + m.mult - 1) / m.mult <= kCountSpan; }

// One CTA per segment of several buckets: the range a sample of 1024 keys spans.
constexpr int kSegPlanBlock = 256;
__global__ void __launch_bounds__(kSegPlanBlock) seg_map_kernel(const PlanDev P) {
  const uint32_t* __restrict__ keys = P.keys;
  const SegBucketsDev& sb = P.sb;
  __shared__ uint32_t s_lo[kSegPlanBlock / 32], s_hi[kSegPlanBlock / 32];
  __shared__ uint32_t s_cnt[kSegBins];
  __shared__ __align__(16) uint32_t s_cell[1u << kSegCellLog2];
  __shared__ uint32_t s_hits, s_most_hits, s_mult, s_shift, s_wide, s_off, s_most;
  const BucketSeg g = sb.seg[blockIdx.x];
  uint32_t lo = 0xFFFFFFFFu, hi = 0;
  uint32_t k[4];
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j) {
    const uint32_t i = j * kSegPlanBlock + threadIdx.x;
    k[j] = keys[g.base + sample_place(i, 10, g.len)];
    lo = min(lo, k[j]);
    hi = max(hi, k[j]);
  }
  for (uint32_t i = threadIdx.x; i < (1u << g.nb_bits); i += kSegPlanBlock) s_cnt[i] = 0;
  if (g.len < kSegCrowdLeast)
    for (uint32_t i = threadIdx.x; i < (1u << kSegCellLog2) / 4; i += kSegPlanBlock)
      reinterpret_cast<uint4*>(s_cell)[i] = make_uint4(kFull, kFull, kFull, kFull);
  if (threadIdx.x == 0) s_hits = 0;
  lo = __reduce_min_sync(kFull, lo);
  hi = __reduce_max_sync(kFull, hi);
  if ((threadIdx.x & 31u) == 0) {
    s_lo[threadIdx.x >> 5] = lo;
    s_hi[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  for (int w = 0; w < kSegPlanBlock / 32; ++w) {
    lo = min(lo, s_lo[w]);
    hi = max(hi, s_hi[w]);
  }
  uint32_t pad = (hi - lo) >> 7;  // (about eight keys of the sample's spacing)
  const uint32_t most_values = kCountSpan << g.nb_bits;  // (as in bucket_plan_kernel)
  if (hi - lo < most_values && hi - lo + 2 * pad >= most_values) pad = 0;
  lo -= min(lo, pad);
  hi += min(0xFFFFFFFFu - hi, pad);
  if (hi - lo >= 0xE0000000u) {
    lo = 0;
    hi = 0xFFFFFFFFu;
  }
  if (threadIdx.x < 32) {  // (the divisions, by one warp)
    const unsigned long long range = (unsigned long long)(hi - lo) + 1;
    const uint32_t mult = (uint32_t)min(0xFFFFFFFFull, ((unsigned long long)1 << (32 + g.nb_bits)) / range);
    const unsigned long long width = ((1ull << 32) + mult - 1) / mult, per = g.len >> g.nb_bits;
    uint32_t cell_shift = 0;
    while (((width - 1) >> cell_shift) >= kCells) ++cell_shift;
    // Keys of the sample in taken cells: what evenly spread ones have, and what they
    // have where buckets reach the finish kernel's limit.
    const float nb = (float)(1u << g.nb_bits), pairs = 1024.f * 1024.f / 2.f, len = (float)g.len;
    const float even = pairs / (nb * (float)(width >> cell_shift)), full = 2.f * kFinishBlock * pairs * nb / (len * len);
    if (threadIdx.x == 0) {
      s_mult = mult;
      s_shift = cell_shift;
      s_wide = width > kCountSpan ? 1u : 0u;
      // (few values a bucket, but too many to count: as in bucket_plan_kernel)
      s_off = width > kCountSpan && per * per > 400 * width ? 1u : 0u;
      s_most = 12u + (uint32_t)(((unsigned long long)(4 * kFinishCap) << 10) / g.len);
      s_most_hits = (uint32_t)fmaxf(even + 3.f * sqrtf(even) + 2.f, 0.8f * full);
    }
  }
  __syncthreads();
  const uint32_t mult = s_mult, cell_shift = s_shift, most = s_most;
  const bool cells = s_wide && g.len < kSegCrowdLeast;
  // The fullest bucket of the sample: a segment with one far beyond the finish
  // kernel is left to the digit passes before its keys are counted.
  uint32_t mx = 0, hits = 0;
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j) {
    const uint32_t t = map_t<uint32_t>(k[j], lo, 0u);
    const uint32_t c = atomicAdd(s_cnt + map_bucket(t, mult, (1u << g.nb_bits) - 1u), 1u) + 1u;
    mx = max(mx, c);
    if (!cells || c > most) continue;
    // (up to two keys a cell, so that a few frequent values, which crowd one bucket,
    // weigh little)
    constexpr uint32_t kOne = 1u << 30, kTwo = 1u << 31;
    const uint32_t cell = t >> cell_shift;
    uint32_t* slot = s_cell + ((cell * 0x9E3779B9u) >> (32 - kSegCellLog2));
    const uint32_t old = atomicCAS(slot, kFull, cell);
    if (old != kFull && (old & ~(kOne | kTwo)) == cell)
      hits += !(atomicOr(slot, kOne) & kOne) || !(atomicOr(slot, kTwo) & kTwo) ? 1u : 0u;
  }
  if (cells) {
    hits = __reduce_add_sync(kFull, hits);
    if (hits && (threadIdx.x & 31u) == 0) atomicAdd(&s_hits, hits);
  }
  const bool off = __syncthreads_or(mx > most || s_off) != 0 || s_hits > s_most_hits;
  if (!off && !cells && s_wide)
    for (uint32_t i = threadIdx.x; i < kCrowdEntries; i += kSegPlanBlock) seg_crowd(P, g)[i] = make_uint2(0u, 0u);
  if (threadIdx.x != 0) return;
  SegMap m{};
  m.off = off ? 1u : 0u;
  m.lo = lo;
  m.mult = mult;
  m.plain = lo == 0 && hi == 0xFFFFFFFFu ? 1u : 0u;
  m.inv = (1ull << 63) / mult;
  m.cell_shift = cell_shift;
  sb.map[blockIdx.x] = m;
}

// Counts per bucket: chunks of 64 K keys, dealt out round robin.
constexpr int kSegCountBlock = 512;
__global__ void __launch_bounds__(kSegCountBlock, 3) seg_count_kernel(const PlanDev P) {
  __shared__ uint32_t s_cnt[kSegBins];
  for (uint32_t c = blockIdx.x; c < P.sb.chunks; c += gridDim.x) {
    const seg::Item it = P.items[c];
    const uint32_t s = P.sb.of_large[it.seg];
    if (s == 0xFFFFFFFFu) continue;
    const BucketSeg g = P.sb.seg[s];
    const SegMap m = P.sb.map[s];
    if (m.off) continue;
    const uint32_t nb = 1u << g.nb_bits, mult = m.plain ? 0u : m.mult;
    for (uint32_t i = threadIdx.x; i < nb; i += kSegCountBlock) s_cnt[i] = 0;
    __syncthreads();
    const uint32_t lo = it.idx * seg::kHistChunk;
    const uint32_t len = min(seg::kHistChunk, g.len - lo);
    const uint32_t* src = P.keys + g.base + lo;
    const uint32_t head = min(len, (4u - skew_of(src)) & 3u);
    const uint32_t nvec = (len - head) / 4u, tail = head + nvec * 4u;
    const uint4* vec = reinterpret_cast<const uint4*>(src + head);
    const uint32_t pick = g.len < kSegCrowdLeast || seg_counted(m) ? 0xFFFFFFFFu : nb / 2;
    auto bucket = [&](uint32_t key) { return seg_bucket(key, m.lo, mult, g.nb_bits); };
    auto look = [&](uint32_t key, uint32_t b) {
      if (b == pick) crowd_add(seg_crowd(P, g), (key - m.lo) >> m.cell_shift, s);
    };
    auto add = [&](const uint4& q) {
      const uint32_t b0 = bucket(q.x), b1 = bucket(q.y), b2 = bucket(q.z), b3 = bucket(q.w);
      atomicAdd(s_cnt + b0, 1u);
      atomicAdd(s_cnt + b1, 1u);
      atomicAdd(s_cnt + b2, 1u);
      atomicAdd(s_cnt + b3, 1u);
      if (b0 == pick || b1 == pick || b2 == pick || b3 == pick) {
        look(q.x, b0);
        look(q.y, b1);
        look(q.z, b2);
        look(q.w, b3);
      }
    };
    constexpr uint32_t U = 4;
    uint32_t v = threadIdx.x;
    for (; v + (U - 1) * kSegCountBlock < nvec; v += U * kSegCountBlock) {
      uint4 q[U];
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) q[u] = ld_stream_v4(vec + v + u * kSegCountBlock);
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) add(q[u]);
    }
    for (; v < nvec; v += kSegCountBlock) add(ld_stream_v4(vec + v));
    if (threadIdx.x < head) atomicAdd(s_cnt + bucket(src[threadIdx.x]), 1u);
    if (threadIdx.x < len - tail) atomicAdd(s_cnt + bucket(src[tail + threadIdx.x]), 1u);
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < nb; i += kSegCountBlock)
      if (s_cnt[i]) atomicAdd(P.sb.count + g.first_bucket + i, s_cnt[i]);
    __syncthreads();
  }
}

// One CTA per large segment: its counts become cursors and jobs, or it is
// declined: no bucket map (longer than the bins allow), or too many of its keys
// in buckets beyond the finish kernel's shared memory.
constexpr int kSegScanBlock = 256;
__global__ void __launch_bounds__(kSegScanBlock) seg_jobs_kernel(const PlanDev P) {
  __shared__ uint32_t s_warp[kSegScanBlock / 32];
  __shared__ uint32_t s_over, s_hits, s_seen, s_first, s_chunk, s_job0, s_tile0;
  const uint32_t L = blockIdx.x, tid = threadIdx.x;
  const uint32_t s = P.sb.of_large[L];
  bool off = s == 0xFFFFFFFFu;
  if (!off) {
    const BucketSeg g = P.sb.seg[s];
    const SegMap m = P.sb.map[s];
    const uint32_t nb = 1u << g.nb_bits;
    uint32_t* cnt = P.sb.count + g.first_bucket;
    if (tid == 0) s_over = s_hits = s_seen = 0;
    __syncthreads();
    uint32_t over = 0;
    for (uint32_t i = tid; i < nb; i += kSegScanBlock) {
      const uint32_t c = cnt[i];
      if (c > kFinishCap) over += c > 4 * kFinishCap ? g.len : c;
    }
    if (over) atomicAdd(&s_over, min(over, g.len));
    const bool counted = seg_counted(m);
    bool crowded = false;
    if (!m.off && !counted && g.len >= kSegCrowdLeast) {
      uint32_t hits = 0, full = 0, seen = 0;
      for (uint32_t i = tid; i < kCrowdEntries; i += kSegScanBlock) {
        const uint2 e = seg_crowd(P, g)[i];
        hits += e.y - __popc(e.x);
        seen += e.y;
        full |= e.y - __popc(e.x) > kEntryHits ? 1u : 0u;
      }
      hits = __reduce_add_sync(kFull, hits);
      seen = __reduce_add_sync(kFull, seen);
      if ((tid & 31u) == 0) {
        atomicAdd(&s_hits, hits);
        atomicAdd(&s_seen, seen);
      }
      full = __syncthreads_or((int)full) != 0 ? 1u : 0u;
      crowded = crowd_listed(cnt[nb / 2], s_hits, full, s_seen);
    }
    __syncthreads();
    off = m.off || crowded || s_over > g.len / 32;
    if (!off) {
      // room for its jobs behind those of the segments before it
      const uint32_t tiles = (g.len + 3u + kSegTile - 1u) / kSegTile;
      if (tid == 0) {
        s_job0 = counted ? P.sb.buckets - nb - atomicAdd(&P.declined[seg::kJobCounted], nb)
                         : P.sb.whole + atomicAdd(&P.declined[seg::kJobBuckets], nb);
        s_tile0 = atomicAdd(&P.declined[seg::kJobTiles], tiles);
      }
      __syncthreads();
      const uint32_t job0 = s_job0, tile0 = s_tile0;
      const uint32_t per = (nb + kSegScanBlock - 1) / kSegScanBlock;
      uint32_t local = 0;
      for (uint32_t i = tid * per; i < min(nb, (tid + 1) * per); ++i) local += cnt[i];
      uint32_t run = os::block_exclusive_scan<kSegScanBlock>(local, s_warp);
      for (uint32_t i = tid * per; i < min(nb, (tid + 1) * per); ++i) {
        const uint32_t c = cnt[i];
        SegBucketJob j;
        j.at = g.base + run;
        j.cnt = c;
        j.first = m.plain ? i << (32u - g.nb_bits) : m.lo + bucket_first_t(i, m.mult, m.inv);
        j.in_keys = 0;
        j.edge = i == 0 || i == nb - 1 ? 1u : 0u;
        j.cell_shift = m.cell_shift;
        P.sb.bucket_job[job0 + i] = j;
        cnt[i] = run;
        run += c;
      }
      for (uint32_t t = tid; t < tiles; t += kSegScanBlock) {
        SegTileJob j;
        j.base = g.base;
        j.len = g.len;
        j.tile = t;
        j.first_bucket = g.first_bucket;
        j.nb_bits = g.nb_bits;
        j.lo = m.lo;
        j.mult = m.plain ? 0u : m.mult;
        P.sb.tile_job[tile0 + t] = j;
      }
    }
  }
  if (off) {
    const uint32_t chunks = P.large[L].hist_chunks;
    if (tid == 0) {
      s_chunk = atomicAdd(&P.declined[seg::kDeclinedChunks], chunks);
      P.declined[seg::kDeclinedHead + atomicAdd(&P.declined[seg::kDeclinedSegs], 1u)] = L;
      s_first = atomicAdd(&P.declined[seg::kDeclinedTiles], (P.large[L].len + seg::kPassTile - 1) / seg::kPassTile);
    }
    __syncthreads();
    const uint32_t tiles = (P.large[L].len + seg::kPassTile - 1) / seg::kPassTile;
    for (uint32_t t = tid; t < tiles; t += kSegScanBlock)
      P.declined_tile[s_first + t] = {P.large[L].base, P.large[L].len, L, s_first, {}};
    for (uint32_t c = tid; c < chunks; c += kSegScanBlock) P.declined_chunk[s_chunk + c] = make_uint2(L, c);
  }
}

// The partition pass (bucket_scatter_kernel's steps) with up to kSegBins bins.
// A tile's job is copied in a tile ahead, its keys while the tile before it is
// written out.
struct SegScatterSmem {
  uint32_t keys[kSegTile];
  uint32_t cnt[kSegBins], start[kSegBins], base[kSegBins];
  SegTileJob job[2];
  uint32_t warp[kScatterBlock / 32];
};

__global__ void __launch_bounds__(kScatterBlock, kScatterPerSm) seg_scatter_kernel(const PlanDev P) {
  constexpr int ITEMS = kScatterItems<uint32_t>;
  constexpr int Q = ITEMS / 4;
  constexpr int BPT = (int)kSegBins / kScatterBlock;  // bins per thread
  static_assert(BPT == 4, "a thread's bins are read as one 16-byte vector");
  static_assert(kScatterTile<uint32_t> == kSegTile, "one tile geometry");
  extern __shared__ __align__(16) unsigned char raw[];
  SegScatterSmem& sm = *reinterpret_cast<SegScatterSmem*>(raw);
  const uint32_t tid = threadIdx.x;
  const uint32_t tiles = P.declined[seg::kJobTiles];
  auto fetch_job = [&](uint32_t tile, uint32_t slot) {  // thread 0
    if (tile >= tiles) return;
    const char* src = reinterpret_cast<const char*>(P.sb.tile_job + tile);
#pragma unroll
    for (uint32_t i = 0; i < sizeof(SegTileJob); i += 16)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(&sm.job[slot]) + i), "l"(src + i) : "memory");
  };
  auto jobs_here = [&]() { asm volatile("cp.async.wait_all;" ::: "memory"); };
  uint32_t k[ITEMS];
  uint32_t valid = 0;
  long long tlo = 0;  // the tile's first place, counted from its segment's first key
  bool full = false;
  uint32_t nb_bits = 0, lo = 0, mult = 0, first_bucket = 0, seg_len = 0;
  unsigned long long seg_base = 0;
  auto load = [&](uint32_t slot) {
    const SegTileJob j = sm.job[slot];
    seg_base = j.base;
    seg_len = j.len;
    nb_bits = j.nb_bits;
    lo = j.lo;
    mult = j.mult;
    first_bucket = j.first_bucket;
    const uint32_t* in = P.keys + seg_base;
    tlo = (long long)j.tile * kSegTile - skew_of(in);
    full = tlo >= 0 && tlo + (long long)kSegTile <= (long long)seg_len;
    if (full) {
      const uint4* src = reinterpret_cast<const uint4*>(in + tlo) + tid;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const uint4 v = src[q * kScatterBlock];
        k[4 * q] = v.x;
        k[4 * q + 1] = v.y;
        k[4 * q + 2] = v.z;
        k[4 * q + 3] = v.w;
      }
    } else {
      valid = 0;
#pragma unroll
      for (int i = 0; i < ITEMS; ++i) {
        const long long x = tlo + (long long)i * kScatterBlock + tid;
        const bool ok = x >= 0 && x < (long long)seg_len;
        k[i] = ok ? in[x] : 0u;
        valid |= ok ? 1u << i : 0u;
      }
    }
  };
  uint32_t slot = 0;
  if (tid == 0) {
    fetch_job(blockIdx.x, 0);
    fetch_job(blockIdx.x + gridDim.x, 1);
    jobs_here();
  }
  __syncthreads();
  if (blockIdx.x < tiles) load(0);
  for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x, slot ^= 1u) {
    // (the next tile's job is in slot ^ 1; this tile's slot is read: the one after goes there)
    reinterpret_cast<uint4*>(sm.cnt)[tid] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    if (tid == 0) fetch_job(tile + 2 * gridDim.x, slot);
    const uint32_t bins = 1u << nb_bits;
    const uint32_t bits = nb_bits, at0 = first_bucket, l0 = lo, mu = mult, len = seg_len;
    uint32_t* out = P.tmp + seg_base;
    const bool was_full = full;
    // (a segment's last tile is empty when its first key's place in a 16-byte unit left no need for it)
    const uint32_t cnt = (uint32_t)max(0ll, min(tlo + (long long)kSegTile, (long long)len) - max(tlo, 0ll));
    auto digit = [&](uint32_t key) { return seg_bucket(key, l0, mu, bits); };
    uint32_t r[ITEMS / 2];
#pragma unroll
    for (int j = 0; j < ITEMS / 2; ++j) r[j] = 0;
    if (full) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) r[j / 2] |= atomicAdd(sm.cnt + digit(k[j]), 1u) << (16 * (j % 2));
    } else {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j)
        if ((valid >> j) & 1u) r[j / 2] |= atomicAdd(sm.cnt + digit(k[j]), 1u) << (16 * (j % 2));
    }
    __syncthreads();
    const uint4 c4 = reinterpret_cast<const uint4*>(sm.cnt)[tid];
    uint32_t at[BPT];
#pragma unroll
    for (int q = 0; q < BPT; ++q) {  // (consecutive threads, consecutive words)
      const uint32_t b = (uint32_t)q * kScatterBlock + tid;
      at[q] = 0;
      if (b < bins) {
        const uint32_t c = sm.cnt[b];
        if (c) at[q] = atomicAdd(P.sb.count + at0 + b, c);
      }
    }
    const uint32_t excl = os::block_exclusive_scan<kScatterBlock>(c4.x + c4.y + c4.z + c4.w, sm.warp);
    reinterpret_cast<uint4*>(sm.start)[tid] = make_uint4(excl, excl + c4.x, excl + c4.x + c4.y, excl + c4.x + c4.y + c4.z);
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j)
      if (was_full || ((valid >> j) & 1u))
        sm.keys[sm.start[digit(k[j])] + ((r[j / 2] >> (16 * (j % 2))) & 0xFFFFu)] = k[j];
#pragma unroll
    for (int q = 0; q < BPT; ++q) {
      const uint32_t b = (uint32_t)q * kScatterBlock + tid;
      if (b < bins) sm.base[b] = at[q] - sm.start[b];
    }
    if (tile + gridDim.x < tiles) load(slot ^ 1u);
    if (tid == 0) jobs_here();
    __syncthreads();
    if (was_full) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const uint32_t i = (uint32_t)j * kScatterBlock + tid;
        const uint32_t key = sm.keys[i];
        const uint32_t o = sm.base[digit(key)] + i;
        if (o < len) out[o] = key;
      }
    } else {
      for (uint32_t i = tid; i < cnt; i += kScatterBlock) {
        const uint32_t key = sm.keys[i];
        const uint32_t o = sm.base[digit(key)] + i;
        if (o < len) out[o] = key;
      }
    }
    // (no barrier: as in scatter_tiles)
  }
}

// Both arrays have `total` keys: a copy that stays inside one of them is safe.
__device__ __forceinline__ void seg_job(const PlanDev& P, size_t total, const SegBucketJob& j, FinishJob<uint32_t>& job) {
  job.src = (j.in_keys ? P.keys : P.tmp) + j.at;
  job.dst = P.keys + j.at;
  job.other = (j.in_keys ? P.tmp : P.keys) + j.at;
  job.lo = j.in_keys ? P.keys : P.tmp;
  job.hi = job.lo + total;
  job.first = j.first;
  job.cnt = j.cnt;
  job.edge = j.edge;
  job.cell_shift = j.cell_shift;
}

// Whole segments and buckets at the job array's front, then the counted ones at
// its end.
template <typename Make>
__device__ __forceinline__ void seg_finish(const PlanDev& P, Make&& make) {
  // (thread 0) the next bucket's job, read a bucket ahead
  const uint32_t jobs = P.sb.whole + P.declined[seg::kJobBuckets];
  SegBucketJob nj{};
  if (threadIdx.x == 0 && blockIdx.x < jobs) nj = P.sb.bucket_job[blockIdx.x];
  finish_buckets<uint32_t, false>(jobs, P.sb.rare, P.err, [&](uint32_t b, FinishJob<uint32_t>& job) {
    make(nj, job);
    job.number = b;
    if (b + gridDim.x < jobs) nj = P.sb.bucket_job[b + gridDim.x];
  });
  const uint32_t counted = P.declined[seg::kJobCounted], first = P.sb.buckets - counted;
  if (counted == 0) return;
  __syncthreads();
  if (threadIdx.x == 0 && blockIdx.x < counted) nj = P.sb.bucket_job[first + blockIdx.x];
  finish_buckets<uint32_t, false, kFinishBlock, kFinishCap, kCellBits, false, true>(
      counted, P.sb.rare, P.err, [&](uint32_t b, FinishJob<uint32_t>& job) {
        make(nj, job);
        job.number = first + b;
        if (b + gridDim.x < counted) nj = P.sb.bucket_job[first + b + gridDim.x];
      });
}

__global__ void __launch_bounds__(kFinishBlock, kFinishPerSm<uint32_t>) seg_finish_kernel(const PlanDev P, size_t total) {
  seg_finish(P, [&](const SegBucketJob& j, FinishJob<uint32_t>& job) { seg_job(P, total, j, job); });
}

__global__ void __launch_bounds__(kRareBlock) seg_rare_kernel(const PlanDev P, size_t total) {
  rare_buckets<uint32_t>(P.sb.rare, [&](uint32_t b, FinishJob<uint32_t>& job) {
    seg_job(P, total, P.sb.bucket_job[b], job);
  });
}

__global__ void clear_kernel(uint4* p, size_t words, uint32_t* tail, uint32_t tail_words, const uint32_t* off) {
  if (off && *off) return;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t i0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (size_t i = i0; i < words; i += stride) p[i] = make_uint4(0u, 0u, 0u, 0u);
  if (i0 < tail_words) tail[i0] = 0;
}

}  // namespace

cudaError_t launch_small_keys(void* keys, size_t n, int key_bytes, bool is_float, uint32_t* err, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  if (n > small_sort_max_keys(key_bytes, false)) return cudaErrorInvalidValue;
  if (key_bytes == 8) return small_cells_k<unsigned long long, false>(static_cast<unsigned long long*>(keys), n, err, stream);
  return is_float ? small_cells_k<uint32_t, true>(static_cast<uint32_t*>(keys), n, err, stream)
                  : small_cells_k<uint32_t, false>(static_cast<uint32_t*>(keys), n, err, stream);
}

cudaError_t launch_clear(void* p, size_t bytes, const uint32_t* off, cudaStream_t stream) {
  if (bytes % 4 || (reinterpret_cast<uintptr_t>(p) & 15u)) return cudaErrorInvalidValue;
  const size_t vec = bytes / 16;
  const unsigned grid = (unsigned)std::min(ceil_div(vec, (size_t)256 * 4) + 1, (size_t)device_info().sm_count * 4);
  clear_kernel<<<grid, 256, 0, stream>>>(static_cast<uint4*>(p), vec, reinterpret_cast<uint32_t*>(static_cast<uint4*>(p) + vec),
                                         (uint32_t)(bytes % 16 / 4), off);
  return cudaGetLastError();
}

// A synchronous call of n uniform keys, this sort against the LSD passes (us):
// 32-bit 8193 52 against 67, 100 K 50 against 69, 400 K 54 against 75, 2.2M 80
// against 112, 10M 144 against 233, 100M 918 against 1640; 64-bit 100 K 51 against
// 119, 1M 74 against 154, 10M 222 against 550.  Keys that the plan turns away pay
// for it, 12 to 18 us (32-bit Zipf keys: 100 K 83 against 67, 1M 104 against 84;
// constant ones 62 against 49), so every size beyond the one-CTA sort comes here.
// Above kBucketsMax * kBucketTarget keys a bucket would no longer fit the finish
// kernel with room for uneven filling.
bool bucket_sort_supported(size_t n, int key_bytes) {
  if (key_bytes != 4 && key_bytes != 8) return false;
  return n > small_sort_max_keys(key_bytes, false) && n <= kBucketMostKeys;
}

size_t bucket_scratch_layout(char* base, size_t n, BucketScratch* s) {
  uint32_t nb = 256;
  while (nb < kBucketsMax && n > (size_t)nb * kBucketTarget) nb *= 2;
  uint32_t lb = 0;
  while ((1u << lb) < nb) ++lb;
  s->nb = nb;
  s->low_bits = nb <= kGroups ? 0u : lb / 2;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    off = (off + 255) & ~(size_t)255;
    char* p = base + off;
    off += bytes;
    return p;
  };
  s->map = reinterpret_cast<BucketMap*>(take(sizeof(BucketMap)));
  s->count = reinterpret_cast<uint32_t*>(take((size_t)nb * 4));
  s->start = reinterpret_cast<uint32_t*>(take(((size_t)nb + 1) * 4));
  s->cursor = reinterpret_cast<uint32_t*>(take((size_t)nb * 4));
  s->group_cursor = reinterpret_cast<uint32_t*>(take(kGroups * 4));
  s->tile_first = reinterpret_cast<uint32_t*>(take((kGroups + 1) * 4));
  s->rare = reinterpret_cast<uint32_t*>(take(((size_t)nb + 1) * 4));
  return off;
}

namespace {

template <typename K>
cudaError_t plan_and_count(const BucketScratch& s, const void* keys, void* tmp, size_t n, SortCtrl* ctrl,
                           SortWords* words, cudaStream_t stream) {
  BucketArgs a = make_args(s, static_cast<const K*>(tmp), n, ctrl, nullptr);
  a.words = words;
  const BucketLimits most = make_limits(a.nb, n, static_cast<const K*>(tmp));
  const cudaError_t e = plan_t(a, most, static_cast<const K*>(keys), n, stream);
  return e != cudaSuccess ? e : count_t(a, most, static_cast<const K*>(keys), n, stream);
}

}  // namespace

cudaError_t enqueue_bucket_plan(const BucketScratch& s, const void* keys, void* tmp, size_t n, int key_bytes,
                                SortCtrl* ctrl, SortWords* words, cudaStream_t stream) {
  return key_bytes == 8 ? plan_and_count<unsigned long long>(s, keys, tmp, n, ctrl, words, stream)
                        : plan_and_count<uint32_t>(s, keys, tmp, n, ctrl, words, stream);
}

cudaError_t enqueue_bucket_sort(const BucketScratch& s, void* keys, void* tmp, size_t n, int key_bytes, SortCtrl* ctrl,
                                uint32_t* err, cudaStream_t stream, const std::function<cudaError_t()>& mark) {
  if (key_bytes == 8) {
    auto *k = static_cast<unsigned long long*>(keys), *t = static_cast<unsigned long long*>(tmp);
    return sort_t(make_args(s, t, n, ctrl, err), k, t, n, stream, mark);
  }
  auto *k = static_cast<uint32_t*>(keys), *t = static_cast<uint32_t*>(tmp);
  return sort_t(make_args(s, t, n, ctrl, err), k, t, n, stream, mark);
}

namespace seg {

cudaError_t launch_seg_plan(const PlanDev& pd, cudaStream_t s) {
  const unsigned sms = (unsigned)device_info().sm_count;
  cudaError_t e = cudaSuccess;
  if (pd.sb.num) {
    seg_map_kernel<<<pd.sb.num, kSegPlanBlock, 0, s>>>(pd);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    seg_count_kernel<<<std::min(pd.sb.chunks, sms * 3), kSegCountBlock, 0, s>>>(pd);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (pd.num_large) {
    seg_jobs_kernel<<<pd.num_large, kSegScanBlock, 0, s>>>(pd);
    e = cudaGetLastError();
  }
  return e;
}

cudaError_t launch_seg_buckets(const PlanDev& pd, size_t total_keys, cudaStream_t s) {
  const unsigned sms = (unsigned)device_info().sm_count;
  cudaError_t e = cudaSuccess;
  if (pd.sb.tiles) {
    if ((e = ensure_dynamic_smem(seg_scatter_kernel, sizeof(SegScatterSmem))) != cudaSuccess) return e;
    seg_scatter_kernel<<<std::min(pd.sb.tiles, sms * kScatterPerSm), kScatterBlock, sizeof(SegScatterSmem), s>>>(pd);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  if (pd.sb.buckets) {
    if ((e = ensure_dynamic_smem(seg_finish_kernel, finish_smem<uint32_t>())) != cudaSuccess) return e;
    seg_finish_kernel<<<std::min(pd.sb.buckets, sms * kFinishPerSm<uint32_t>), kFinishBlock, finish_smem<uint32_t>(), s>>>(
        pd, total_keys);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = ensure_dynamic_smem(seg_rare_kernel, rare_smem<uint32_t>())) != cudaSuccess) return e;
    seg_rare_kernel<<<std::min(pd.sb.buckets, sms * 4), kRareBlock, rare_smem<uint32_t>(), s>>>(pd, total_keys);
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace seg
}  // namespace pa
