// 64-bit LSD sorts by the keys' leading digits.
//
// An LSD sort of 64-bit keys runs eight passes, one per byte, though the top 32
// bits in which keys differ nearly always tell 100M keys apart: of n keys spread
// evenly about n^2 / 2^33 pairs agree in them and differ below.  So the passes of
// the four highest bytes in which keys differ are run alone (they are stable, so
// keys that agree in those bytes are left in input order), and what they leave
// undone is looked for and mended:
//   window_test_kernel    a random sample of up to 131072 keys: many pairs that agree in
//                         the window (the bytes from the lowest pass run on) and
//                         differ below mean that too much would be left, and all
//                         passes run;
//   window_mend_kernel    one read: where two neighbours agree in the window and are
//                         out of order, the run of keys that agree in it is put in
//                         order by one thread, up to kShortRun keys; longer runs are
//                         listed;
//   window_long_kernel    a long run per CTA: stable digit passes on the bytes
//                         below the window.
// Marks and lists lie in the look-back words of the passes left out.
// Equal keys are never out of order, so frequent values cost nothing.  Too long a
// run, or too many long ones, raise a flag the caller reads when the stream is
// done: the passes then all run over what is there, which keeps equal keys in
// their order.
//
// 100M 64-bit keys with payloads, eight passes -> four and the mending (us): 6008
// -> 3395 evenly spread (580K places; the mending 219), 5713 -> 3254 from 1M
// values, few of them frequent (no places: 190, of which 118 is the read at the
// measured copy rate); the test 24.  Listing the places in one kernel and mending
// them in the next was 561: a counter that 580K threads add to.
#include <algorithm>

#include "pa_common.cuh"
#include "pa_kernels.cuh"
#include "pa_onesweep_tile.cuh"

namespace pa {
namespace {

using K = unsigned long long;
constexpr uint32_t kFull = 0xFFFFFFFFu;
constexpr int kWindowPasses = 4;   // passes run (even: the result ends in the caller's array)
constexpr int kWindowLeast = 6;    // bytes in which keys must differ for it to pay
constexpr int kTestBlock = 1024;
constexpr uint32_t kTestMostLog2 = 17;  // keys of the sample, at most
constexpr uint32_t kShortRun = 32;
constexpr uint32_t kLongRun = 1u << 18;  // keys of a run one CTA is given, at most
constexpr int kLongBlock = 512;

// The sample (keys drawn at random) goes into a hash table by window, in the
// other key buffer; a key that meets another one of its window is compared with
// it.  The last CTA decides.
__global__ void __launch_bounds__(kTestBlock) window_test_kernel(const K* __restrict__ keys, size_t n, WindowScratch s,
                                                                 K* table, uint32_t slots_log2, uint32_t most_hits,
                                                                 SortCtrl* ctrl) {
  __shared__ uint32_t s_low, s_go, s_last;
  const uint32_t tid = threadIdx.x;
  if (tid == 0) {
    int run = 0, low = 0;
    for (int p = kMaxPasses - 1; p >= 0; --p)
      if (!ctrl->pass[p].skip && ++run == kWindowPasses) low = p;
    s_low = (uint32_t)low;
    s_go = run >= kWindowLeast ? 1u : 0u;
  }
  __syncthreads();
  if (!s_go) return;
  const uint32_t shift = 8u * s_low;
  const uint32_t slots = 1u << slots_log2;
  // (2^64 / golden ratio: the high bits of the product spread evenly)
  const unsigned long long g = ((unsigned long long)blockIdx.x * kTestBlock + tid + 1) * 0x9E3779B97F4A7C15ull;
  const K k = keys[(size_t)__umul64hi(g * g ^ (g >> 29), n)];
  bool bad = false;
  if (k != ~(K)0) {  // (the empty mark)
    const K w = k >> shift;
    uint32_t h = (uint32_t)((w * 0x9E3779B97F4A7C15ull) >> (64 - slots_log2));
    for (int probe = 0; probe < 64; ++probe, h = (h + 1) & (slots - 1)) {
      const K old = atomicCAS(table + h, ~(K)0, k);
      if (old == ~(K)0) break;
      if ((old >> shift) == w) {
        bad = old != k;
        break;
      }
    }
  }
  const int hits = __syncthreads_count(bad);
  if (tid == 0) {
    if (hits) atomicAdd(&s.state->hits, (uint32_t)hits);
    __threadfence();
    s_last = atomicAdd(&s.state->ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
    __threadfence();
  }
  __syncthreads();
  if (!s_last || *(volatile uint32_t*)&s.state->hits > most_hits) return;
  if (tid != 0) return;
  // the passes below the window are left out, and the others' buffers follow
  s.state->shift = shift;
  uint32_t in_tmp = 0;
  for (int p = 0; p < kMaxPasses; ++p) {
    PassCtrl& pc = ctrl->pass[p];
    if (p < (int)s_low) pc.skip = 1;
    pc.src_is_tmp = in_tmp;
    if (!pc.skip) in_tmp ^= 1u;
  }
  ctrl->final_in_tmp = in_tmp;
  ctrl->executed = kWindowPasses;
}

// First index in [0, n) whose window is at least w.
__device__ __forceinline__ size_t lower_bound(const K* keys, size_t n, uint32_t shift, K w) {
  size_t lo = 0, hi = n;
  while (lo < hi) {
    const size_t mid = lo + (hi - lo) / 2;
    if ((keys[mid] >> shift) < w) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Mends the run of keys of place i's window: nothing moves out of its run, so
// windows can be read while other threads mend their runs.
__device__ __noinline__ void mend_run(K* keys, uint32_t* vals, size_t n, size_t i, uint32_t shift, const WindowScratch& s) {
  const K w = keys[i] >> shift;
  size_t lo = i, hi = i + 2;
  while (lo > 0 && hi - lo <= kShortRun && (keys[lo - 1] >> shift) == w) --lo;
  while (hi < n && hi - lo <= kShortRun && (keys[hi] >> shift) == w) ++hi;
  if (hi - lo <= kShortRun) {
    // the thread that marks the run's first place mends it
    const uint32_t bit = 1u << (lo & 31u);
    if (atomicOr(s.claim + lo / 32, bit) & bit) return;
    for (size_t a = lo + 1; a < hi; ++a) {
      const K x = keys[a];
      const uint32_t v = vals ? vals[a] : 0u;
      size_t b = a;
      for (; b > lo && keys[b - 1] > x; --b) {
        keys[b] = keys[b - 1];
        if (vals) vals[b] = vals[b - 1];
      }
      if (b == a) continue;
      keys[b] = x;
      if (vals) vals[b] = v;
    }
    return;
  }
  const uint32_t first = (uint32_t)lower_bound(keys, n, shift, w);
  const uint32_t slots = 1u << s.slots_log2;
  uint32_t h = (first * 2654435761u) >> (32 - s.slots_log2);
  for (int probe = 0; probe < 256; ++probe, h = (h + 1) & (slots - 1)) {
    const uint32_t old = atomicCAS(s.set + h, 0u, first + 1);
    if (old == first + 1) return;
    if (old != 0) continue;
    const uint32_t x = atomicAdd(&s.state->runs, 1u);  // (at most one per slot)
    const size_t end = lower_bound(keys, n, shift, w + 1);
    s.run[2 * x] = first;
    s.run[2 * x + 1] = (uint32_t)end;
    if (end - first > kLongRun) s.state->fail = 1;
    return;
  }
  s.state->fail = 1;
}

// Finds places i with keys[i] and keys[i + 1] of one window and out of order, and
// mends them.  A warp reads kFindRows rows of 32 keys at a time: one read of the
// keys.  (A neighbour may be read in the middle of its run's mending; its run is
// marked by then.)
constexpr int kFindRows = 8;
__global__ void __launch_bounds__(256) window_mend_kernel(K* keys, uint32_t* vals, size_t n, WindowScratch s) {
  chain_wait();
  chain_next();
  const uint32_t shift = s.state->shift;
  if (shift == 0) return;
  const uint32_t lane = lane_id();
  const size_t stride = (size_t)gridDim.x * (256 / 32) * (kFindRows * 32);
  for (size_t i = ((size_t)blockIdx.x * (256 / 32) + (threadIdx.x >> 5)) * (kFindRows * 32); i < n; i += stride) {
    K k[kFindRows + 1];  // (past the end: never below; the last row is its first key alone)
#pragma unroll
    for (int j = 0; j <= kFindRows; ++j) {
      const size_t at = i + j * 32 + lane;
      k[j] = at < n && (j < kFindRows || lane == 0) ? keys[at] : ~(K)0;
    }
    uint32_t found = 0;
#pragma unroll
    for (int j = 0; j < kFindRows; ++j) {
      K next = __shfl_down_sync(kFull, k[j], 1);
      const K first = __shfl_sync(kFull, k[j + 1], 0);
      if (lane == 31) next = first;
      if (k[j] > next && (k[j] >> shift) == (next >> shift)) found |= 1u << j;
    }
    for (; found; found &= found - 1) mend_run(keys, vals, n, i + (__ffs(found) - 1) * 32 + lane, shift, s);
    __syncwarp();
  }
}

__global__ void __launch_bounds__(kLongBlock) window_long_kernel(K* keys, K* tkeys, uint32_t* vals, uint32_t* tvals,
                                                                  WindowScratch s) {
  constexpr int B = kLongBlock, W = B / 32;
  __shared__ uint32_t s_cur[256], s_wc[W * 256], s_warp[W];
  chain_wait();
  const uint32_t shift = s.state->shift;
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  if (shift == 0 || s.state->fail) {
    if (shift && blockIdx.x == 0 && tid == 0 && s.again) {
      __threadfence_system();
      *reinterpret_cast<volatile uint32_t*>(s.again) = kAgainAllDigits;
    }
    return;
  }
  const uint32_t runs = s.state->runs;
  for (uint32_t q = blockIdx.x; q < runs; q += gridDim.x) {
    const uint32_t at = s.run[2 * q], m = s.run[2 * q + 1] - at;
    K *src = keys + at, *dst = tkeys + at;
    uint32_t *vs = vals ? vals + at : nullptr, *vd = vals ? tvals + at : nullptr;
    for (uint32_t sh = 0; sh < shift; sh += 8) {
      __syncthreads();
      for (uint32_t i = tid; i < 256; i += B) s_cur[i] = 0;
      __syncthreads();
      for (uint32_t i = tid; i < m; i += B) atomicAdd(s_cur + ((uint32_t)(src[i] >> sh) & 255u), 1u);
      __syncthreads();
      const uint32_t c = tid < 256 ? s_cur[tid] : 0u;
      const bool one = __syncthreads_or(c == m) != 0;  // (every key has this byte)
      if (one) continue;
      const uint32_t e = os::block_exclusive_scan<B>(c, s_warp);
      if (tid < 256) s_cur[tid] = e;
      for (uint32_t base = 0; base < m; base += B) {
        for (uint32_t i = tid; i < (uint32_t)W * 256; i += B) s_wc[i] = 0;
        __syncthreads();
        const uint32_t i = base + tid;
        const bool ok = i < m;
        const K x = ok ? src[i] : 0;
        const uint32_t v = ok && vs ? vs[i] : 0u;
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
          if (o < m) {
            dst[o] = x;
            if (vs) vd[o] = v;
          }
        }
        __syncthreads();
      }
      K* sw = src;
      src = dst;
      dst = sw;
      uint32_t* vw = vs;
      vs = vd;
      vd = vw;
    }
    __syncthreads();
    if (src != keys + at)
      for (uint32_t i = tid; i < m; i += B) {
        keys[at + i] = src[i];
        if (vals) vals[at + i] = vs[i];
      }
    __syncthreads();
  }
}

}  // namespace

bool window_sort_supported(size_t n, int key_bytes) {
  return key_bytes == 8 && n >= kWindowLeastKeys && n < ((size_t)3 << 28);
}

WindowScratch window_scratch(size_t n, char* skipped, size_t skipped_bytes, WindowState* state) {
  WindowScratch s;
  uint32_t lg = 0;
  while (((size_t)2 << lg) <= n / 256) ++lg;
  const size_t claim_bytes = (n / 32 + 1) * 4;
  if (claim_bytes + ((size_t)12 << lg) > skipped_bytes) return s;
  s.slots_log2 = lg;
  s.state = state;
  s.claim = reinterpret_cast<uint32_t*>(skipped);
  s.set = s.claim + claim_bytes / 4;
  s.run = s.set + ((size_t)1 << lg);
  return s;
}

cudaError_t enqueue_window_test(const WindowScratch& s, const void* keys, void* tmp, size_t n, SortCtrl* ctrl,
                                cudaStream_t stream) {
  // A share p of all pairs agreeing in the window and no further makes sample^2
  // p / 2 hits.  The window is used up to p = 1 / (2 n), where places out of order
  // are a fair part of all keys and a run of sqrt(n / 2) keys would explain them
  // (128 hits at 2^19, 64 at 2^20, 42 at 100M, where evenly spread keys have 2).
  uint32_t lg = 12;
  while (lg < kTestMostLog2 && ((size_t)1 << (2 * lg)) < 256 * n) ++lg;
  const size_t sample = (size_t)1 << lg;
  const uint32_t most_hits = (uint32_t)(((sample * sample) >> 2) / n);
  cudaError_t e = cudaMemsetAsync(tmp, 0xFF, 2 * sample * sizeof(K), stream);
  if (e != cudaSuccess) return e;
  window_test_kernel<<<(unsigned)(sample / kTestBlock), kTestBlock, 0, stream>>>(static_cast<const K*>(keys), n, s,
                                                                               static_cast<K*>(tmp), lg + 1, most_hits, ctrl);
  return cudaGetLastError();
}

cudaError_t enqueue_window_mend(const WindowScratch& s, void* keys, void* tmp, uint32_t* vals, uint32_t* tvals, size_t n,
                                cudaStream_t stream) {
  const unsigned sms = (unsigned)device_info().sm_count;
  K* k = static_cast<K*>(keys);
  const cudaError_t e = launch_chained(
      window_mend_kernel, (unsigned)std::min(ceil_div(n, (size_t)256 * kFindRows), (size_t)sms * 8), 256, 0, stream, k, vals, n, s);
  if (e != cudaSuccess) return e;
  return launch_chained(window_long_kernel, sms, kLongBlock, 0, stream, k, static_cast<K*>(tmp), vals, tvals, s);
}

}  // namespace pa
