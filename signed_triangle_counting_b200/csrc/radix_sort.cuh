// Stable LSD radix sort of 64-bit keys over a bit window [lo, hi), plus the
// range-partitioned scans the graph build and the sharded count use.  The
// kernels have internal linkage: every translation unit that includes this
// header gets its own copy.
//
// Design (B200), after the published one-sweep method (Adinets and Merrill,
// "Onesweep: A Faster Least Significant Digit Radix Sort for GPUs", 2022):
//   histogram  one read of the keys counts the digits of every pass; the last
//              CTA to finish scans the counts into each digit's first output
//   pass       one kernel per 8-bit digit: a CTA takes the next tile, ranks
//              its keys by digit (warp multi-split, stable), reorders them in
//              shared memory, adds up the counts of the tiles before it by
//              looking back over their published states, and writes each
//              digit's keys in a row (reads 8 B/key, writes 8 B/key).
// A CTA waits only for tiles taken before its own, whose CTAs are already
// running; the wait is bounded all the same.  A wait that expires ends the
// sort and leaves the output undefined: the kernels after it see the error
// word (device_failed) and touch nothing, or the host reads it first.
// Bits of the key outside [lo, hi) ride along untouched, which is how the
// edge sign travels in bit 63 without a separate payload array.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "internal.h"
#include "stc_device.cuh"

namespace stc {

constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSortTile = 4096;  // granularity of range partitions
constexpr int kRadix = 256;
static_assert(kSortThreads == kRadix, "thread d of a pass owns digit d");
constexpr int kMaxSortGrid = kSMs * 4;
constexpr int kMaxPasses = 8;
constexpr int kHistItems = 8;  // keys in flight per thread of the histogram

struct RangePartition {
  uint32_t grid;     // CTAs
  uint64_t per_cta;  // keys per CTA, a multiple of the tile
};

inline RangePartition range_partition(uint64_t m, uint64_t tile, uint32_t max_grid) {
  uint64_t tiles = (m + tile - 1) / tile;
  if (tiles == 0) tiles = 1;
  uint64_t grid = tiles < max_grid ? tiles : max_grid;
  uint64_t per = (tiles + grid - 1) / grid;
  grid = (tiles + per - 1) / per;
  return RangePartition{(uint32_t)grid, per * tile};
}

// Workspace of one sort, in 32-bit words: the digit counts of every pass
// (scanned in place), one tile ticket per pass, the histogram's CTA count and
// the abort flag, then two arrays of tile states (a pass clears the one the
// next pass uses).
constexpr uint32_t kSortTickets = kMaxPasses * kRadix;
constexpr uint32_t kSortDone = kSortTickets + kMaxPasses;
constexpr uint32_t kSortAbort = kSortDone + 1;
constexpr uint32_t kSortStates = kSortTickets + 2 * kMaxPasses;
// Set in the tickets of an aborted sort: every tile taken from then on lies past
// the keys, so no CTA of this or a later pass starts (reading the abort flag
// beside the ticket instead cost the skewed workload 17.27 -> 17.45 ms).
constexpr uint32_t kSortClosed = 1u << 31;

// Keys per thread of a pass: 16 once the tiles fill the GPU; smaller sorts
// take smaller tiles, which spreads them over more SMs and shortens each
// CTA's serial part (a pass over 100,000 keys takes 12 us, over 1,000,000
// 19 us, over 2,400,000 32 us).
constexpr uint64_t kSortMax4 = (uint64_t)kSMs * 4 * kSortThreads * 4;  // the largest sort of 4,
constexpr uint64_t kSortMax8 = (uint64_t)kSMs * 8 * kSortThreads * 8;  // and of 8 keys a thread
inline int sort_items(uint64_t m) { return m > kSortMax8 ? 16 : m > kSortMax4 ? 8 : 4; }
inline uint64_t sort_tiles(uint64_t m) {
  const uint64_t tile = (uint64_t)kSortThreads * sort_items(m);
  return (m + tile - 1) / tile;
}
// A tile state holds a count of keys and two flag bits: 32 bits a word while
// counts stay below 2^30, else 64.
inline bool sort_wide(uint64_t m) { return m >= (1ull << 30); }
// What a sort of m keys clears and publishes.
inline size_t sort_words(uint64_t m) {
  return kSortStates + 2 * (size_t)kRadix * sort_tiles(m) * (sort_wide(m) ? 2 : 1);
}
// The workspace of a sort of m keys or of any fewer: one key past a limit
// above halves the tiles, so the largest sorts of the smaller tiles count too.
inline size_t sort_workspace_words(uint64_t m) {
  return std::max({sort_words(m), sort_words(std::min(m, kSortMax4)),
                   sort_words(std::min(m, kSortMax8))});
}
struct SortSpace {
  uint32_t* words = nullptr;
  size_t count = 0;
};
// The context's workspace for sorts of at most m keys (and at least `words`).
inline SortSpace sort_space(stc_ctx* c, uint64_t m, size_t words = 0) {
  const size_t n = std::max(words, sort_workspace_words(m));
  return SortSpace{buffer<uint32_t>(c, B_SORT_WS, n), n};
}

// Digit counts of every pass over [lo, hi) into ws[pass][digit]; the last CTA
// turns them into exclusive prefixes.
static __global__ void __launch_bounds__(kSortThreads) k_radix_hist(
    const uint64_t* __restrict__ keys, uint64_t m, int lo, int hi, uint32_t* __restrict__ ws,
    const unsigned long long* __restrict__ m_dev) {
  __shared__ uint32_t hist[kMaxPasses][kRadix];
  __shared__ uint32_t scan_tmp[kSortWarps + 1];
  __shared__ bool s_last;
  const unsigned tid = threadIdx.x, lane = lane_id();
  if (m_dev && *m_dev < m) m = *m_dev;
  const int passes = (hi - lo + 7) / 8;
  for (int i = tid; i < passes * kRadix; i += kSortThreads) (&hist[0][0])[i] = 0;
  __syncthreads();
  const uint64_t step = (uint64_t)gridDim.x * kSortThreads * kHistItems;
  for (uint64_t base = ((uint64_t)blockIdx.x * kSortThreads + (tid & ~31u)) * kHistItems; base < m;
       base += step) {
    uint64_t k[kHistItems];
#pragma unroll
    for (int j = 0; j < kHistItems; j++) {
      const uint64_t i = base + j * 32 + lane;
      k[j] = i < m ? __ldcs(keys + i) : ~0ull;
    }
    for (int p = 0; p < passes; p++) {
      const int shift = lo + 8 * p;
      const uint32_t dmask = hi - shift < 8 ? (1u << (hi - shift)) - 1 : 255u;
#pragma unroll
      for (int j = 0; j < kHistItems; j++)
        if (base + j * 32 + lane < m) atomicAdd(&hist[p][(uint32_t)(k[j] >> shift) & dmask], 1u);
    }
  }
  __syncthreads();
  for (int i = tid; i < passes * kRadix; i += kSortThreads) {
    const uint32_t c = (&hist[0][0])[i];
    if (c) atomicAdd(ws + i, c);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(ws + kSortDone, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  for (int p = 0; p < passes; p++) {
    uint32_t total;
    const uint32_t c = __ldcg(ws + p * kRadix + tid);
    ws[p * kRadix + tid] = block_exclusive_scan<kSortThreads>(c, scan_tmp, total);
  }
}

// Tile states: flag bits above the count.
template <class W>
struct TileState {
  static constexpr int kShift = sizeof(W) * 8 - 2;
  static constexpr W kCount = (W(1) << kShift) - 1;
  static constexpr W kLocal = W(1) << kShift;    // the tile's own count
  static constexpr W kPrefix = W(2) << kShift;   // with all tiles before it
  __device__ static void put(W* p, W v) { *(volatile W*)p = v; }
  __device__ static W get(const W* p) { return *(const volatile W*)p; }
};
constexpr uint32_t kLookbackPolls = 1u << 22;  // bound of one wait, a few seconds

// Thread d of tile `tile`: the count of digit d in all tiles before it (its
// own state at `own`, holding its count `cnt`, becomes the sum), four
// predecessors' states in flight at a time.  A wait that expires raises the
// abort flag.
template <class W>
__device__ __forceinline__ W look_back(W* own, uint32_t tile, uint32_t cnt, uint32_t* ws,
                                       uint32_t& abort) {
  using TS = TileState<W>;
  W before = 0;
  if (tile == 0) return before;
  const W* p = own - kRadix;
  uint32_t left = tile, polls = 0;  // predecessors not yet added
  bool done = false;
  while (!done) {
    W s[4];
#pragma unroll
    for (int q = 0; q < 4; q++) s[q] = (uint32_t)q < left ? TS::get(p - (size_t)q * kRadix) : 0;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (done || s[q] == 0) break;
      before += s[q] & TS::kCount;
      done = (s[q] & TS::kPrefix) != 0;
      p -= kRadix;
      left--;
    }
    if (!done && ++polls > kLookbackPolls) {
      ((volatile uint32_t*)ws)[kSortAbort] = 1;
      done = true;
    }
    if (!done && (polls & 1023u) == 0 && ((volatile uint32_t*)ws)[kSortAbort]) done = true;
  }
  if (polls >= 1023u && ((volatile uint32_t*)ws)[kSortAbort]) abort = 1;
  TS::put(own, TS::kPrefix | (before + cnt));
  return before;
}

// The digit (key >> shift) & dmask; kHigh: it lies in the upper word.
template <bool kHigh>
__device__ __forceinline__ uint32_t key_digit(uint64_t key, int shift, uint32_t dmask) {
  const uint32_t lo = (uint32_t)key, hi = (uint32_t)(key >> 32);
  return (kHigh ? hi >> (shift & 31) : __funnelshift_r(lo, hi, shift)) & dmask;
}

template <int ITEMS>
struct PassSmem {
  union {
    uint64_t keys[kSortThreads * ITEMS];       // the tile, by digit
    uint32_t mask[2][kSortWarps][kRadix];      // lanes by digit, two keys in turn
  };
  uint32_t whist[kSortWarps][kRadix];
  uint32_t gofs[kRadix];
  uint32_t scan_tmp[kSortWarps + 1];
  uint32_t tile, abort;
};

// Stable ranks of the warp's keys among its keys of the digit, 16 bits each,
// and the digits' counts in `whist`.  Per key, the lanes that share a digit
// find each other by or-ing their bit into the digit's word of a table (an
// 8-ballot match took 32 integer instructions a key and made the integer
// pipe the pass's limit: 0.70 against 0.57 ms a pass over 100 M keys); the
// lowest of them adds their number to the count, clears the word and hands
// the old count to the others.  Two tables in turn: a table's next use comes
// after the barriers of the other's.
template <int ITEMS, bool kHigh, bool kFullTile>
__device__ __forceinline__ void rank_keys(const uint64_t (&k)[ITEMS], uint32_t wbase,
                                          uint32_t valid, int shift, uint32_t dmask,
                                          uint32_t (*mask)[kSortWarps][kRadix], uint32_t* whist,
                                          uint32_t (&r)[ITEMS / 2]) {
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5, lt = lanemask_lt();
#pragma unroll
  for (int j0 = 0; j0 < ITEMS; j0 += 2) {
    unsigned peers[2];
    uint32_t old[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      uint32_t dg = key_digit<kHigh>(k[j0 + q], shift, dmask);
      if (!kFullTile && wbase + 32 * (j0 + q) >= valid) dg = kRadix - 1;
      uint32_t* word = &mask[q][warp][dg];
      atomicOr(word, 1u << lane);
      __syncwarp();
      peers[q] = *word;
      __syncwarp();
      old[q] = 0;
      if ((peers[q] & lt) == 0) {
        *word = 0;
        old[q] = atomicAdd(whist + dg, (uint32_t)__popc(peers[q]));
      }
    }
    uint32_t x[2];
#pragma unroll
    for (int q = 0; q < 2; q++)
      x[q] = __shfl_sync(kFull, old[q], __ffs(peers[q]) - 1) + __popc(peers[q] & lt);
    r[j0 / 2] = x[0] | (x[1] << 16);
  }
}

// One pass: stable by the digit, one tile per CTA.  Bound by the shared-
// memory pipe, not by DRAM: over the 67 M arc keys of RMAT scale 22, 367 us for
// an evenly spread digit (83% busy, 32 wavefronts per warp and key for the
// match, the counts and the exchange; 2.9 TB/s of DRAM) and 534 us for a skewed
// one (90% busy, 59 wavefronts, lanes or-ing into one word).
// The version before (a count pass over the keys, a one-CTA scan of 256
// counts per CTA, then this) took 2.0 ms a pass over 268 M keys, this 1.5 with
// its share of the histogram; over 2.4 M keys 78 us (58 of them the scan),
// this 31.  Tiles of several pieces with the counts taken first, to look back
// less often, were slower (1.9 ms), as were warp matches by ballots (1.8) or
// match.any (2.6).
template <int ITEMS, class W, bool kHigh>
static __global__ void __launch_bounds__(kSortThreads, 4) k_radix_pass(
    const uint64_t* __restrict__ in, uint64_t* __restrict__ out, uint64_t m, int shift,
    uint32_t dmask, uint32_t* __restrict__ ws, int pass, W* __restrict__ state,
    W* __restrict__ next_state, const unsigned long long* __restrict__ m_dev,
    unsigned long long* __restrict__ err) {
  constexpr uint32_t kTile = kSortThreads * ITEMS;
  using TS = TileState<W>;
  __shared__ PassSmem<ITEMS> sm;
  const unsigned tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  if (m_dev && *m_dev < m) m = *m_dev;
  if (tid == 0) {
    sm.tile = atomicAdd(ws + kSortTickets + pass, 1u);
    sm.abort = 0;
  }
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) {
    sm.whist[w][tid] = 0;
    sm.mask[0][w][tid] = 0;
    sm.mask[1][w][tid] = 0;
  }
  __syncthreads();
  const uint32_t tile = sm.tile;
  const uint64_t begin = (uint64_t)tile * kTile;
  if (begin >= m) return;  // past the keys, or after an expired wait (kSortClosed)
  const uint32_t valid = m - begin < kTile ? (uint32_t)(m - begin) : kTile;
  next_state[(size_t)tile * kRadix + tid] = 0;
  const uint32_t wbase = warp * (32 * ITEMS) + lane;
  const uint64_t* src = in + begin + wbase;
  uint64_t k[ITEMS];
  uint32_t r[ITEMS / 2];
  if (valid == kTile) {
#pragma unroll
    for (int j = 0; j < ITEMS; j++) k[j] = __ldcs(src + 32 * j);
    rank_keys<ITEMS, kHigh, true>(k, wbase, valid, shift, dmask, sm.mask, sm.whist[warp], r);
  } else {
    // Keys past the end take the last digit: they are last in the tile, so
    // they rank behind every real key.
#pragma unroll
    for (int j = 0; j < ITEMS; j++) k[j] = wbase + 32 * j < valid ? __ldcs(src + 32 * j) : ~0ull;
    rank_keys<ITEMS, kHigh, false>(k, wbase, valid, shift, dmask, sm.mask, sm.whist[warp], r);
  }
  __syncthreads();
  // Thread d: the tile's count of digit d, its first position in the tile
  // and every warp's slot for it.
  uint32_t cnt = 0, c[kSortWarps];
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) {
    c[w] = sm.whist[w][tid];
    cnt += c[w];
  }
  if (tid == kRadix - 1) cnt -= kTile - valid;
  W* own = state + (size_t)tile * kRadix + tid;
  TS::put(own, (tile == 0 ? TS::kPrefix : TS::kLocal) | cnt);
  uint32_t total;
  const uint32_t st = block_exclusive_scan<kSortThreads>(cnt, sm.scan_tmp, total);
  uint32_t run = st;
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) {
    sm.whist[w][tid] = run;
    run += c[w];
  }
  __syncthreads();
  const uint32_t* wh = sm.whist[warp];
#pragma unroll
  for (int j = 0; j < ITEMS; j++)
    if (valid == kTile || wbase + 32 * j < valid)
      sm.keys[wh[key_digit<kHigh>(k[j], shift, dmask)] + ((r[j / 2] >> (16 * (j & 1))) & 0xFFFFu)] =
          k[j];
  const W before = look_back(own, tile, cnt, ws, sm.abort);
  sm.gofs[tid] = ws[pass * kRadix + tid] + (uint32_t)before - st;
  __syncthreads();
  if (sm.abort) {  // a wait expired: the keys will not match the passes' digit counts
    if (tid < kMaxPasses) atomicOr(ws + kSortTickets + tid, kSortClosed);
    if (tid == 0) atomicExch(err, (unsigned long long)kDeviceErrTimeout);
    return;
  }
  // Position i of the tile goes to gofs[digit] + i (modulo 2^32; below m).
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const uint32_t i = tid + j * kSortThreads;
    if (valid == kTile || i < valid) {
      const uint64_t key = sm.keys[i];
      out[sm.gofs[key_digit<kHigh>(key, shift, dmask)] + i] = key;
    }
  }
}

template <int ITEMS, class W>
inline void launch_radix_pass(const uint64_t* in, uint64_t* out, uint64_t m, int shift,
                              uint32_t dmask, uint32_t* ws, int pass, uint64_t tiles,
                              cudaStream_t st, const unsigned long long* m_dev,
                              unsigned long long* err) {
  W* a = reinterpret_cast<W*>(ws + kSortStates);
  W* b = a + (size_t)kRadix * tiles;
  auto kernel = shift >= 32 ? k_radix_pass<ITEMS, W, true> : k_radix_pass<ITEMS, W, false>;
  kernel<<<(uint32_t)tiles, kSortThreads, 0, st>>>(in, out, m, shift, dmask, ws, pass,
                                                   pass & 1 ? b : a, pass & 1 ? a : b, m_dev, err);
}

// Sorts keys[0, m) by bits [lo, hi) stably; returns the buffer that holds the
// result (`keys` or `alt`).  m must be below 2^32.  `space` is checked to hold
// sort_words(m) words before anything is launched; `err` receives
// kDeviceErrTimeout if a device-side wait expired, and the result then is
// not even a permutation of the keys.  With `m_dev`, the sort covers only the first min(m, *m_dev) keys,
// a count known on the device alone (the launches are sized for m, so the
// sequence can be captured).
inline uint64_t* radix_sort(uint64_t* keys, uint64_t* alt, uint64_t m, int lo, int hi,
                            const SortSpace& space, unsigned long long* err, cudaStream_t st,
                            int* launches = nullptr, const unsigned long long* m_dev = nullptr) {
  if (m <= 1 || hi <= lo) return keys;
  if (space.count < sort_words(m)) fail(STC_ERR_INTERNAL, "sort workspace too small");
  uint32_t* ws = space.words;
  const uint64_t tiles = sort_tiles(m);
  const int items = sort_items(m);
  const bool wide = sort_wide(m);
  cudaMemsetAsync(ws, 0, (kSortStates + (size_t)kRadix * tiles * (wide ? 2 : 1)) * sizeof(uint32_t), st);
  const uint64_t per = (uint64_t)kSortThreads * kHistItems;
  const uint32_t grid = (uint32_t)((m + per - 1) / per < kSMs * 8 ? (m + per - 1) / per : kSMs * 8);
  k_radix_hist<<<grid, kSortThreads, 0, st>>>(keys, m, lo, hi, ws, m_dev);
  uint64_t* src = keys;
  uint64_t* dst = alt;
  int pass = 0;
  for (int shift = lo; shift < hi; shift += 8, pass++) {
    const int w = hi - shift < 8 ? hi - shift : 8;
    const uint32_t dmask = (1u << w) - 1;
    auto run = [&](auto launch) {
      launch(src, dst, m, shift, dmask, ws, pass, tiles, st, m_dev, err);
    };
    if (wide) run(launch_radix_pass<16, uint64_t>);
    else if (items == 16) run(launch_radix_pass<16, uint32_t>);
    else if (items == 8) run(launch_radix_pass<8, uint32_t>);
    else run(launch_radix_pass<4, uint32_t>);
    uint64_t* t = src;
    src = dst;
    dst = t;
  }
  if (launches) *launches += 1 + pass;
  return src;
}

// ------------------------------------------------------- range scans ----
// Exclusive scan of 32-bit values produced by functor F (F(i) for i < n)
// into 64-bit outputs; `emit(i, prefix, value)` receives each element's
// exclusive prefix.  Three launches, no inter-CTA waiting:
//   k_range_reduce -> k_scan_small -> k_range_apply.
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

template <class F>
__global__ void __launch_bounds__(kScanThreads) k_range_reduce(F f, uint64_t n, uint64_t per_cta,
                                                               uint64_t* __restrict__ sums) {
  __shared__ uint64_t tmp[kScanThreads / 32 + 1];
  const uint64_t begin = (uint64_t)blockIdx.x * per_cta;
  const uint64_t end = begin + per_cta < n ? begin + per_cta : n;
  uint64_t s = 0;
  for (uint64_t i = begin + threadIdx.x; i < end; i += kScanThreads) s += f(i);
  s = warp_sum(s);
  if (lane_id() == 0) tmp[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t t = 0;
    for (int w = 0; w < kScanThreads / 32; w++) t += tmp[w];
    sums[blockIdx.x] = t;
  }
}

// Exclusive scan of a[0, n) in place; a[n] receives the total, or with `err`
// (a scan over what a sort left) 0 once the error word is set, and a[n + 1]
// the error word.
static __global__ void __launch_bounds__(1024) k_scan_small(
    uint64_t* __restrict__ a, uint32_t n, const unsigned long long* __restrict__ err) {
  __shared__ uint64_t tmp[33];
  const uint32_t per = (n + 1023) / 1024;
  const uint32_t b = threadIdx.x * per, e = b + per < n ? b + per : n;
  uint64_t s = 0;
  for (uint32_t i = b; i < e; i++) s += a[i];
  uint64_t total;
  uint64_t run = block_exclusive_scan<1024>(s, tmp, total);
  for (uint32_t i = b; i < e; i++) {
    uint64_t x = a[i];
    a[i] = run;
    run += x;
  }
  if (threadIdx.x == 0) {
    const uint64_t word = err ? *err : 0;
    a[n] = word ? 0 : total;
    a[n + 1] = word;
  }
}

// Index into a tile buffer with one padding word per 32: the blocked reads
// (thread t, item j at t * kScanItems + j) then hit 32 distinct banks.
__device__ __forceinline__ uint32_t tile_pad(uint32_t x) { return x + (x >> 5); }

// Every element's exclusive prefix to `emit`, tile by tile: f is evaluated
// and emit called in a striped order (consecutive threads on consecutive
// elements, so that the loads inside f and the stores inside emit
// coalesce), while the scan itself runs over a blocked copy of the tile's
// values in shared memory.
template <class F, class E>
__global__ void __launch_bounds__(kScanThreads) k_range_apply(F f, E emit, uint64_t n,
                                                              uint64_t per_cta,
                                                              const uint64_t* __restrict__ offs) {
  constexpr uint32_t kPadded = kScanTile + kScanTile / 32;
  __shared__ uint64_t tmp[kScanThreads / 32 + 1];
  __shared__ uint32_t sv[kPadded];  // values
  __shared__ uint64_t sp[kPadded];  // tile-relative exclusive prefixes
  const uint64_t begin = (uint64_t)blockIdx.x * per_cta;
  const uint64_t end = begin + per_cta < n ? begin + per_cta : n;
  uint64_t carry = offs[blockIdx.x];
  for (uint64_t tile = begin; tile < end; tile += kScanTile) {
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
      const uint32_t x = j * kScanThreads + threadIdx.x;
      sv[tile_pad(x)] = tile + x < end ? f(tile + x) : 0u;
    }
    __syncthreads();
    uint32_t v[kScanItems];
    uint64_t s = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
      v[j] = sv[tile_pad(threadIdx.x * kScanItems + j)];
      s += v[j];
    }
    uint64_t total;
    uint64_t run = block_exclusive_scan<kScanThreads>(s, tmp, total);
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
      sp[tile_pad(threadIdx.x * kScanItems + j)] = run;
      run += v[j];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
      const uint32_t x = j * kScanThreads + threadIdx.x;
      if (tile + x < end) emit(tile + x, carry + sp[tile_pad(x)], sv[tile_pad(x)]);
    }
    carry += total;
    __syncthreads();  // the next tile reuses sv and sp
  }
}

// The first two launches of a range scan: per-CTA totals, then their
// exclusive scan in place; the grand total and the error word (k_scan_small)
// land in sums[grid] and sums[grid + 1], and the returned grid is what
// range_apply needs.  `sums` needs kScanSums words.
constexpr uint32_t kScanSums = kMaxSortGrid + 2;
template <class F>
inline uint32_t range_reduce_scan(F f, uint64_t n, uint64_t* sums, cudaStream_t st,
                                  int* launches = nullptr,
                                  const unsigned long long* err = nullptr) {
  RangePartition p = range_partition(n, kScanTile, kMaxSortGrid);
  k_range_reduce<<<p.grid, kScanThreads, 0, st>>>(f, n, p.per_cta, sums);
  k_scan_small<<<1, 1024, 0, st>>>(sums, p.grid, err);
  if (launches) *launches += 2;
  return p.grid;
}

// The third launch: every element's exclusive prefix to `emit`, from the
// offsets range_reduce_scan left in `sums` (which the caller may read, e.g.
// the total, in between).
template <class F, class E>
inline void range_apply(F f, E emit, uint64_t n, const uint64_t* sums, cudaStream_t st,
                        int* launches = nullptr) {
  RangePartition p = range_partition(n, kScanTile, kMaxSortGrid);
  k_range_apply<<<p.grid, kScanThreads, 0, st>>>(f, emit, n, p.per_cta, sums);
  if (launches) *launches += 1;
}

// The whole three-launch scan.
template <class F, class E>
inline void range_scan(F f, E emit, uint64_t n, uint64_t* sums, cudaStream_t st,
                       int* launches = nullptr) {
  range_reduce_scan(f, n, sums, st, launches);
  range_apply(f, emit, n, sums, st, launches);
}

}  // namespace stc
