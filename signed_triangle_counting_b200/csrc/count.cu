// Intersection engine: per-type signed triangle counts over the rank-space
// forward CSR.
//
// Reference: count_triangles / merge_intersect / classify
// (MC/tc_serial.cpp:95-170), intersect_signed_ranked
// (MC/tc_merge_sign_enu.cpp:12-44) and the hash probe
// (MC/tc_hash_sign_enu.cpp:125-165), MC = "Signed_TC/Multicore
// Implementations".  In rank space every list is sorted and every head has a
// higher rank than its tail, so for the arc u -> v stored at position k of
// N+(u), the third vertex w of a triangle lies in the suffix
// A' = N+(u)[k+1 ..] and in B = N+(v); the reference's rank filter
// (tc_serial.cpp:126) is implied.
//
// Work is grouped by source vertex u, in classes of d = |N+(u)|:
//   tiny   2 <= d <= 8        one thread per vertex, A in registers,
//                             monotone binary search of A' in B
//   warp   d <= 128           one warp per vertex     } N+(u) staged in
//   block  d <= 1024          one CTA per vertex      } shared memory
//   large  d <= 4096          one 512-thread CTA      }
//   giant  larger             one CTA per vertex, A read from global memory
// A 16x16 dispatch table per class (warp, block, large, giant) indexed by
// (bucket |A'|, bucket |B|) picks each arc's strategy:
//   HASH    B is streamed and every element is looked up in a shared-memory
//           hash of N+(u) whose keys carry the sign, so one 8-byte bucket
//           read answers membership and the A' sign together
//   MERGE   B is streamed and each 16-byte chunk is located in the staged
//           sorted A' by one binary search, its four keys merged forward
//   SEARCH  a warp takes the arc: each lane holds one pivot of B, an A'
//           element finds its segment with five shuffles and is searched in
//           that short segment of B
// HASH and MERGE arcs of one vertex form a single stream of aligned int4
// chunks (prefix sums over the arcs' chunk counts, a per-thread arc cursor),
// so every lane stays busy across arc boundaries and several loads stay in
// flight per thread.  Counters: per-thread packed 16-bit fields by number of
// negative edges, widened into u64 per vertex, then warp shuffle + block
// reduction and one atomic per counter per CTA.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "internal.h"
#include "radix_sort.cuh"
#include "stc_device.cuh"

namespace stc {

namespace {

constexpr uint32_t kEmpty = 0xFFFFFFFFu;
constexpr uint32_t kTinyMax = 8;
constexpr uint32_t kWarpCap = 128;    // staged capacity of the warp class
constexpr uint32_t kBlockCap = 1024;  // ... of the block class
constexpr uint32_t kLargeCap = 4096;  // ... of the large class
constexpr int kStreamUnroll = 2;      // int4 chunks in flight per thread
// Device error word value: a list exceeded its staged shared-memory capacity
// (the kernel skipped it instead of overrunning).
constexpr unsigned long long kErrStageCapacity = 3;

struct Csr {
  const uint64_t* __restrict__ off;
  const uint32_t* __restrict__ nbr;  // padded by 4 entries for whole int4 chunks
  const int8_t* __restrict__ sgn;
  const uint32_t* __restrict__ verts;  // rank -> id (per-source counts only)
  uint32_t n;
  // Sign-split heads (same offsets, padded likewise) and positives per
  // vertex; null unless a count uses STC_STRATEGY_SPLIT.
  const uint32_t* __restrict__ nbr_split = nullptr;
  const uint32_t* __restrict__ psplit = nullptr;
  // Heads with their signs, id << 1 | negative (same offsets, padded
  // likewise): what the head side streams, one 16-byte load per chunk.
  const uint32_t* __restrict__ nkey = nullptr;
  // Arcs whose shorter list has at most so many entries are counted where the
  // head side's keys are made; the tail side's kernels skip them (0: none).
  uint32_t short_max = 0;
};

// Per-thread type counters indexed by the number of negative edges.
struct TypeCounts {
  unsigned long long c[4] = {0, 0, 0, 0};
  __device__ __forceinline__ void add(uint32_t neg) {
    c[0] += neg == 0;
    c[1] += neg == 1;
    c[2] += neg == 2;
    c[3] += neg == 3;
  }
};

// Four 16-bit counters packed in one word: one add per triangle; widened
// into TypeCounts before any field can reach 2^16.
struct PackedCounts {
  unsigned long long w = 0;
  __device__ __forceinline__ void add(uint32_t neg) { w += 1ull << (16 * neg); }
  __device__ __forceinline__ void add_if(bool hit, uint32_t neg) {
    w += (unsigned long long)hit << (16 * neg);
  }
  __device__ __forceinline__ void drain(TypeCounts& tc) {
    tc.c[0] += w & 0xFFFF;
    tc.c[1] += (w >> 16) & 0xFFFF;
    tc.c[2] += (w >> 32) & 0xFFFF;
    tc.c[3] += w >> 48;
    w = 0;
  }
};

// Four 8-bit counters packed in one 32-bit word, for the streamed chunks:
// one 32-bit shift and add per triangle; widened into TypeCounts before any
// field can reach 2^8.
struct PackedCounts8 {
  uint32_t w = 0;
  __device__ __forceinline__ void add(uint32_t neg) { w += 1u << (8 * neg); }
  // Branch-free: adds nothing unless `hit`; neg <= 3 either way.
  __device__ __forceinline__ void add_if(bool hit, uint32_t neg) { w += (uint32_t)hit << (8 * neg); }
  __device__ __forceinline__ void drain(TypeCounts& tc) {
    tc.c[0] += w & 0xFFu;
    tc.c[1] += (w >> 8) & 0xFFu;
    tc.c[2] += (w >> 16) & 0xFFu;
    tc.c[3] += w >> 24;
    w = 0;
  }
};

__device__ __forceinline__ uint32_t size_bucket(uint32_t x) { return min(15u, 32u - __clz(x)); }

// First index i in [0, len) with a[i] >= x (len if none); `a` may point to
// shared or global memory.
__device__ __forceinline__ uint32_t lower_bound(const uint32_t* a, uint32_t len, uint32_t x) {
  uint32_t lo = 0, hi = len;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (a[mid] < x)
      lo = mid + 1;
    else
      hi = mid;
  }
  return lo;
}

// Multiplicative hash: the top bits of x * an odd constant.
// It hashes 2x, so that a signed key 2x | sign hashes by clearing its sign
// bit (hash_slot_k2) without a shift.
__device__ __forceinline__ uint32_t hash_slot(uint32_t x, uint32_t shift) {
  return ((x << 1) * 0x85EBCA77u) >> shift;
}
__device__ __forceinline__ uint32_t hash_slot_k2(uint32_t k2, uint32_t shift) {
  return (k2 * 0x85EBCA77u) >> shift;
}


// SEARCH for one arc by one warp: each lane holds the pivot B[lane * step];
// an A' element (a[i], i in [i0, d)) finds its segment with five shuffles and
// is searched inside that short segment of B, so a lookup costs about one
// memory latency instead of log2 |B| dependent loads.
template <class Counts>
__device__ __forceinline__ void arc_search(const uint32_t* a, const int8_t* s, uint32_t i0,
                                           uint32_t d, uint32_t nuv, const uint32_t* __restrict__ b,
                                           const int8_t* __restrict__ sb, uint32_t blen,
                                           uint32_t lane, Counts& cnt) {
  const uint32_t step = (blen + 31) >> 5;
  const uint32_t piv = b[min(lane * step, blen - 1)];
  for (uint32_t base = i0; base < d; base += 32) {
    const uint32_t i = base + lane;
    const uint32_t x = i < d ? a[i] : kEmpty;
    uint32_t seg = 0;
#pragma unroll
    for (uint32_t bit = 16; bit; bit >>= 1) {
      const uint32_t p = __shfl_sync(kFull, piv, seg + bit);
      if ((seg + bit) * step < blen && p <= x) seg += bit;
    }
    if (i >= d) continue;
    const uint32_t lo = seg * step;
    const uint32_t j = lo + lower_bound(b + lo, min(step, blen - lo), x);
    if (j < blen && b[j] == x) cnt.add(nuv + (s[i] < 0) + (sb[j] < 0));
  }
}

// MERGE for one arc by one warp over B streamed in int4 chunks (giant lists,
// whose A stays in global memory).
template <class Counts>
__device__ __forceinline__ void arc_merge_global(const uint32_t* a, const int8_t* s, uint32_t a0,
                                                 uint32_t d, uint32_t nuv,
                                                 const uint32_t* __restrict__ b,
                                                 const int8_t* __restrict__ sb, uint32_t blen,
                                                 uint32_t lane, Counts& tc) {
  const uint32_t alen = d - a0;
  const uint32_t alast = a[d - 1];
  for (uint32_t base = 0; base < blen; base += 128) {
    const uint32_t j0 = base + 4 * lane;
    if (__shfl_sync(kFull, j0 < blen ? b[j0] : kEmpty, 0) > alast) return;
    if (j0 >= blen) continue;
    uint32_t p = lower_bound(a + a0, alen, b[j0]);
    for (uint32_t j = j0; j < min(j0 + 4, blen); j++) {
      const uint32_t x = b[j];
      while (p < alen && a[a0 + p] < x) p++;
      if (p < alen && a[a0 + p] == x) tc.add(nuv + (s[a0 + p] < 0) + (sb[j] < 0));
    }
  }
}

// ---------------------------------------------------------- staging ----
// Strategy codes in the per-arc table: STC_STRATEGY_MERGE / _HASH / _SEARCH,
// or kNoArc for the last arc of a list (empty A') and arcs with empty B.
constexpr uint8_t kNoArc = 0xFF;
// Hash keys are id << 1 | (the A' edge is negative).  Ids stay below
// 2^31 - 2, so a key is at most 0xFFFFFFFB: it never equals kEmpty, and no
// key matches kNoId, the id that pads the entries of a chunk outside its arc.
// A query x matches key w exactly when w - 2x is 0 or 1, and that difference
// is the A' sign.
constexpr uint32_t kNoId = 0x7FFFFFFEu;

// Shared-memory image of one staged list of capacity `cap` with `nb` hash
// buckets: the hash (two 32-bit keys per 8-byte bucket), the sorted ids,
// each arc's B extent [lo, hi) as element indices of the CSR, the first
// negative head of a SPLIT arc's B in the split copy, the chunk prefix
// sums, then the byte arrays (list signs, arc strategies).
struct StageMem {
  uint32_t* hk;
  uint32_t* a;
  uint32_t* lo;
  uint32_t* hi;
  uint32_t* sp;
  uint32_t* pre;
  int8_t* s;
  uint8_t* st;
  __host__ __device__ static constexpr size_t bytes(uint32_t cap, uint32_t nb) {
    return 8ull * nb + 22ull * cap + 4;
  }
  __device__ static StageMem carve(unsigned char* p, uint32_t cap, uint32_t nb) {
    StageMem m;
    uint32_t* w = reinterpret_cast<uint32_t*>(p);
    m.hk = w;
    w += 2 * nb;
    m.a = w;
    w += cap;
    m.lo = w;
    w += cap;
    m.hi = w;
    w += cap;
    m.sp = w;
    w += cap;
    m.pre = w;
    w += cap + 1;
    int8_t* b = reinterpret_cast<int8_t*>(w);
    m.s = b;
    b += cap;
    m.st = reinterpret_cast<uint8_t*>(b);
    return m;
  }
};

// Hash geometry for a list of length d: next_pow2(hf d) buckets of two keys
// (hf = 4: load <= 1/8), at most `nb_cap` buckets.
struct Geo {
  uint32_t nb, shift;
  __device__ static Geo of(uint32_t d, uint32_t nb_cap, uint32_t hf) {
    Geo g;
    g.nb = 4;
    while (g.nb < hf * d && g.nb < nb_cap) g.nb <<= 1;
    g.shift = 32 - (31 - __clz(g.nb));
    return g;
  }
};

struct WarpSync {
  __device__ __forceinline__ void operator()() const { __syncwarp(); }
};
struct BlockSync {
  __device__ __forceinline__ void operator()() const { __syncthreads(); }
};

// Stages N+(u) (d entries at ub) for a team of TS threads (index t): clears
// the hash, copies ids and signs, fetches every arc's B extent, then fills
// the hash and picks each arc's strategy from the table.
template <int TS, class Sync>
__device__ __forceinline__ void stage(const Csr& g, uint64_t ub, uint32_t d, uint32_t t,
                                      const StageMem& m, const Geo& geo,
                                      const uint8_t (*table)[16], Sync sync) {
  for (uint32_t i = t; i < 2 * geo.nb; i += TS) m.hk[i] = kEmpty;
  for (uint32_t i = t; i < d; i += TS) {
    const uint32_t v = g.nbr[ub + i];
    m.a[i] = v;
    m.s[i] = g.sgn[ub + i];
    m.lo[i] = (uint32_t)g.off[v];
    m.hi[i] = (uint32_t)g.off[v + 1];
  }
  sync();
  for (uint32_t i = t; i < d; i += TS) {
    const uint32_t x = m.a[i];
    const uint32_t key = (x << 1) | (uint32_t)(m.s[i] < 0);
    uint32_t b = hash_slot(x, geo.shift);
    while (atomicCAS(&m.hk[2 * b], kEmpty, key) != kEmpty &&
           atomicCAS(&m.hk[2 * b + 1], kEmpty, key) != kEmpty)
      b = (b + 1) & (geo.nb - 1);
    const uint32_t blen = m.hi[i] - m.lo[i];
    uint8_t st = (i + 1 < d && blen) ? table[size_bucket(d - i - 1)][size_bucket(blen)] : kNoArc;
    if (st == STC_STRATEGY_HEAD || min(d - i - 1, blen) <= g.short_max)
      st = kNoArc;  // counted by the head-side pass, or with its keys
    m.st[i] = st;
    if (st == STC_STRATEGY_SPLIT) m.sp[i] = m.lo[i] + g.psplit[x];
  }
  sync();
}

// Exact lookup of x from its home bucket on: 0 if x is not in the hash,
// else 1 | (the key's sign flag << 1).
__device__ __noinline__ uint32_t probe_rest(const uint32_t* hk, uint32_t nb, uint32_t shift,
                                            uint32_t x) {
  const uint32_t q = x << 1;
  uint32_t b = hash_slot(x, shift);
  while (true) {
    const uint2 w = *reinterpret_cast<const uint2*>(hk + 2 * b);
    const uint32_t d0 = w.x - q, d1 = w.y - q;
    if (d0 < 2) return 1u | (d0 << 1);
    if (d1 < 2) return 1u | (d1 << 1);
    if (w.y == kEmpty) return 0;
    b = (b + 1) & (nb - 1);
  }
}

// Chunks of arc i's streamed extent: aligned groups of 4 entries (16
// bytes), or of 8 entries (32 bytes) with kWide (the head side's stream).
template <bool kWide = false>
__device__ __forceinline__ uint32_t arc_chunks(const StageMem& m, uint32_t i) {
  const uint8_t st = m.st[i];
  if (st != STC_STRATEGY_HASH && st != STC_STRATEGY_MERGE && st != STC_STRATEGY_SPLIT) return 0;
  return kWide ? ((m.hi[i] + 7) >> 3) - (m.lo[i] >> 3) : ((m.hi[i] + 3) >> 2) - (m.lo[i] >> 2);
}

// pre[i] = chunks of the streamed arcs before arc i; pre[d] = total.
template <bool kWide = false>
__device__ __forceinline__ void warp_chunk_scan(const StageMem& m, uint32_t d, uint32_t lane) {
  uint32_t carry = 0;
  for (uint32_t r = 0; r < d; r += 32) {
    const uint32_t i = r + lane;
    const uint32_t c = i < d ? arc_chunks<kWide>(m, i) : 0;
    const uint32_t inc = warp_inclusive_scan(c);
    if (i < d) m.pre[i] = carry + inc - c;
    carry += __shfl_sync(kFull, inc, 31);
  }
  if (lane == 0) m.pre[d] = carry;
  __syncwarp();
}

template <int THREADS, bool kWide = false>
__device__ __forceinline__ void block_chunk_scan(const StageMem& m, uint32_t d, uint32_t* tmp) {
  uint32_t carry = 0;
  for (uint32_t r = 0; r < d; r += THREADS) {
    const uint32_t i = r + threadIdx.x;
    const uint32_t c = i < d ? arc_chunks<kWide>(m, i) : 0;
    uint32_t total;
    const uint32_t excl = block_exclusive_scan<THREADS>(c, tmp, total);
    if (i < d) m.pre[i] = carry + excl;
    carry += total;
  }
  if (threadIdx.x == 0) m.pre[d] = carry;
  __syncthreads();
}

__device__ __forceinline__ uint32_t pick4(const uint4& q, uint32_t e) {
  const uint32_t lo = (e & 1) ? q.y : q.x;
  const uint32_t hi = (e & 1) ? q.w : q.z;
  return (e & 2) ? hi : lo;
}

// Mask of the entries of int4 chunk ci (elements 4 ci .. 4 ci + 3) that lie
// inside the arc's extent [lo, hi).
__device__ __forceinline__ uint32_t chunk_mask(uint32_t ci, uint32_t lo, uint32_t hi) {
  const uint32_t g0 = 4 * ci;
  const uint32_t first = lo > g0 ? lo - g0 : 0;
  const uint32_t last = min(hi - g0, 4u);
  return ((1u << last) - 1) & ~((1u << first) - 1);
}

// Chunk ci of an arc's B: from the sorted heads with their sign bytes, or,
// for a SPLIT arc, from the sign-split copy, where an element is negative
// exactly when its index is at least `sp` (the sign word is synthesised in
// the layout of the sign bytes: bit 8 e + 7 for element e).
__device__ __forceinline__ void load_chunk(const Csr& g, uint32_t ci, uint32_t st, uint32_t sp,
                                           uint4& q, uint32_t& sw) {
  if (st == STC_STRATEGY_SPLIT) {
    q = reinterpret_cast<const uint4*>(g.nbr_split)[ci];
    const uint32_t g0 = 4 * ci;
    sw = ((uint32_t)(g0 >= sp) << 7) | ((uint32_t)(g0 + 1 >= sp) << 15) |
         ((uint32_t)(g0 + 2 >= sp) << 23) | ((uint32_t)(g0 + 3 >= sp) << 31);
  } else {
    q = reinterpret_cast<const uint4*>(g.nbr)[ci];
    sw = reinterpret_cast<const uint32_t*>(g.sgn)[ci];
  }
}

// One int4 chunk of B for arc k of a staged list: four ids q, their four sign
// bytes sw, and the mask vm (non-zero) of the ids inside the arc.  HASH looks
// every id up in the staged hash (one 8-byte bucket read gives membership and
// the A' sign): ids outside the arc are replaced by kNoId, which matches no
// key, and the rare id whose home bucket is full without a match is looked up
// again past it, once per chunk.  MERGE locates the chunk in the sorted
// A' = a[k+1 ..) by one binary search and merges its ascending ids forward.
// At most four adds per chunk reach any one field of `pc`.  The HASH
// lookups are branch-free: with a few percent of ids hitting, some lane of a
// warp hits at almost every step, so a branch per hit would diverge at
// almost every step.
template <class PC>
__device__ __forceinline__ void process_chunk(const StageMem& m, uint32_t d, const Geo& geo,
                                              const uint4& q, uint32_t sw, uint32_t vm, uint32_t k,
                                              uint32_t nuv, uint32_t st, PC& pc) {
  if (st != STC_STRATEGY_MERGE) {  // HASH or SPLIT
    uint4 x4 = q;
    if (vm != 0xFu) {
      x4.x = (vm & 1u) ? x4.x : kNoId;
      x4.y = (vm & 2u) ? x4.y : kNoId;
      x4.z = (vm & 4u) ? x4.z : kNoId;
      x4.w = (vm & 8u) ? x4.w : kNoId;
    }
    bool again = false;
#pragma unroll
    for (uint32_t e = 0; e < 4; e++) {
      const uint32_t x = pick4(x4, e);
      const uint2 w = *reinterpret_cast<const uint2*>(m.hk + 2 * hash_slot(x, geo.shift));
      const uint32_t d0 = w.x - 2 * x, d1 = w.y - 2 * x;
      const bool hit = d0 < 2 || d1 < 2;
      again |= !hit && w.y != kEmpty;
      pc.add_if(hit, nuv + (d0 < 2 ? d0 : d1 & 1u) + ((sw >> (8 * e + 7)) & 1u));
    }
    if (again) {
#pragma unroll 1
      for (uint32_t e = 0; e < 4; e++) {
        const uint32_t x = pick4(x4, e);
        const uint2 w = *reinterpret_cast<const uint2*>(m.hk + 2 * hash_slot(x, geo.shift));
        if (w.x - 2 * x < 2 || w.y - 2 * x < 2 || w.y == kEmpty) continue;  // settled above
        const uint32_t r = probe_rest(m.hk, geo.nb, geo.shift, x);
        if (r) pc.add(nuv + (r >> 1) + ((sw >> (8 * e + 7)) & 1u));
      }
    }
  } else {  // MERGE
    const uint32_t a0 = k + 1, alen = d - a0;
    const uint32_t* a = m.a + a0;
    const uint32_t e0 = __ffs(vm) - 1;
    uint32_t p = lower_bound(a, alen, pick4(q, e0));
    for (uint32_t e = e0; e < 4 && ((vm >> e) & 1u); e++) {
      const uint32_t x = pick4(q, e);
      while (p < alen && a[p] < x) p++;
      if (p < alen && a[p] == x) pc.add(nuv + (m.s[a0 + p] < 0) + ((sw >> (8 * e + 7)) & 1u));
    }
  }
}

// HASH for an aligned chunk of eight signed heads (id << 1 | negative, the
// head side's stream; a, then b), vm its 8-bit mask: as process_chunk's HASH
// path, with each entry's sign taken from its own low bit instead of a
// separate sign word, one mask test and one overflow test per eight keys.
template <class PC>
__device__ __forceinline__ void process_keyed_chunk8(const StageMem& m, const Geo& geo, uint4 a,
                                                     uint4 b, uint32_t vm, uint32_t nuv,
                                                     PC& pc) {
  constexpr uint32_t kNoKey = kNoId << 1;
  if (vm != 0xFFu) {
    a.x = (vm & 1u) ? a.x : kNoKey;
    a.y = (vm & 2u) ? a.y : kNoKey;
    a.z = (vm & 4u) ? a.z : kNoKey;
    a.w = (vm & 8u) ? a.w : kNoKey;
    b.x = (vm & 16u) ? b.x : kNoKey;
    b.y = (vm & 32u) ? b.y : kNoKey;
    b.z = (vm & 64u) ? b.z : kNoKey;
    b.w = (vm & 128u) ? b.w : kNoKey;
  }
  bool again = false;
#pragma unroll
  for (uint32_t e = 0; e < 8; e++) {
    const uint32_t key = e < 4 ? pick4(a, e) : pick4(b, e - 4);
    const uint32_t k2 = key & ~1u;  // 2 x
    const uint2 w = *reinterpret_cast<const uint2*>(m.hk + 2 * hash_slot_k2(k2, geo.shift));
    const uint32_t d0 = w.x - k2, d1 = w.y - k2;
    const bool hit = d0 < 2 || d1 < 2;
    again |= !hit && w.y != kEmpty;
    pc.add_if(hit, nuv + (d0 < 2 ? d0 : d1 & 1u) + (key & 1u));
  }
  if (again) {
#pragma unroll 1
    for (uint32_t e = 0; e < 8; e++) {
      const uint32_t key = e < 4 ? pick4(a, e) : pick4(b, e - 4), x = key >> 1;
      const uint2 w = *reinterpret_cast<const uint2*>(m.hk + 2 * hash_slot(x, geo.shift));
      if (w.x - (key & ~1u) < 2 || w.y - (key & ~1u) < 2 || w.y == kEmpty) continue;
      const uint32_t r = probe_rest(m.hk, geo.nb, geo.shift, x);
      if (r) pc.add(nuv + (r >> 1) + (key & 1u));
    }
  }
}

// Adds a chunk's packed counts (8-bit fields) to an arc's two words of 16-bit
// fields.
__device__ __forceinline__ void add_to_arc(uint32_t p, uint32_t* w0, uint32_t* w1) {
  const uint32_t a = (p & 0xFFu) | ((p << 8) & 0xFF0000u);
  const uint32_t b = ((p >> 16) & 0xFFu) | ((p >> 8) & 0xFF0000u);
  if (a) atomicAdd(w0, a);
  if (b) atomicAdd(w1, b);
}

// The head side's stream: the staged in-arcs' A' extents of signed heads
// (g.nkey) as one sequence of aligned 8-entry (32-byte) chunks, shared out
// as in stream_pass (warp shares, lanes on consecutive chunks, the last
// eighth claimed from `next`).  A lane loads a chunk with two 16-byte
// loads, UK chunks per round, and the cursor, mask and branch work per
// chunk is spread over eight keys instead of four.  pre[] counts 8-entry
// chunks (block_chunk_scan / warp_chunk_scan with kWide).  kArc: each arc's
// counts go to its words in m.a and m.sp (zero on entry) instead of tc.
template <int UK, bool kArc>
__device__ __forceinline__ void stream_pass_keyed(const Csr& g, const StageMem& m, uint32_t d,
                                                  uint32_t warp, uint32_t warps, uint32_t lane,
                                                  const Geo& geo, TypeCounts& tc,
                                                  uint32_t* next) {
  const uint32_t total = m.pre[d];
  const uint32_t fixed = next ? total - total / 8 : total;
  const uint32_t per = (fixed + warps - 1) / warps;
  uint32_t seg_begin = min(fixed, warp * per), seg_end = min(fixed, seg_begin + per);
  uint32_t k = 0, pk, pk1, cb, mf, ml, anuv;
  auto enter = [&](uint32_t kk) {
    pk = m.pre[kk];
    pk1 = m.pre[kk + 1];
    const uint32_t alo = m.lo[kk], ahi = m.hi[kk];
    cb = (alo >> 3) - pk;
    mf = (0xFFu << (alo & 7u)) & 0xFFu;
    ml = 0xFFu >> (7u - ((ahi - 1u) & 7u));
    anuv = m.s[kk] < 0;
  };
  // 8-bit fields: at most 8 UK adds per field per round.
  constexpr uint32_t kDrainRounds = 255 / (8 * UK);
  constexpr uint32_t kClaim = 32 * UK;  // 8-entry chunks a warp claims at a time (one round)
  const uint4* src = reinterpret_cast<const uint4*>(g.nkey);
  PackedCounts8 p8;
  uint32_t rounds = 0;
  while (true) {
    if (seg_begin < seg_end) {
      {
        uint32_t lo_k = k, hi_k = d;
        const uint32_t c0 = seg_begin + lane;
        while (hi_k - lo_k > 1) {
          const uint32_t mid = (lo_k + hi_k) >> 1;
          if (m.pre[mid] <= c0) lo_k = mid; else hi_k = mid;
        }
        k = lo_k;
        enter(k);
      }
      for (uint32_t base = seg_begin; base < seg_end; base += 32 * UK) {
        uint4 qa[UK], qb[UK];
        uint32_t vm[UK], snuv[UK], sk[UK];
#pragma unroll
        for (int u = 0; u < UK; u++) {
          const uint32_t c = base + 32 * u + lane;
          vm[u] = 0;
          if (c < seg_end) {
            if (c >= pk1) {
              do {
                k++;
              } while (m.pre[k + 1] <= c);
              enter(k);
            }
            const uint32_t ci = cb + c;
            qa[u] = src[2 * ci];
            qb[u] = src[2 * ci + 1];
            vm[u] = (c == pk ? mf : 0xFFu) & (c + 1 == pk1 ? ml : 0xFFu);
            snuv[u] = anuv;
            sk[u] = k;
          }
        }
#pragma unroll
        for (int u = 0; u < UK; u++) {
          if (!vm[u]) continue;
          process_keyed_chunk8(m, geo, qa[u], qb[u], vm[u], snuv[u], p8);
          if (kArc) {
            add_to_arc(p8.w, m.a + sk[u], m.sp + sk[u]);
            p8.w = 0;
          }
        }
        if (++rounds == kDrainRounds) {
          p8.drain(tc);
          rounds = 0;
        }
      }
    }
    if (!next) break;
    uint32_t s0 = 0;
    if (lane == 0) s0 = atomicAdd(next, kClaim);
    s0 = fixed + __shfl_sync(kFull, s0, 0);
    if (s0 >= total) break;
    seg_begin = s0;
    seg_end = min(total, s0 + kClaim);
  }
  p8.drain(tc);
}

// The streamed arcs of a staged list as one sequence of aligned int4
// chunks.  Warp w takes a contiguous 1/warps share of the sequence and its
// lanes take consecutive chunks (coalesced); each lane keeps the extent of
// its current arc in registers and moves its cursor only at an arc
// boundary.  With `next` (a shared counter, zero on entry), the shares
// cover the first 7/8 of the sequence and the warps then claim the rest
// 64 U chunks at a time, so that a warp held up by B lists from DRAM or
// by SEARCH arcs takes less of it and the CTA reaches its next barrier
// together.
// Per chunk: the four ids (one 16-byte load) and their four sign bytes (one
// 4-byte load), a 4-bit mask of the ids inside the arc, then for HASH one
// 8-byte bucket read per id answers membership and the A' sign together;
// MERGE chunks are merged against the sorted A' instead.
// kSplit: compiled with the SPLIT path (a split index per arc, a per-chunk
// choice of source); kernels without it stay as lean as before SPLIT.
template <int U, bool kSplit>
__device__ __forceinline__ void stream_pass(const Csr& g, const StageMem& m, uint32_t d,
                                            uint32_t warp, uint32_t warps, uint32_t lane,
                                            const Geo& geo, TypeCounts& tc, uint32_t* next) {
  const uint32_t total = m.pre[d];
  const uint32_t fixed = next ? total - total / 8 : total;
  const uint32_t per = (fixed + warps - 1) / warps;
  uint32_t seg_begin = min(fixed, warp * per), seg_end = min(fixed, seg_begin + per);
  // Arc cursor k and, per arc: chunk index = cb + flattened index; the masks
  // of its first and last chunk (every chunk between is whole).
  uint32_t k = 0, pk, pk1, cb, mf, ml, ast, anuv, asp = 0;
  auto enter = [&](uint32_t kk) {
    pk = m.pre[kk];
    pk1 = m.pre[kk + 1];
    const uint32_t alo = m.lo[kk], ahi = m.hi[kk];
    cb = (alo >> 2) - pk;
    mf = (0xFu << (alo & 3u)) & 0xFu;
    ml = 0xFu >> (3u - ((ahi - 1u) & 3u));
    ast = m.st[kk];
    anuv = m.s[kk] < 0;
    if (kSplit) asp = m.sp[kk];
  };
  // 8-bit fields: at most 4 U adds per field per round.
  constexpr uint32_t kDrainRounds = 255 / (4 * U);
  constexpr uint32_t kClaim = 64 * U;  // chunks a warp claims at a time
  PackedCounts8 p8;
  uint32_t rounds = 0;
  while (true) {
    if (seg_begin < seg_end) {
      // Forward to the last arc with pre[k] <= the lane's first chunk (the
      // chunks of a lane only grow, and pre[d] = total exceeds every chunk).
      {
        uint32_t lo_k = k, hi_k = d;
        const uint32_t c0 = seg_begin + lane;
        while (hi_k - lo_k > 1) {
          const uint32_t mid = (lo_k + hi_k) >> 1;
          if (m.pre[mid] <= c0) lo_k = mid; else hi_k = mid;
        }
        k = lo_k;
        enter(k);
      }
      for (uint32_t base = seg_begin; base < seg_end; base += 32 * U) {
        uint4 q[U];
        uint32_t sw[U], vm[U], sk[U], snuv[U], sst[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const uint32_t c = base + 32 * u + lane;
          vm[u] = 0;
          if (c < seg_end) {
            if (c >= pk1) {
              do {
                k++;
              } while (m.pre[k + 1] <= c);
              enter(k);
            }
            const uint32_t ci = cb + c;
            load_chunk(g, ci, kSplit ? ast : (uint32_t)STC_STRATEGY_HASH, asp, q[u], sw[u]);
            vm[u] = (c == pk ? mf : 0xFu) & (c + 1 == pk1 ? ml : 0xFu);
            sk[u] = k;
            snuv[u] = anuv;
            sst[u] = ast;
          }
        }
#pragma unroll
        for (int u = 0; u < U; u++)
          if (vm[u]) process_chunk(m, d, geo, q[u], sw[u], vm[u], sk[u], snuv[u], sst[u], p8);
        if (++rounds == kDrainRounds) {
          p8.drain(tc);
          rounds = 0;
        }
      }
    }
    if (!next) break;
    uint32_t s0 = 0;
    if (lane == 0) s0 = atomicAdd(next, kClaim);
    s0 = fixed + __shfl_sync(kFull, s0, 0);
    if (s0 >= total) break;
    seg_begin = s0;
    seg_end = min(total, s0 + kClaim);
  }
  p8.drain(tc);
}

// SEARCH arcs of a staged list, one arc per warp.
__device__ __forceinline__ void search_pass(const Csr& g, const StageMem& m, uint32_t d,
                                            uint32_t warp, uint32_t warps, uint32_t lane,
                                            PackedCounts& pc, TypeCounts& tc) {
  for (uint32_t k = warp; k + 1 < d; k += warps) {
    if (m.st[k] != STC_STRATEGY_SEARCH) continue;
    const uint32_t lo = m.lo[k];
    arc_search(m.a, m.s, k + 1, d, m.s[k] < 0, g.nbr + lo, g.sgn + lo, m.hi[k] - lo, lane, pc);
    pc.drain(tc);
  }
}

// ------------------------------------------------------ arc timing ----
// Timing recorder (CountConfig::arc_cycles): per dispatch cell
// (class, bucket |A'|, bucket |B|), the SM cycles spent on its arcs and the
// number of arcs.  In this mode every arc is processed alone by one warp,
// timed from the first load of its B to the last count it adds, so three runs
// with the strategy forced give every cell's cost under every strategy: the
// training data of the learned dispatcher and the measure of a dispatch
// table's regret.  The counting kernels proper pack the int4 chunks of all
// HASH and MERGE arcs of a list into one stream that keeps every lane busy,
// so such an arc of c chunks is charged its share of the lanes it would
// occupy there, c / (32 ceil(c / 32)) of the warp's time; a SEARCH arc holds
// a whole warp in both modes and is charged the warp's time.
struct ArcTimes {
  unsigned long long* cycles;  // kTableClasses * 256 cells
  unsigned long long* arcs;
};

// SM clock read that the compiler cannot hoist above the computation of
// `dep` (an input operand of the read).
__device__ __forceinline__ long long clock_after(unsigned long long dep) {
  long long t;
  asm volatile("mov.u64 %0, %%clock64;" : "=l"(t) : "l"(dep) : "memory");
  return t;
}

__device__ __forceinline__ void record_arc(const ArcTimes& at, uint32_t tclass, uint32_t alen,
                                           uint32_t blen, unsigned cycles) {
  const uint32_t cell = tclass * 256 + size_bucket(alen) * 16 + size_bucket(blen);
  atomicAdd(at.cycles + cell, (unsigned long long)cycles);
  atomicAdd(at.arcs + cell, 1ull);
}

// HASH or MERGE for arc k alone: the warp's lanes take consecutive int4
// chunks of B.
__device__ __forceinline__ void arc_stream(const Csr& g, const StageMem& m, uint32_t d, uint32_t k,
                                           uint32_t lane, const Geo& geo, PackedCounts& pc) {
  const uint32_t lo = m.lo[k], hi = m.hi[k], st = m.st[k], nuv = m.s[k] < 0;
  const uint32_t sp = st == STC_STRATEGY_SPLIT ? m.sp[k] : 0u;
  const uint32_t c1 = (hi + 3) >> 2;
  for (uint32_t ci = (lo >> 2) + lane; ci < c1; ci += 32) {
    uint4 q;
    uint32_t sw;
    load_chunk(g, ci, st, sp, q, sw);
    process_chunk(m, d, geo, q, sw, chunk_mask(ci, lo, hi), k, nuv, st, pc);
  }
}

// All arcs of a staged list, one arc per warp at a time, each timed.
__device__ __forceinline__ void timed_pass(const Csr& g, const StageMem& m, uint32_t d,
                                           uint32_t warp, uint32_t warps, uint32_t lane,
                                           const Geo& geo, PackedCounts& pc, TypeCounts& tc,
                                           const ArcTimes& at, uint32_t tclass) {
  for (uint32_t k = warp; k + 1 < d; k += warps) {
    const uint32_t st = m.st[k];
    if (st == kNoArc) continue;
    const uint32_t lo = m.lo[k], hi = m.hi[k], blen = hi - lo;
    __syncwarp();
    const long long t0 = clock_after(0);
    if (st == STC_STRATEGY_SEARCH)
      arc_search(m.a, m.s, k + 1, d, m.s[k] < 0, g.nbr + lo, g.sgn + lo, blen, lane, pc);
    else
      arc_stream(g, m, d, k, lane, geo, pc);
    // The arc's time is the latest lane's (each lane stops its clock once its
    // own counts are in).
    unsigned dt = __reduce_max_sync(kFull, (unsigned)(clock_after(pc.w) - t0));
    if (st != STC_STRATEGY_SEARCH) {  // lane share in the packed stream
      const uint32_t chunks = ((hi + 3) >> 2) - (lo >> 2);
      dt = (unsigned)((unsigned long long)dt * chunks / (32ull * ((chunks + 31) >> 5)));
    }
    pc.drain(tc);
    if (lane == 0) record_arc(at, tclass, d - k - 1, blen, max(dt, 1u));
  }
}

// ------------------------------------------------------- reductions ----
// Block reduction of the four counters and one atomic per counter.
// Slot C_T0 + k receives type Tk = 3 - (negative edges).
template <int THREADS>
__device__ __forceinline__ void flush_counts(const TypeCounts& tc, unsigned long long* __restrict__ ctr) {
  __shared__ unsigned long long red[THREADS / 32][4];
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const unsigned long long v = warp_sum(tc.c[k]);
    if (lane == 0) red[warp][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    unsigned long long s = 0;
    for (int w = 0; w < THREADS / 32; w++) s += red[w][threadIdx.x];
    if (s) atomicAdd(ctr + C_T0 + (3 - threadIdx.x), s);
  }
}

// Where per-vertex totals go when a kernel reports per vertex.
// kKeyed: the head side adds up the items of one key (sink.key(head)) and
// hands them over together; kPerArc: it hands over each in-arc's counts, which
// belong to the arc's tail.
struct TotalSink {  // only the four global counters
  static constexpr bool kPerVertex = false, kKeyed = false, kPerArc = false;
  __device__ void put(uint32_t, const unsigned long long*) const {}
};
struct VertexSink {  // per-source counts by original id: vcounts[4 * id + type]
  static constexpr bool kPerVertex = true, kKeyed = false, kPerArc = true;
  unsigned long long* vcounts;
  const uint32_t* verts;
  __device__ void put(uint32_t u, const unsigned long long* c) const {
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (c[k]) atomicAdd(vcounts + 4ull * verts[u] + (3 - k), c[k]);
  }
  __device__ void add(uint32_t u, uint32_t neg) const {
    atomicAdd(vcounts + 4ull * verts[u] + (3 - neg), 1ull);
  }
  // The head side's counts of one arc with tail u: fewer than 2^16 of each
  // number of negative edges, 0 and 1 in w0, 2 and 3 in w1.
  __device__ void add_arc(uint32_t u, uint32_t w0, uint32_t w1) const {
    if ((w0 | w1) == 0) return;
    unsigned long long* c = vcounts + 4ull * verts[u];
    if (w0 & 0xFFFFu) atomicAdd(c + 3, (unsigned long long)(w0 & 0xFFFFu));
    if (w0 >> 16) atomicAdd(c + 2, (unsigned long long)(w0 >> 16));
    if (w1 & 0xFFFFu) atomicAdd(c + 1, (unsigned long long)(w1 & 0xFFFFu));
    if (w1 >> 16) atomicAdd(c + 0, (unsigned long long)(w1 >> 16));
  }
};
struct GraphSink {  // per-graph counts of a batch: gcounts[4 * graph + type]
  static constexpr bool kPerVertex = true, kKeyed = true, kPerArc = false;
  unsigned long long* gcounts;
  const uint64_t* gbase;  // G + 1 rank boundaries (graphs are contiguous in rank space)
  uint32_t G;
  __device__ uint32_t graph_of(uint32_t u) const {
    uint32_t lo = 0, hi = G;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (gbase[mid] <= u) lo = mid; else hi = mid;
    }
    return lo;
  }
  __device__ void put(uint32_t u, const unsigned long long* c) const { put_key(graph_of(u), c); }
  // Keyed form (the head side adds up the items of one key): the graph.
  __device__ uint32_t key(uint32_t u) const { return graph_of(u); }
  __device__ void put_key(uint32_t g, const unsigned long long* c) const {
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (c[k]) atomicAdd(gcounts + 4ull * g + (3 - k), c[k]);
  }
};

// Reduces one vertex's counters over the CTA and hands them to the sink.
template <int THREADS, class Sink>
__device__ __forceinline__ void block_vertex_flush(const TypeCounts& vc, uint32_t u, const Sink& sink) {
  __shared__ unsigned long long red[THREADS / 32][4];
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const unsigned long long v = warp_sum(vc.c[k]);
    if (lane == 0) red[warp][k] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long s[4] = {0, 0, 0, 0};
    for (int w = 0; w < THREADS / 32; w++)
      for (int k = 0; k < 4; k++) s[k] += red[w][k];
    sink.put(u, s);
  }
  __syncthreads();
}

// Reduces a key's counters over the CTA and hands them to the sink's keyed
// form (every thread calls it, with the same key).
template <int THREADS, class Sink>
__device__ __forceinline__ void block_key_flush(const TypeCounts& vc, uint32_t key,
                                                const Sink& sink) {
  __shared__ unsigned long long red[THREADS / 32][4];
  const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const unsigned long long v = warp_sum(vc.c[k]);
    if (lane == 0) red[warp][k] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long s[4] = {0, 0, 0, 0};
    for (int w = 0; w < THREADS / 32; w++)
      for (int k = 0; k < 4; k++) s[k] += red[w][k];
    sink.put_key(key, s);
  }
  __syncthreads();
}

template <class Sink>
__device__ __forceinline__ void warp_vertex_flush(const TypeCounts& vc, uint32_t u, uint32_t lane,
                                                  const Sink& sink) {
  unsigned long long s[4];
#pragma unroll
  for (int k = 0; k < 4; k++) s[k] = warp_sum(vc.c[k]);
  if (lane == 0) sink.put(u, s);
}

// ------------------------------------------------------------ classes ----
struct ClassBounds {
  uint32_t tiny_max, warp_max, block_max, large_max;
  __device__ __forceinline__ uint32_t of(uint32_t d) const {
    if (d < 2) return 5;
    if (d <= tiny_max) return 0;
    if (d <= warp_max) return 1;
    if (d <= block_max) return 2;
    if (d <= large_max) return 3;
    return 4;
  }
};
constexpr int kClasses = 5;
// Device plan of a persistent count: plan[c] = first list entry of class c
// (plan[kClasses] = total), plan[kPlanCounts + c] = its vertex count.
constexpr uint32_t kPlanCounts = 8;
constexpr uint32_t kPlanWords = kPlanCounts + kClasses;

// Source vertices [range[0], range[1]) of rank space, or all n when `range`
// is null (a sharded count reads its range from the counters).
__device__ __forceinline__ void source_range(const unsigned long long* range, uint32_t n,
                                             uint32_t& u0, uint32_t& u1) {
  u0 = range ? (uint32_t)range[0] : 0u;
  u1 = range ? (uint32_t)range[1] : n;
}

// `need` (optional): a vertex whose flag is 0 has no arc for the tail side
// (the head-side pass counts all of them) and joins no class.
__global__ void k_classify_count(const uint64_t* __restrict__ off, uint32_t n, ClassBounds cb,
                                 unsigned long long* __restrict__ ctr,
                                 const unsigned long long* __restrict__ range,
                                 const uint8_t* __restrict__ need = nullptr) {
  if (device_failed(ctr + C_ERROR)) return;  // no vertex in any class
  uint32_t cnt[kClasses] = {0, 0, 0, 0, 0};
  uint32_t dmax = 0;
  uint32_t u0, u1;
  source_range(range, n, u0, u1);
  for (uint32_t u = u0 + blockIdx.x * blockDim.x + threadIdx.x; u < u1; u += gridDim.x * blockDim.x) {
    const uint32_t d = (uint32_t)(off[u + 1] - off[u]);
    const uint32_t c = (need && !need[u]) ? 5u : cb.of(d);
    dmax = max(dmax, d);
#pragma unroll
    for (int i = 0; i < kClasses; i++) cnt[i] += c == (uint32_t)i;
  }
  dmax = __reduce_max_sync(kFull, dmax);
  if (lane_id() == 0) atomicMax(ctr + C_MAX_FDEG, (unsigned long long)dmax);
#pragma unroll
  for (int i = 0; i < kClasses; i++) {
    const uint32_t s = __reduce_add_sync(kFull, cnt[i]);
    if (lane_id() == 0 && s) atomicAdd(ctr + C_WORK + i, (unsigned long long)s);
  }
}

// Appends each vertex to its class list (order within a class is free: the
// counts are sums of integers); the cursors are ctr[C_WORK + class].
__global__ void k_classify_fill(const uint64_t* __restrict__ off, uint32_t n, ClassBounds cb,
                                uint32_t* __restrict__ lists, const uint32_t* __restrict__ starts,
                                unsigned long long* __restrict__ ctr,
                                const unsigned long long* __restrict__ range,
                                const uint8_t* __restrict__ need = nullptr) {
  if (device_failed(ctr + C_ERROR)) return;
  unsigned long long* cursor = ctr + C_WORK;
  uint32_t u0, u1;
  source_range(range, n, u0, u1);
  for (uint32_t base = u0 + blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < u1;
       base += gridDim.x * blockDim.x) {
    const uint32_t u = base + lane_id();
    const uint32_t c = (u >= u1 || (need && !need[u])) ? 5u : cb.of((uint32_t)(off[u + 1] - off[u]));
    if (!__any_sync(kFull, c < kClasses)) continue;
    const unsigned peers = __match_any_sync(kFull, c);
    const uint32_t leader = __ffs(peers) - 1;
    uint32_t pos = 0;
    if (c < kClasses && lane_id() == leader) pos = (uint32_t)atomicAdd(cursor + c, (unsigned long long)__popc(peers));
    pos = __shfl_sync(kFull, pos, leader) + __popc(peers & lanemask_lt());
    if (c < kClasses) lists[starts[c] + pos] = u;
  }
}

// Tiny class: one thread per vertex, A in registers, B in global memory.
// One tiny list (one thread): A in registers, a monotone binary search of
// each later A' element in B; arcs whose cell in `table` (the warp class's)
// is HEAD are left to the head-side pass.
template <int TMAX, class Sink>
__device__ __forceinline__ void tiny_vertex(const Csr& g, uint32_t u, const Sink& sink,
                                            const uint8_t (*table)[16], TypeCounts& tc) {
  constexpr bool kVC = Sink::kPerVertex;
  const uint64_t ub = g.off[u];
  const uint32_t d = (uint32_t)(g.off[u + 1] - ub);
  uint32_t a[TMAX];
  uint32_t neg[TMAX];
#pragma unroll
  for (int i = 0; i < TMAX; i++) {
    a[i] = i < (int)d ? g.nbr[ub + i] : kEmpty;
    neg[i] = i < (int)d ? (g.sgn[ub + i] < 0) : 0u;
  }
  TypeCounts vc;
#pragma unroll
  for (int k = 0; k < TMAX - 1; k++) {
    if (k + 1 >= (int)d) break;
    const uint64_t vb = g.off[a[k]];
    const uint32_t blen = (uint32_t)(g.off[a[k] + 1] - vb);
    if (table[size_bucket(d - k - 1)][size_bucket(blen)] == STC_STRATEGY_HEAD ||
        min(d - k - 1, blen) <= g.short_max)
      continue;
    const uint32_t* b = g.nbr + vb;
    uint32_t pos = 0;
#pragma unroll
    for (int i = k + 1; i < TMAX; i++) {
      if (i >= (int)d || pos >= blen) break;
      pos += lower_bound(b + pos, blen - pos, a[i]);
      if (pos < blen && b[pos] == a[i]) {
        const uint32_t t = neg[k] + neg[i] + (g.sgn[vb + pos] < 0);
        if (kVC) vc.add(t); else tc.add(t);
        pos++;
      }
    }
  }
  if (kVC) sink.put(u, vc.c);
}

// Tiny class: one thread per vertex, A in registers, B in global memory.
template <int TMAX, class Sink>
__global__ void __launch_bounds__(256) k_tiny(Csr g, const uint32_t* __restrict__ list, uint32_t cnt,
                                              unsigned long long* __restrict__ ctr, Sink sink,
                                              const uint8_t* __restrict__ gtable) {
  __shared__ uint8_t table[16][16];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) (&table[0][0])[i] = gtable[i];
  __syncthreads();
  TypeCounts tc;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < cnt; idx += gridDim.x * blockDim.x)
    tiny_vertex<TMAX>(g, list[idx], sink, table, tc);
  if (!Sink::kPerVertex) flush_counts<256>(tc, ctr);
}

// Warp class: one warp per vertex, staged in the warp's slice of shared
// memory (256 hash buckets).
constexpr uint32_t kWarpBuckets = 2 * kWarpCap;
constexpr size_t kWarpStageBytes = (StageMem::bytes(kWarpCap, kWarpBuckets) + 15) & ~size_t(15);

// One warp-class list, staged in the warp's shared-memory slice `m` with
// up to hf hash buckets per element; U int4 chunks in flight per lane.
template <class Sink, bool kTime, int U, bool kSplit>
__device__ __forceinline__ void warp_vertex(const Csr& g, uint32_t u, uint32_t lane,
                                            const StageMem& m, const uint8_t (*table)[16],
                                            uint32_t hf, unsigned long long* __restrict__ ctr,
                                            const Sink& sink, const ArcTimes& at, TypeCounts& tc) {
  constexpr bool kVC = Sink::kPerVertex;
  const uint64_t ub = g.off[u];
  const uint32_t d = (uint32_t)(g.off[u + 1] - ub);
  if (d > kWarpCap) {  // uniform over the warp
    if (lane == 0) atomicExch(ctr + C_ERROR, kErrStageCapacity);
    return;
  }
  const Geo geo = Geo::of(d, kWarpBuckets, hf);
  stage<32>(g, ub, d, lane, m, geo, table, WarpSync{});
  TypeCounts vc;
  TypeCounts& out = kVC ? vc : tc;
  PackedCounts pc;
  if (kTime) {
    timed_pass(g, m, d, 0, 1, lane, geo, pc, out, at, kTableWarp);
  } else {
    warp_chunk_scan(m, d, lane);
    stream_pass<U, kSplit>(g, m, d, 0, 1, lane, geo, out, nullptr);
    search_pass(g, m, d, 0, 1, lane, pc, out);
  }
  pc.drain(out);
  if (kVC) warp_vertex_flush(vc, u, lane, sink);
  __syncwarp();
}

template <class Sink, bool kTime, int U, bool kSplit>
__global__ void __launch_bounds__(256, U >= 4 ? 3 : 4) k_warp(Csr g, const uint32_t* __restrict__ list, uint32_t cnt,
                                              unsigned long long* __restrict__ ctr, Sink sink,
                                              const uint8_t* __restrict__ gtable, ArcTimes at,
                                              uint32_t hf) {
  constexpr bool kVC = Sink::kPerVertex;
  constexpr int kWarps = 8;
  __shared__ __align__(16) unsigned char smem[kWarps * kWarpStageBytes];
  __shared__ uint8_t table[16][16];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) (&table[0][0])[i] = gtable[i];
  __syncthreads();
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  const StageMem m = StageMem::carve(smem + w * kWarpStageBytes, kWarpCap, kWarpBuckets);
  TypeCounts tc;
  const uint32_t warps = gridDim.x * kWarps;
  for (uint32_t idx = blockIdx.x * kWarps + w; idx < cnt; idx += warps)
    warp_vertex<Sink, kTime, U, kSplit>(g, list[idx], lane, m, table, hf, ctr, sink, at, tc);
  if (!kVC) flush_counts<256>(tc, ctr);
}

// Block classes: one CTA per vertex from a dynamic queue, the list staged in
// dynamic shared memory of capacity `cap` with `nb` hash buckets
// (nb >= 2 * cap, powers of two).
inline size_t block_stage_bytes(uint32_t cap, uint32_t nb) { return StageMem::bytes(cap, nb); }
constexpr size_t kMaxStageSmem = 220 * 1024;  // dynamic shared memory a staged CTA may use

// One block-class list (the whole CTA), staged in `m` of capacity `cap`
// with `nb` hash buckets.  scan_tmp has THREADS / 32 + 2 words: the chunk
// scan's and the stream's claim counter.
template <int THREADS, class Sink, bool kTime, int U, bool kSplit>
__device__ __forceinline__ void block_vertex(const Csr& g, uint32_t u, uint32_t cap, uint32_t nb,
                                             uint32_t hf, const StageMem& m,
                                             const uint8_t (*table)[16],
                                             uint32_t* scan_tmp, unsigned long long* __restrict__ ctr,
                                             const Sink& sink, const ArcTimes& at, uint32_t tclass,
                                             TypeCounts& tc) {
  constexpr bool kVC = Sink::kPerVertex;
  constexpr uint32_t kWarps = THREADS / 32;
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  const uint64_t ub = g.off[u];
  const uint32_t d = (uint32_t)(g.off[u + 1] - ub);
  if (d > cap) {  // uniform over the CTA
    if (threadIdx.x == 0) atomicExch(ctr + C_ERROR, kErrStageCapacity);
    return;
  }
  const Geo geo = Geo::of(d, nb, hf);
  // The stream's claim counter: the CTA passed a barrier since the last list
  // used it, and stage() passes another before this one does.
  uint32_t* next = scan_tmp + kWarps + 1;
  if (threadIdx.x == 0) *next = 0;
  stage<THREADS>(g, ub, d, threadIdx.x, m, geo, table, BlockSync{});
  TypeCounts vc;
  TypeCounts& out = kVC ? vc : tc;
  PackedCounts pc;
  if (kTime) {
    timed_pass(g, m, d, w, kWarps, lane, geo, pc, out, at, tclass);
  } else {
    block_chunk_scan<THREADS>(m, d, scan_tmp);
    search_pass(g, m, d, w, kWarps, lane, pc, out);
    stream_pass<U, kSplit>(g, m, d, w, kWarps, lane, geo, out, next);
  }
  pc.drain(out);
  if (kVC) block_vertex_flush<THREADS>(vc, u, sink);
}

template <int THREADS, class Sink, bool kTime, int U, bool kSplit>
__global__ void __launch_bounds__(THREADS) k_block(Csr g, const uint32_t* __restrict__ list,
                                                   uint32_t cnt, uint32_t cap, uint32_t nb, uint32_t hf,
                                                   unsigned long long* __restrict__ queue,
                                                   unsigned long long* __restrict__ ctr, Sink sink,
                                                   const uint8_t* __restrict__ gtable, ArcTimes at,
                                                   uint32_t tclass, const uint32_t* __restrict__ plan,
                                                   uint32_t pclass) {
  constexpr bool kVC = Sink::kPerVertex;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint8_t table[16][16];
  __shared__ uint32_t scan_tmp[THREADS / 32 + 2];
  __shared__ uint32_t s_item;
  for (int i = threadIdx.x; i < 256; i += THREADS) (&table[0][0])[i] = gtable[i];
  if (plan) {  // list and count planned on the device
    list += plan[pclass];
    cnt = plan[kPlanCounts + pclass];
  }
  const StageMem m = StageMem::carve(smem, cap, nb);
  TypeCounts tc;
  while (true) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = (uint32_t)atomicAdd(queue, 1ull);
    __syncthreads();
    const uint32_t item = s_item;
    if (item >= cnt) break;
    block_vertex<THREADS, Sink, kTime, U, kSplit>(g, list[item], cap, nb, hf, m, table, scan_tmp,
                                                  ctr, sink, at, tclass, tc);
  }
  if (!kVC) flush_counts<THREADS>(tc, ctr);
}

// Giant lists (d > kLargeCap): one CTA per vertex, A read from global memory,
// one arc per warp; HASH falls back to MERGE (no staged hash).
template <int THREADS, class Sink, bool kTime>
__global__ void __launch_bounds__(THREADS) k_giant(Csr g, const uint32_t* __restrict__ list,
                                                   uint32_t cnt, unsigned long long* __restrict__ queue,
                                                   unsigned long long* __restrict__ ctr, Sink sink,
                                                   const uint8_t* __restrict__ gtable, ArcTimes at,
                                                   const uint32_t* __restrict__ plan, uint32_t pclass) {
  constexpr bool kVC = Sink::kPerVertex;
  __shared__ uint8_t table[16][16];
  __shared__ uint32_t s_item;
  for (int i = threadIdx.x; i < 256; i += THREADS) (&table[0][0])[i] = gtable[i];
  if (plan) {  // list and count planned on the device
    list += plan[pclass];
    cnt = plan[kPlanCounts + pclass];
  }
  constexpr uint32_t kWarps = THREADS / 32;
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  TypeCounts tc;
  while (true) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = (uint32_t)atomicAdd(queue, 1ull);
    __syncthreads();
    const uint32_t item = s_item;
    if (item >= cnt) break;
    const uint32_t u = list[item];
    const uint64_t ub = g.off[u];
    const uint32_t d = (uint32_t)(g.off[u + 1] - ub);
    const uint32_t* a = g.nbr + ub;
    const int8_t* s = g.sgn + ub;
    TypeCounts vc;
    TypeCounts& out = kVC ? vc : tc;
    for (uint32_t k = w; k + 1 < d; k += kWarps) {
      const uint32_t v = a[k];
      const uint64_t vb = g.off[v];
      const uint32_t blen = (uint32_t)(g.off[v + 1] - vb);
      if (blen == 0) continue;
      const uint32_t st = table[size_bucket(d - k - 1)][size_bucket(blen)];
      if (st == STC_STRATEGY_HEAD || min(d - k - 1, blen) <= g.short_max)
        continue;  // counted by the head-side pass, or with its keys
      long long t0 = 0;
      if (kTime) {
        __syncwarp();
        t0 = clock_after(0);
      }
      // 64-bit counters: a giant list may be long enough to overflow the
      // packed 16-bit fields within one arc.
      if (st == STC_STRATEGY_SEARCH)
        arc_search(a, s, k + 1, d, s[k] < 0, g.nbr + vb, g.sgn + vb, blen, lane, out);
      else
        arc_merge_global(a, s, k + 1, d, s[k] < 0, g.nbr + vb, g.sgn + vb, blen, lane, out);
      if (kTime) {
        const unsigned long long dep = out.c[0] + out.c[1] + out.c[2] + out.c[3];
        const unsigned dt = __reduce_max_sync(kFull, (unsigned)(clock_after(dep) - t0));
        if (lane == 0) record_arc(at, kTableGiant, d - k - 1, blen, dt);
      }
    }
    if (kVC) block_vertex_flush<THREADS>(vc, u, sink);
  }
  if (!kVC) flush_counts<THREADS>(tc, ctr);
}

// Compile-time choices of the tuned kernels, selected at run time.
template <int V> struct Int { static constexpr int value = V; };
template <class F> void with_unroll(uint32_t u, F&& f) {
  if (u == 1) f(Int<1>{});
  else if (u == 4) f(Int<4>{});
  else f(Int<2>{});
}
template <class F> void with_split(bool split, F&& f) {
  if (split) f(std::true_type{});
  else f(std::false_type{});
}
template <class F> void with_block_threads(uint32_t t, F&& f) {
  if (t == 128) f(Int<128>{});
  else if (t == 512) f(Int<512>{});
  else f(Int<256>{});
}

// Largest hash factor whose staged image of `cap` entries fits the
// shared memory of one CTA.
inline uint32_t fit_hash_factor(uint32_t hf, uint32_t cap) {
  while (hf > 1 && StageMem::bytes(cap, hf * cap) > kMaxStageSmem) hf >>= 1;
  return hf;
}

// Launches the class kernels for one sink kind.  `d_tables` holds one
// 256-byte table per TableClass; `tu` gives the tuned block size, hash
// factors and stream widths; classes outside `mask` are skipped.  The timing
// recorder (kTime) uses the default widths and block size, which its
// per-arc passes do not depend on.
template <class Sink, bool kTime>
void launch_classes(cudaStream_t st, const Csr& csr, const uint32_t* lists, const uint32_t* counts,
                    const uint32_t* starts, uint32_t max_fdeg, unsigned long long* ctr,
                    const uint8_t* d_tables, const Sink& sink, const ArcTimes& at,
                    const Tuning& tu, uint32_t mask, int& launches) {
  if (counts[0] && (mask & 1u)) {
    const uint32_t grid = std::min<uint32_t>((counts[0] + 255) / 256, kSMs * 8);
    k_tiny<kTinyMax, Sink><<<grid, 256, 0, st>>>(csr, lists + starts[0], counts[0], ctr, sink,
                                                  d_tables + 256 * kTableWarp);
    launches++;
  }
  if (counts[1] && (mask & 2u)) {
    const uint32_t grid = std::min<uint32_t>((counts[1] + 7) / 8, kSMs * 8);
    const uint32_t u = kTime ? kStreamUnroll : tu.unroll[0];
    with_split(!kTime && csr.nbr_split != nullptr, [&](auto S) {
      with_unroll(u, [&](auto U) {
        if constexpr (!kTime || (decltype(U)::value == kStreamUnroll && !decltype(S)::value))
          k_warp<Sink, kTime, decltype(U)::value, decltype(S)::value><<<grid, 256, 0, st>>>(
              csr, lists + starts[1], counts[1], ctr, sink, d_tables + 256 * kTableWarp, at,
              tu.hash_factor[0]);
      });
    });
    launches++;
  }
  if (counts[2] && (mask & 4u)) {
    const uint32_t cap = kBlockCap;
    const uint32_t hf = fit_hash_factor(tu.hash_factor[1], cap);
    const uint32_t nb = hf * cap;
    const size_t smem = block_stage_bytes(cap, nb);
    const uint32_t threads = kTime ? 256 : tu.block_threads;
    const uint32_t u = kTime ? kStreamUnroll : tu.unroll[1];
    with_split(!kTime && csr.nbr_split != nullptr, [&](auto S) {
      with_block_threads(threads, [&](auto T) {
        with_unroll(u, [&](auto U) {
          constexpr int kT = decltype(T)::value, kU = decltype(U)::value;
          constexpr bool kS = decltype(S)::value;
          if constexpr (!kTime || (kT == 256 && kU == kStreamUnroll && !kS)) {
            STC_CUDA(cudaFuncSetAttribute(k_block<kT, Sink, kTime, kU, kS>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
            const uint32_t grid = std::min<uint32_t>(counts[2], kSMs * 8);
            k_block<kT, Sink, kTime, kU, kS><<<grid, kT, smem, st>>>(
                csr, lists + starts[2], counts[2], cap, nb, hf, ctr + C_WORK + 0, ctr, sink,
                d_tables + 256 * kTableBlock, at, kTableBlock, nullptr, 0);
          }
        });
      });
    });
    launches++;
  }
  if (counts[3] && (mask & 8u)) {
    // Capacity: the class's largest list rounded up to a power of two.
    uint32_t cap = kBlockCap;
    while (cap < std::min<uint32_t>(max_fdeg, kLargeCap)) cap <<= 1;
    const uint32_t hf = fit_hash_factor(tu.hash_factor[2], cap);
    const uint32_t nb = hf * cap;
    const size_t smem = block_stage_bytes(cap, nb);
    const uint32_t u = kTime ? kStreamUnroll : tu.unroll[2];
    with_split(!kTime && csr.nbr_split != nullptr, [&](auto S) {
      with_unroll(u, [&](auto U) {
        constexpr int kU = decltype(U)::value;
        constexpr bool kS = decltype(S)::value;
        if constexpr (!kTime || (kU == kStreamUnroll && !kS)) {
          STC_CUDA(cudaFuncSetAttribute(k_block<512, Sink, kTime, kU, kS>,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
          const uint32_t grid = std::min<uint32_t>(counts[3], kSMs * 2);
          k_block<512, Sink, kTime, kU, kS><<<grid, 512, smem, st>>>(
              csr, lists + starts[3], counts[3], cap, nb, hf, ctr + C_WORK + 1, ctr, sink,
              d_tables + 256 * kTableLarge, at, kTableLarge, nullptr, 0);
        }
      });
    });
    launches++;
  }
  if (counts[4] && (mask & 16u)) {
    const uint32_t grid = std::min<uint32_t>(counts[4], kSMs * 2);
    k_giant<512, Sink, kTime><<<grid, 512, 0, st>>>(csr, lists + starts[4], counts[4],
                                                     ctr + C_WORK + 2, ctr, sink,
                                                     d_tables + 256 * kTableGiant, at, nullptr, 0);
    launches++;
  }
}

// ------------------------------------------------------- head side ----
// Arcs whose dispatch cell says STC_STRATEGY_HEAD are counted from their
// head.  For the arc u -> v, the third vertex w of a triangle lies in
// A' = the part of N+(u) after v and in B = N+(v).  The tail side (the
// kernels above) stages N+(u) and streams B; the head side stages N+(v) as
// the shared-memory hash and streams A' through it, so an arc costs |A'|
// probes instead of |B|.  Over a power-law graph in (degree, id) order,
// A' is the shorter list for almost every arc (the reference's hash
// program iterates the shorter of its two lists for the same reason,
// MC/tc_hash_sign_enu.cpp:146-160).
//
// The head side finds each vertex's in-arcs by a sort: every HEAD arc i
// (its index in the CSR) is appended as a key that holds its sign, |A'|, v and
// i (HeadKey; a CTA adds a tile's keys with one atomic, so their order varies
// from run to run; the counts are sums and do not depend on it), a radix sort
// over the vertex bits of the appended keys, their number known on the device
// only, groups each head's in-arcs, and the runs of equal v are its in-arc
// ranges.  Head vertices are classed by |N+(v)|, the list they stage: warp
// (<= 128), block (<= 1024) and large (<= 4095), the lists longer than the
// warp class's inside the bitmap's window making a fourth class.  A work item
// is a piece of one head's run that does not cross a multiple of its class's
// item size (a hub with millions of in-arcs becomes thousands of items, each
// staging its small N+(v) again), so no warp or CTA is left with one huge
// run.  In the hash classes each in-arc is one "arc" of the staged tile with
// extent [i + 1, end of u's list), its sign s(u, v), strategy HASH: the
// stream pass then probes hash keys that carry s(v, w) with signed heads that
// carry s(u, w).
constexpr uint32_t kHeadMaxB = kLargeCap - 1;  // |N+(v)| of a HEAD arc: bucket <= 12
static_assert(32 - __builtin_clz(kHeadMaxB) == 12 && 32 - __builtin_clz(kHeadMaxB + 1) == 13,
              "HEAD cells (bucket |B| <= 12) are exactly the arcs whose head fits the large class");
constexpr int kHeadClasses = 5;
constexpr uint32_t kHeadBits = 3;   // the bitmap classes (k_head_bits): ranks streamed whole,
constexpr uint32_t kHeadShort = 4;  // or as their low 16 bits
// A warp's item; small, because hubs with short lists own thousands of in-arcs
// (counting an RMAT graph of 1.6 M edges took 534 us at 2,048, 415 at 512, 378 at 256, 368 at 128).
constexpr uint32_t kHeadItemMin = 256;

// In-arcs per work item of head class c (powers of two).
__host__ __device__ __forceinline__ uint32_t head_item(uint32_t c) {
  return c == 0 ? kHeadItemMin : c == 2 ? 16384u : 8192u;  // (both bitmap classes: 8,192)
}

// Table class of a list of d arcs (tiny lists use the warp class's table).
__device__ __forceinline__ uint32_t table_class(uint32_t d) {
  return d <= kWarpCap ? kTableWarp : d <= kBlockCap ? kTableBlock
                                    : d <= kLargeCap ? kTableLarge : kTableGiant;
}
// Head class of a head vertex with d = |N+(v)| in [1, kHeadMaxB].
__device__ __forceinline__ uint32_t head_class(uint32_t d) {
  return d <= kWarpCap ? 0u : d <= kBlockCap ? 1u : 2u;
}

// Ranks a bitmap covers, two bits each, and the shortest |N+(v)| that is worth
// a CTA and a bitmap of its own.  The wide window takes 64 KB (two CTAs of 512
// threads and an L1 for the stream share an SM); at RMAT scale 24 the top
// 2^18 ranks are the heads of 90% of the arcs and 97% of the probes, and the
// heads below keep the hash.  In the short window, 16 KB, a rank's low 16 bits
// are enough, so it streams 16-bit heads: half the bytes for the 83% of the
// probes whose heads it holds there.  Its CTAs are small, so it takes lists
// down to 33 entries from the warp class's hash (128-graph batch: 22.2 ms at
// 129 entries, 19.5 at 65, 19.4 at 33, 19.8 at 9).
constexpr uint32_t kBitsWindow = 1u << 18;
constexpr uint32_t kShortWindow = 1u << 16;
constexpr uint32_t kBitsMinB = kWarpCap, kShortMinB = 32;
constexpr int kBitsThreads = 512, kBitsCtas = 2;  // wide window; CTAs per SM
constexpr int kShortThreads = 128, kShortCtas = 10;

// Which head vertices take the bitmap: v's list and every A' of its in-arcs
// lie in (v, last rank of v's graph], so the bitmap, indexed by the low bits
// of the rank, holds them without collision when that range is at most a
// window long (`window` 0: no bitmap).
struct BitsRule {
  uint32_t window;
  uint32_t n;
  const uint64_t* gbase;  // G + 1 rank boundaries of a batch, or null
  uint32_t G;
  __device__ __forceinline__ uint32_t head_class_of(uint32_t v, uint32_t d) const {
    if (d > min(kBitsMinB, kShortMinB) && window) {
      uint32_t end = n;
      if (gbase) {
        uint32_t lo = 0, hi = G;
        while (hi - lo > 1) {
          const uint32_t mid = (lo + hi) >> 1;
          if (gbase[mid] <= v) lo = mid; else hi = mid;
        }
        end = (uint32_t)gbase[lo + 1];
      }
      if (end - v <= kShortWindow && d > kShortMinB) return kHeadShort;
      if (end - v <= window && d > kBitsMinB) return kHeadBits;
    }
    return head_class(d);
  }
};

// A HEAD arc's sort key: the arc index i in the low ibits, then v (vbits),
// then |A'| in the bits left below the sign in bit 63 (at most 31).  An |A'|
// that its field cannot hold is stored as all ones and the arc's list end
// is looked up in `aend` instead.  With the extent in the key, a work item
// reads its in-arcs with one coalesced load each: gathering list ends and
// signs by arc index cost two 32-byte sectors and a dependent latency an
// in-arc.
struct HeadKey {
  uint32_t ibits, vbits, amax;
  static HeadKey of(uint32_t n, uint64_t m) {
    HeadKey f;
    f.ibits = std::max<uint32_t>(1, bit_width64(m - 1));
    f.vbits = std::max<uint32_t>(1, bit_width64(n - 1));
    f.amax = (1u << std::min<uint32_t>(31, 63 - f.ibits - f.vbits)) - 1;
    return f;
  }
  __device__ __forceinline__ uint64_t pack(uint32_t v, uint64_t i, uint32_t alen, bool neg) const {
    return ((uint64_t)neg << 63) | ((uint64_t)min(alen, amax) << (ibits + vbits)) |
           ((uint64_t)v << ibits) | i;
  }
  __device__ __forceinline__ uint32_t vertex(uint64_t k) const {
    return (uint32_t)(k >> ibits) & ((1u << vbits) - 1);
  }
  __device__ __forceinline__ uint32_t arc(uint64_t k) const {
    return (uint32_t)(k & ((1ull << ibits) - 1));
  }
  // |A'|, or amax when it did not fit.
  __device__ __forceinline__ uint32_t alen(uint64_t k) const {
    return (uint32_t)((k & ~(1ull << 63)) >> (ibits + vbits));
  }
};

// The work items (first entries) of the head classes, in three arrays of
// `cap` words, two of them filled from both ends: classes 0 and 1 from the
// front and the back of the first, 2 and 3 likewise in the second, 4 in the
// third.  A head has one class, so the two lists of an array never meet, and
// no counting pass is needed.
struct HeadLists {
  uint32_t* base;
  uint32_t cap;
  __device__ __forceinline__ uint32_t& at(uint32_t c, uint32_t pos) const {
    return base[(size_t)(c >> 1) * cap + (c & 1 ? cap - 1 - pos : pos)];
  }
};

struct HeadArcs {
  const uint64_t* __restrict__ keys;  // sorted by v (HeadKey)
  const uint32_t* __restrict__ aend;  // list end of an arc whose |A'| did not fit its key
  const uint32_t* __restrict__ end;   // per head vertex: one past its last in-arc entry
  const uint32_t* __restrict__ asrc;  // per arc: its tail (timing recorder only)
  HeadKey fmt;
  HeadLists lists;
  // Work item starting at entry j0 of head class c: its head and its end.
  __device__ __forceinline__ void item(uint32_t j0, uint32_t c, uint32_t& v, uint32_t& j1) const {
    v = fmt.vertex(keys[j0]);
    j1 = min(end[v], (j0 | (head_item(c) - 1)) + 1);
  }
  // A' of the in-arc with this key.
  __device__ __forceinline__ void extent(uint64_t key, uint32_t& lo, uint32_t& hi) const {
    const uint32_t i = fmt.arc(key), al = fmt.alen(key);
    lo = i + 1;
    hi = al == fmt.amax ? aend[i] : lo + al;  // > lo: a HEAD arc has a non-empty A'
  }
};

// An arc counted by one thread: the entries of the shorter of its lists
// A' = [i + 1, i + 1 + alen) and B = [vb, vb + blen), searched in the longer
// one from the last hit on; hit(negative edges) per triangle.
template <class Hit>
__device__ __forceinline__ void short_arc(const Csr& g, uint32_t i, uint32_t alen, uint32_t vb,
                                          uint32_t blen, uint32_t nuv, Hit hit) {
  const bool swap = alen > blen;
  const uint32_t s0 = swap ? vb : i + 1, l0 = swap ? i + 1 : vb;
  const uint32_t sn = swap ? blen : alen, ln = swap ? alen : blen;
  const uint32_t* l = g.nbr + l0;
  uint32_t pos = 0;
  for (uint32_t k = 0; k < sn; k++) {
    const uint32_t x = g.nbr[s0 + k];
    pos += lower_bound(l + pos, ln - pos, x);
    if (pos >= ln) return;
    if (l[pos] == x) {
      hit(nuv + (g.sgn[s0 + k] < 0) + (g.sgn[l0 + pos] < 0));
      pos++;
    }
  }
}
// The longest shorter list of an arc counted that way: staging a list for it
// costs more than so many searches (128-graph batch: 19.4 ms without, 16.3
// with lists up to 4, 15.7 up to 8, 15.9 up to 16, 16.3 up to 32; the skewed
// workload 19.2 -> 17.4 ms from 8 on).
constexpr uint32_t kShortArc = 8;

// Where k_head_keys's short arcs are counted.  Totals add up per thread.  A
// batch adds up per warp while the warp's arcs stay in one graph, whose rank
// range it keeps; a warp whose arcs of a tile span graphs hands over hit by
// hit.  Per-vertex counts go to the tail hit by hit.
template <class Sink>
struct ShortCounts {
  static constexpr bool kGraph = Sink::kKeyed;
  TypeCounts tc;
  uint32_t graph = 0, lo = 1, hi = 0;  // the warp's graph and its ranks [lo, hi)
  bool spans = false;
  // The warp's arcs of a tile have tails in [first, last].
  __device__ __forceinline__ void tile(const Sink& sink, uint32_t first, uint32_t last) {
    if constexpr (kGraph) {
      if (first < lo || first >= hi) {
        flush(sink);
        graph = sink.graph_of(first);
        lo = (uint32_t)sink.gbase[graph];
        hi = (uint32_t)sink.gbase[graph + 1];
      }
      spans = last >= hi;
    }
  }
  __device__ __forceinline__ void hit(const Sink& sink, uint32_t u, uint32_t neg) {
    if constexpr (Sink::kPerArc) {
      sink.add(u, neg);
    } else if (kGraph && spans) {
      if constexpr (kGraph) atomicAdd(sink.gcounts + 4ull * sink.graph_of(u) + (3 - neg), 1ull);
    } else {
      tc.add(neg);
    }
  }
  __device__ __forceinline__ void flush(const Sink& sink) {
    if constexpr (kGraph) {
      unsigned long long c[4];
#pragma unroll
      for (int k = 0; k < 4; k++) c[k] = warp_sum(tc.c[k]);
      if (lane_id() == 0) sink.put_key(graph, c);
      tc = TypeCounts{};
    }
  }
};

// Appends the keys of the HEAD arcs (count in ctr[C_HEAD_NKEYS]), records
// the list end of each HEAD arc whose |A'| its key cannot hold, and sets
// need[u] = 1 for each tail u with an arc left to the tail side (the array
// starts at 0; tails without such arcs are not staged there).  `range` (a
// sharded count) keeps only tails in [range[0], range[1]).  With kBytes it
// also adds up the algorithmic bytes of every arc (arc_bytes), whose inputs
// it reads anyway: a pass of its own took 0.82 ms at RMAT scale 24.
// A CTA appends a tile of 1,024 arcs with one atomic; with one per warp and
// load the 8 M atomics on the one counter took 6.8 ms at RMAT scale 24.
// With kShort, an arc that is not HEAD and whose shorter list has at most
// kShortArc entries is counted on the spot, by its thread: its extents are at
// hand, and no list is classified, queued or staged for it.
template <class Sink, bool kBytes, bool kShort>
__global__ void __launch_bounds__(256) k_head_keys(Csr g, const uint32_t* __restrict__ asrc,
                                                   const uint32_t* __restrict__ fdeg, uint64_t m,
                                                   const unsigned long long* __restrict__ m_dev,
                                                   const uint8_t* __restrict__ gtables,
                                                   const unsigned long long* __restrict__ range,
                                                   HeadKey fmt, uint64_t* __restrict__ keys,
                                                   uint32_t* __restrict__ aend,
                                                   uint8_t* __restrict__ need,
                                                   unsigned long long* __restrict__ ctr, Sink sink) {
  constexpr int kItems = 4;  // arcs per lane with their gathers in flight together
  constexpr int kWarps = 8;
  __shared__ uint8_t tab[kTableBytes];
  __shared__ uint32_t wcnt[2][kWarps];  // alternating tiles
  __shared__ uint32_t tbase[2];
  if (device_failed(ctr + C_ERROR)) return;  // no keys, so no head-side work
  if (m_dev) m = min(m, (uint64_t)*m_dev);  // m a capacity, *m_dev the arc count
  for (uint32_t i = threadIdx.x; i < kTableBytes; i += blockDim.x) tab[i] = gtables[i];
  __syncthreads();
  const uint32_t r0 = range ? (uint32_t)range[0] : 0u;
  const uint32_t r1 = range ? (uint32_t)range[1] : 0xFFFFFFFFu;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  unsigned long long bytes = 0, probe = 0;
  ShortCounts<Sink> sc;
  uint32_t flip = 0;
  for (uint64_t tile = (uint64_t)blockIdx.x * (256 * kItems); tile < m;
       tile += (uint64_t)gridDim.x * (256 * kItems), flip ^= 1) {
    const uint64_t base = tile + warp * (32 * kItems) + lane;
    uint32_t u[kItems], v[kItems], blen[kItems];
    uint32_t ub[kItems], ue[kItems], neg = 0;
#pragma unroll
    for (int q = 0; q < kItems; q++) {
      const uint64_t i = base + 32 * q;
      u[q] = i < m ? asrc[i] : 0u;
      v[q] = i < m ? g.nbr[i] : 0u;
      neg |= (i < m && g.sgn[i] < 0 ? 1u : 0u) << q;
    }
#pragma unroll
    for (int q = 0; q < kItems; q++) {
      const uint64_t i = base + 32 * q;
      ub[q] = i < m ? (uint32_t)g.off[u[q]] : 0;
      ue[q] = i < m ? (uint32_t)g.off[u[q] + 1] : 0;
      blen[q] = i < m ? fdeg[v[q]] : 0u;
    }
    uint32_t heads = 0, mine = 0, total = 0;  // HEAD flags; keys of the lanes below; of the warp
    uint32_t shorts = 0;                      // arcs counted here
#pragma unroll
    for (int q = 0; q < kItems; q++) {
      const uint64_t i = base + 32 * q;
      bool head = false;
      if (i < m) {
        const uint32_t alen = ue[q] - (uint32_t)i - 1, d = ue[q] - ub[q];
        if (kBytes) {
          bytes += 5ull * d + 5ull * blen[q] + 25ull;
          probe += 5ull * min(alen, blen[q]) + 30ull;
        }
        if (alen && blen[q] && u[q] >= r0 && u[q] < r1) {
          head = tab[256 * table_class(d) + 16 * size_bucket(alen) + size_bucket(blen[q])] ==
                 STC_STRATEGY_HEAD;
          if (!head) {
            if (kShort && min(alen, blen[q]) <= kShortArc) shorts |= 1u << q;
            else need[u[q]] = 1;  // u keeps an arc for the tail side
          }
        }
      }
      const unsigned hb = __ballot_sync(kFull, head);
      heads |= (uint32_t)head << q;
      mine += __popc(hb & lanemask_lt());
      total += __popc(hb);
    }
    if (lane == 0) wcnt[flip][warp] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t run = 0;
      for (int w = 0; w < kWarps; w++) {
        const uint32_t c = wcnt[flip][w];
        wcnt[flip][w] = run;
        run += c;
      }
      tbase[flip] = run ? (uint32_t)atomicAdd(ctr + C_HEAD_NKEYS, (unsigned long long)run) : 0u;
    }
    uint32_t vb[kItems];
    if (kShort) {
#pragma unroll
      for (int q = 0; q < kItems; q++) vb[q] = (shorts >> q) & 1u ? (uint32_t)g.off[v[q]] : 0u;
    }
    __syncthreads();
    // The keys of one lane in a row: any order within the tile will do.
    uint32_t at = tbase[flip] + wcnt[flip][warp] + mine;
#pragma unroll
    for (int q = 0; q < kItems; q++) {
      const uint64_t i = base + 32 * q;
      if ((heads >> q) & 1u) {
        const uint32_t alen = ue[q] - (uint32_t)i - 1;
        keys[at++] = fmt.pack(v[q], i, alen, (neg >> q) & 1u);
        if (alen >= fmt.amax) aend[i] = ue[q];
      }
    }
    if (kShort && __any_sync(kFull, shorts != 0)) {
      if (ShortCounts<Sink>::kGraph) {
        const uint32_t first = __shfl_sync(kFull, u[0], 0);
        uint32_t last = 0;
#pragma unroll
        for (int q = 0; q < kItems; q++) last = max(last, u[q]);  // past the end: 0
        sc.tile(sink, first, __reduce_max_sync(kFull, last));
      }
#pragma unroll
      for (int q = 0; q < kItems; q++) {
        if (!((shorts >> q) & 1u)) continue;
        const uint32_t i = (uint32_t)(base + 32 * q), tail = u[q];
        short_arc(g, i, ue[q] - i - 1, vb[q], blen[q], (neg >> q) & 1u,
                  [&](uint32_t n) { sc.hit(sink, tail, n); });
      }
    }
  }
  if (kShort) {
    if (ShortCounts<Sink>::kGraph) sc.flush(sink);
    else if (!Sink::kPerVertex) flush_counts<256>(sc.tc, ctr);
  }
  if (kBytes) {
    bytes = warp_sum(bytes);
    probe = warp_sum(probe);
    if (lane == 0 && bytes) {
      atomicAdd(ctr + C_ALG_BYTES, bytes);
      atomicAdd(ctr + C_PROBE_BYTES, probe);
    }
  }
}

// Work items in the sorted keys: an entry starts one where its head's run
// starts or where it is a multiple of its class's item size.  Appends each
// item's first entry to its class list (through shared memory, one atomic
// per class and tile) and records the end of every run.
constexpr int kItemTile = 2048;

__global__ void __launch_bounds__(256) k_head_items(const uint64_t* __restrict__ keys,
                                                    const uint64_t* __restrict__ off, HeadKey fmt,
                                                    BitsRule rule, HeadLists lists,
                                                    uint32_t* __restrict__ end,
                                                    unsigned long long* __restrict__ ctr) {
  constexpr int kPer = kItemTile / 256;
  __shared__ uint32_t found[kItemTile];  // first entries, by class: cnt[c] from start[c]
  __shared__ uint32_t cnt[kHeadClasses], start[kHeadClasses], gbase[kHeadClasses];
  if (device_failed(ctr + C_ERROR)) return;  // no items
  const uint64_t m = ctr[C_HEAD_NKEYS];
  for (uint64_t tile = (uint64_t)blockIdx.x * kItemTile; tile < m;
       tile += (uint64_t)gridDim.x * kItemTile) {
    if (threadIdx.x < kHeadClasses) cnt[threadIdx.x] = 0;
    __syncthreads();
    uint32_t cls = 0xFFFFFFFFu;  // four bits an entry; 15: starts no item
    uint32_t pos[kPer];
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      const uint64_t j = tile + q * 256 + threadIdx.x;
      pos[q] = 0;
      if (j >= m) continue;
      const uint32_t v = fmt.vertex(keys[j]);
      const bool run = j == 0 || fmt.vertex(keys[j - 1]) != v;
      if (j + 1 == m || fmt.vertex(keys[j + 1]) != v) end[v] = (uint32_t)(j + 1);
      if (run || (j & (kHeadItemMin - 1)) == 0) {
        const uint32_t hc = rule.head_class_of(v, (uint32_t)(off[v + 1] - off[v]));
        if (run || (j & (head_item(hc) - 1)) == 0) {
          cls ^= (15u ^ hc) << (4 * q);
          pos[q] = atomicAdd(&cnt[hc], 1u);
        }
      }
    }
    __syncthreads();
    if (threadIdx.x < kHeadClasses) {
      uint32_t s = 0;
      for (uint32_t c = 0; c < threadIdx.x; c++) s += cnt[c];
      start[threadIdx.x] = s;
      const uint32_t k = cnt[threadIdx.x];
      gbase[threadIdx.x] =
          k ? (uint32_t)atomicAdd(ctr + C_HEAD_COUNT + threadIdx.x, (unsigned long long)k) : 0u;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPer; q++) {
      const uint32_t c = (cls >> (4 * q)) & 15u;
      if (c < kHeadClasses) found[start[c] + pos[q]] = (uint32_t)(tile + q * 256 + threadIdx.x);
    }
    __syncthreads();
    for (uint32_t c = 0; c < kHeadClasses; c++)
      for (uint32_t p = threadIdx.x; p < cnt[c]; p += 256) lists.at(c, gbase[c] + p) = found[start[c] + p];
    __syncthreads();
  }
}

// N+(v) (d entries from vb) as the staged hash of a team of TS threads.
template <int TS, class Sync>
__device__ __forceinline__ void stage_hash(const Csr& g, uint64_t vb, uint32_t d, uint32_t t,
                                           const StageMem& m, const Geo& geo, Sync sync) {
  for (uint32_t i = t; i < 2 * geo.nb; i += TS) m.hk[i] = kEmpty;
  sync();
  for (uint32_t i = t; i < d; i += TS) {
    const uint32_t x = g.nbr[vb + i];
    const uint32_t key = (x << 1) | (uint32_t)(g.sgn[vb + i] < 0);
    uint32_t b = hash_slot(x, geo.shift);
    while (atomicCAS(&m.hk[2 * b], kEmpty, key) != kEmpty &&
           atomicCAS(&m.hk[2 * b + 1], kEmpty, key) != kEmpty)
      b = (b + 1) & (geo.nb - 1);
  }
  sync();
}

// In-arcs [j0, j0 + tn) of a head vertex as the arcs of the staged tile.
template <int TS, bool kArc, class Sync>
__device__ __forceinline__ void stage_in_arcs(const Csr& g, const HeadArcs& h, uint32_t j0,
                                              uint32_t tn, uint32_t t, const StageMem& m,
                                              Sync sync) {
  for (uint32_t k = t; k < tn; k += TS) {
    const uint64_t key = h.keys[j0 + k];
    h.extent(key, m.lo[k], m.hi[k]);
    m.s[k] = (key >> 63) ? (int8_t)-1 : (int8_t)1;
    m.st[k] = STC_STRATEGY_HASH;
    if (kArc) m.a[k] = m.sp[k] = 0;
  }
  sync();
}

// Timing recorder, head side: each in-arc of the tile alone on one warp,
// timed and charged as a streamed arc is; its cell is that of the arc
// u -> v (class of N+(u), bucket |A'|, bucket |B| = |N+(v)|).
__device__ __forceinline__ void timed_head_pass(const Csr& g, const HeadArcs& h, const StageMem& m,
                                                uint32_t tn, uint32_t dv, uint32_t warp,
                                                uint32_t warps, uint32_t lane, const Geo& geo,
                                                PackedCounts& pc, TypeCounts& tc,
                                                const ArcTimes& at) {
  for (uint32_t k = warp; k < tn; k += warps) {
    const uint32_t lo = m.lo[k], hi = m.hi[k];
    __syncwarp();
    const long long t0 = clock_after(0);
    arc_stream(g, m, tn, k, lane, geo, pc);
    unsigned dt = __reduce_max_sync(kFull, (unsigned)(clock_after(pc.w) - t0));
    const uint32_t chunks = ((hi + 3) >> 2) - (lo >> 2);
    dt = (unsigned)((unsigned long long)dt * chunks / (32ull * ((chunks + 31) >> 5)));
    pc.drain(tc);
    if (lane == 0) {
      const uint32_t u = h.asrc[lo - 1];
      record_arc(at, table_class((uint32_t)(hi - g.off[u])), hi - lo, dv, max(dt, 1u));
    }
  }
}

// Head vertices of the warp class: one warp per vertex from a dynamic
// queue, N+(v) and up to kWarpCap in-arcs at a time staged in the warp's
// slice of shared memory.
template <class Sink, bool kTime, int U>
__global__ void __launch_bounds__(256) k_head_warp(Csr g, HeadArcs h,
                                                   unsigned long long* __restrict__ ctr, Sink sink,
                                                   ArcTimes at, uint32_t hf) {
  constexpr bool kVC = Sink::kKeyed, kArc = Sink::kPerArc;
  constexpr int kWarps = 8;
  __shared__ __align__(16) unsigned char smem[kWarps * kWarpStageBytes];
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  const StageMem m = StageMem::carve(smem + w * kWarpStageBytes, kWarpCap, kWarpBuckets);
  const uint32_t cnt = (uint32_t)ctr[C_HEAD_COUNT + 0];
  TypeCounts tc;
  // Per-key counts (a sink that reports per graph): a warp's items come in
  // increasing order of their heads, so the counts of one key are added up
  // and handed to the sink once, when the key changes.
  uint32_t cur = 0xFFFFFFFFu;
  auto flush = [&]() {
    if constexpr (kVC) {
      if (cur == 0xFFFFFFFFu) return;
      unsigned long long s[4];
#pragma unroll
      for (int k = 0; k < 4; k++) s[k] = warp_sum(tc.c[k]);
      if (lane == 0) sink.put_key(cur, s);
      tc = TypeCounts{};
    }
  };
  while (true) {
    uint32_t item = 0;
    if (lane == 0) item = (uint32_t)atomicAdd(ctr + C_HEAD_QUEUE + 0, 1ull);
    item = __shfl_sync(kFull, item, 0);
    if (item >= cnt) break;
    uint32_t v, j1;
    const uint32_t j00 = h.lists.at(0, item);
    h.item(j00, 0, v, j1);
    const uint64_t vb = g.off[v];
    const uint32_t d = (uint32_t)(g.off[v + 1] - vb);
    if (d > kWarpCap) {  // uniform over the warp
      if (lane == 0) atomicExch(ctr + C_ERROR, kErrStageCapacity);
      continue;
    }
    if constexpr (kVC) {
      const uint32_t key = sink.key(v);
      if (key != cur) {
        flush();
        cur = key;
      }
    }
    const Geo geo = Geo::of(d, kWarpBuckets, hf);
    stage_hash<32>(g, vb, d, lane, m, geo, WarpSync{});
    TypeCounts& out = tc;
    PackedCounts pc;
    for (uint32_t j0 = j00; j0 < j1; j0 += kWarpCap) {
      const uint32_t tn = min(kWarpCap, j1 - j0);
      stage_in_arcs<32, kArc>(g, h, j0, tn, lane, m, WarpSync{});
      if (kTime) {
        timed_head_pass(g, h, m, tn, d, 0, 1, lane, geo, pc, out, at);
      } else {
        warp_chunk_scan<true>(m, tn, lane);
        // U / 2 chunks of 8 entries: U 16-byte loads in flight per lane, as
        // in the tail side (more raise the registers above 64 and cost
        // this kernel a CTA per SM).
        stream_pass_keyed<(U > 1 ? U / 2 : 1), kArc>(g, m, tn, 0, 1, lane, geo, out, nullptr);
      }
      __syncwarp();
      if constexpr (kArc) {
        for (uint32_t k = lane; k < tn; k += 32)
          sink.add_arc(h.asrc[m.lo[k] - 1], m.a[k], m.sp[k]);
        __syncwarp();
      }
    }
    pc.drain(out);
    __syncwarp();
  }
  flush();
  if (!Sink::kPerVertex) flush_counts<256>(tc, ctr);
}

// Head vertices of the block and large classes: one CTA per vertex from a
// dynamic queue, N+(v) (up to `cap` entries, `nb` buckets) and up to `cap`
// in-arcs at a time staged in dynamic shared memory.
template <int THREADS, class Sink, bool kTime, int U>
__global__ void __launch_bounds__(THREADS) k_head_block(Csr g, HeadArcs h,
                                                        uint32_t hclass, uint32_t cap, uint32_t nb,
                                                        uint32_t hf,
                                                        unsigned long long* __restrict__ ctr,
                                                        Sink sink, ArcTimes at) {
  constexpr bool kVC = Sink::kKeyed, kArc = Sink::kPerArc;
  constexpr uint32_t kWarps = THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t scan_tmp[THREADS / 32 + 2];
  __shared__ uint32_t s_item;
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  const StageMem m = StageMem::carve(smem, cap, nb);
  const uint32_t cnt = (uint32_t)ctr[C_HEAD_COUNT + hclass];
  unsigned long long* queue = ctr + C_HEAD_QUEUE + hclass;
  uint32_t* next = scan_tmp + kWarps + 1;  // the stream's claim counter
  TypeCounts tc;
  // Per-key counts as in k_head_warp, reduced over the CTA at a key change.
  uint32_t cur = 0xFFFFFFFFu;
  auto flush = [&]() {
    if constexpr (kVC) {
      if (cur == 0xFFFFFFFFu) return;
      block_key_flush<THREADS>(tc, cur, sink);
      tc = TypeCounts{};
    }
  };
  while (true) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = (uint32_t)atomicAdd(queue, 1ull);
    __syncthreads();
    const uint32_t item = s_item;
    if (item >= cnt) break;
    uint32_t v, j1;
    const uint32_t j00 = h.lists.at(hclass, item);
    h.item(j00, hclass, v, j1);
    const uint64_t vb = g.off[v];
    const uint32_t d = (uint32_t)(g.off[v + 1] - vb);
    if (d > cap) {  // uniform over the CTA
      if (threadIdx.x == 0) atomicExch(ctr + C_ERROR, kErrStageCapacity);
      continue;
    }
    if constexpr (kVC) {
      const uint32_t key = sink.key(v);  // uniform over the CTA
      if (key != cur) {
        flush();
        cur = key;
      }
    }
    const Geo geo = Geo::of(d, nb, hf);
    stage_hash<THREADS>(g, vb, d, threadIdx.x, m, geo, BlockSync{});
    TypeCounts& out = tc;
    PackedCounts pc;
    for (uint32_t j0 = j00; j0 < j1; j0 += cap) {
      const uint32_t tn = min(cap, j1 - j0);
      // Every warp left the previous tile's stream (barrier at its end), and
      // the staging below passes a barrier before the counter is used.
      if (threadIdx.x == 0) *next = 0;
      stage_in_arcs<THREADS, kArc>(g, h, j0, tn, threadIdx.x, m, BlockSync{});
      if (kTime) {
        timed_head_pass(g, h, m, tn, d, w, kWarps, lane, geo, pc, out, at);
      } else {
        block_chunk_scan<THREADS, true>(m, tn, scan_tmp);
        // U chunks of 8 entries: 2 U 16-byte loads in flight per lane.
        stream_pass_keyed<U, kArc>(g, m, tn, w, kWarps, lane, geo, out, next);
      }
      __syncthreads();
      if constexpr (kArc) {
        for (uint32_t k = threadIdx.x; k < tn; k += THREADS)
          sink.add_arc(h.asrc[m.lo[k] - 1], m.a[k], m.sp[k]);
        __syncthreads();
      }
    }
    pc.drain(out);
  }
  flush();
  if (!Sink::kPerVertex) flush_counts<THREADS>(tc, ctr);
}

// The arcs as the bitmap classes stream them: sign bits, one byte per eight
// arcs (entry e of the group at bit 7 - e, the order in which k_head_bits
// collects its hits), and the low 16 bits of the heads.
struct HeadStream {
  uint8_t* sbits;
  uint16_t* low;
};

__global__ void __launch_bounds__(256) k_head_stream(const uint32_t* __restrict__ nbr,
                                                     const int8_t* __restrict__ sgn, uint64_t m,
                                                     const unsigned long long* __restrict__ m_dev,
                                                     HeadStream hs) {
  if (m_dev) m = min(m, (uint64_t)*m_dev);
  const uint64_t groups = (m + 7) / 8;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < groups; i += stride) {
    const uint2 q = reinterpret_cast<const uint2*>(sgn)[i];
    const uint4 x = reinterpret_cast<const uint4*>(nbr)[2 * i];
    const uint4 y = reinterpret_cast<const uint4*>(nbr)[2 * i + 1];
    // Sign bits at 7, 15, 23, 31; the multiply gathers them at 31..28.
    const uint32_t a = ((q.x >> 7) & 0x01010101u) * 0x80402010u >> 28;
    const uint32_t b = ((q.y >> 7) & 0x01010101u) * 0x80402010u >> 28;
    hs.sbits[i] = (uint8_t)((a << 4) | b);
    reinterpret_cast<uint4*>(hs.low)[i] =
        make_uint4(__byte_perm(x.x, x.y, 0x5410), __byte_perm(x.z, x.w, 0x5410),
                   __byte_perm(y.x, y.y, 0x5410), __byte_perm(y.z, y.w, 0x5410));
  }
}

// Eight consecutive heads by one 32-byte load: with two of 16 bytes a lane,
// each instruction spread over twice the lines it used.
__device__ __forceinline__ void load8(const uint32_t* __restrict__ p, uint32_t (&x)[8]) {
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]),
                 "=r"(x[6]), "=r"(x[7])
               : "l"(p));
}

// Head vertices whose lists fit a bitmap: one CTA per work item from a
// dynamic queue.  N+(v) is staged as a bitmap over the ranks (mod the
// window), two bits per rank, 16 ranks per 32-bit word: for rank x, the
// bit at x & 31 says that x is in N+(v) with a positive sign, the bit at
// (x & 31) ^ 16 that it is with a negative one.  Rotating the word right by x
// brings the two to bits 0 and 16, so a streamed entry costs one 4-byte
// shared load and five integer instructions (address: shift and mask;
// rotate, mask, append to the lane's hit masks), against about 18 and an
// 8-byte load for the hash, and staging an entry is one shared atomic.
// Entries outside an arc's extent alias some other rank's bits; their hits
// are masked out per chunk.
//
// Warps take 32 in-arcs at a time: each lane holds one arc's extent, and the
// arcs' aligned 8-entry chunks form one sequence.  The arc of a lane's chunk
// follows from a bit mask of the arc starts inside the warp's 32 chunks (one
// or-reduction, as every arc has at least one chunk) and its extent from
// shuffles, so there is no tile in shared memory and no CTA barrier between
// tiles.  The eight hits of a chunk are classified together: three
// population counts of the hit masks against the chunk's sign byte.
//
// A CTA waits as little as its two barriers an item allow: the next item's
// four dependent loads run under this item's stream, the old list's bits go
// off in the step that sets the new ones, a claim's keys are loaded while the
// claim before is streamed, and small items are claimed in small pieces.
//
// RMAT scale 24 (97% of the 41.8 G probes): 28.8 ms for the two windows (20.5
// the short one, at 2.9 TB/s of DRAM, 8.3 the wide one, at 3.2), against 78.8
// ms of hash probes for the same heads.  At scale 22 the short one takes 4.5 ms
// for 230 M warp loads of the bitmap and is bound by the shared-memory pipe (76%
// busy, 2.8 wavefronts a load, ranks being random over the banks) and the integer
// pipe (75%); DRAM is at a tenth of its rate there.  One 32-byte load a chunk instead
// of two of 16 took 3.4 ms off, the short window 1.6, its CTAs of 128
// threads, ten an SM, instead of 512, two an SM, 3.8 (fewer warps wait at an
// item's barriers; 256 x 5 was 0.4 slower, 128 x 12 2.3); chunks in flight 1,
// 3 or 4 instead of 2 were slower.
//
// kShort: the heads of the short window, streamed as 16-bit ranks.
template <int THREADS, bool kShort, class Sink>
__global__ void __launch_bounds__(THREADS, kShort ? kShortCtas : kBitsCtas) k_head_bits(
    Csr g, HeadArcs h, HeadStream hs, unsigned long long* __restrict__ ctr, Sink sink) {
  constexpr uint32_t kClass = kShort ? kHeadShort : kHeadBits;
  constexpr uint32_t kWords = (kShort ? kShortWindow : kBitsWindow) / 16;
  constexpr bool kVC = Sink::kKeyed, kArc = Sink::kPerArc;
  constexpr uint32_t kWarps = THREADS / 32;
  constexpr int U = 2;  // chunks in flight per lane
  constexpr uint32_t kDrainRounds = 255 / (8 * U);  // 8-bit fields, 8 adds a chunk at most
  extern __shared__ __align__(16) uint32_t bm[];  // kWords
  struct Item {
    uint32_t v, j0, arcs, vb, d;  // arcs 0: no more items
  };
  __shared__ Item s_item[2];
  __shared__ uint32_t s_next;
  __shared__ uint32_t arc_counts[kArc ? kWarps : 1][2][32];  // of a warp's 32 in-arcs
  const uint32_t lane = lane_id(), le = lanemask_lt() | (1u << lane);
  const uint32_t cnt = (uint32_t)ctr[C_HEAD_COUNT + kClass];
  TypeCounts tc;
  uint32_t cur = 0xFFFFFFFFu;  // per-key counts as in k_head_block
  auto flush = [&]() {
    if constexpr (kVC) {
      if (cur == 0xFFFFFFFFu) return;
      block_key_flush<THREADS>(tc, cur, sink);
      tc = TypeCounts{};
    }
  };
  // Thread 0: the next work item, by four dependent loads.
  auto fetch = [&](Item& it) {
    const uint32_t item = (uint32_t)atomicAdd(ctr + C_HEAD_QUEUE + kClass, 1ull);
    it.arcs = 0;
    if (item >= cnt) return;
    uint32_t j1;
    it.j0 = h.lists.at(kClass, item);
    h.item(it.j0, kClass, it.v, j1);
    it.arcs = j1 - it.j0;
    it.vb = (uint32_t)g.off[it.v];
    it.d = (uint32_t)g.off[it.v + 1] - it.vb;
  };
  // Switches the bits of the list [vb, vb + d) on, or off again.
  auto toggle = [&](uint32_t vb, uint32_t d) {
    for (uint32_t i = threadIdx.x; i < d; i += THREADS) {
      const uint32_t x = g.nbr[vb + i];
      const uint32_t neg = g.sgn[vb + i] < 0;
      atomicXor(&bm[(x >> 4) & (kWords - 1)], 1u << ((x & 31u) ^ (neg << 4)));
    }
  };
  for (uint32_t i = threadIdx.x; i < kWords; i += THREADS) bm[i] = 0;
  if (threadIdx.x == 0) fetch(s_item[0]);
  __syncthreads();
  uint32_t ovb = 0, od = 0, p = 0;  // the list whose bits are on
  while (true) {
    const Item it = s_item[p];
    if (it.arcs == 0) break;
    if constexpr (kVC) {
      const uint32_t key = sink.key(it.v);  // uniform over the CTA
      if (key != cur) {
        flush();
        cur = key;
      }
    }
    // Exclusive ors commute, so the old list's bits go off and the new one's
    // on in one step, whatever the two share.
    toggle(ovb, od);
    toggle(it.vb, it.d);
    ovb = it.vb;
    od = it.d;
    if (threadIdx.x == 0) s_next = 0;
    __syncthreads();
    // The next item's loads run under this item's stream.
    if (threadIdx.x == 0) fetch(s_item[p ^ 1]);
    // In-arcs per claim: up to a lane each, but small items are shared out
    // over all warps, twice over.
    const uint32_t claim = min(32u, max(4u, (it.arcs + 2 * kWarps - 1) / (2 * kWarps)));
    PackedCounts8 p8;
    uint32_t rounds = 0;
    auto take = [&](uint64_t& key) {  // claims the next in-arcs and loads the lane's key
      uint32_t b = 0;
      if (lane == 0) b = atomicAdd(&s_next, claim);
      b = __shfl_sync(kFull, b, 0);
      if (lane < claim && b + lane < it.arcs) key = h.keys[it.j0 + b + lane];
      return b;
    };
    uint64_t nkey = 0;
    uint32_t nb = take(nkey);
    while (nb < it.arcs) {
      const uint32_t b = nb;
      const uint64_t key = nkey;
      nb = take(nkey);  // in flight while this claim is streamed
      // This lane's in-arc: A' extent [lo, hi), its chunks, and in one word the
      // masks of its first and last chunk and 8 * (arc negative).
      uint32_t lo = 0, hi = 1, c = 0;
      if (lane < claim && b + lane < it.arcs) {
        h.extent(key, lo, hi);
        c = ((hi + 7) >> 3) - (lo >> 3);
      }
      const uint32_t arc = (0xFFu >> (lo & 7)) | ((0xFFu << (7 - ((hi - 1) & 7))) & 0xFFu) << 8 |
                           (uint32_t)(key >> 63) << 19;
      const uint32_t inc = warp_inclusive_scan(c);
      const uint32_t start = c ? inc - c : 0xFFFFFFFFu;
      const uint32_t cb = (lo >> 3) - start;  // group index = cb + chunk index
      const uint32_t total = __shfl_sync(kFull, inc, 31);
      uint32_t k0 = 0xFFFFFFFFu;  // arcs started before the round, less one
      uint32_t* ac = arc_counts[kArc ? threadIdx.x >> 5 : 0][0];
      if (kArc) {
        ac[lane] = ac[32 + lane] = 0;
        __syncwarp();
      }
      // Which of the next 32 chunks start an arc.
      uint32_t ahead = __reduce_or_sync(kFull, start < 32u ? 1u << start : 0u);
      for (uint32_t base = 0; base < total; base += 32 * U) {
        uint32_t q[U][kShort ? 4 : 8], sb[U], vm[U], ash[U], ak[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
          const uint32_t w0 = base + 32 * u;
          const uint32_t starts = ahead, rel = start - w0 - 32;
          ahead = __reduce_or_sync(kFull, rel < 32u ? 1u << rel : 0u);
          const uint32_t k = k0 + __popc(starts & le);
          k0 += __popc(starts);
          const uint32_t ci = __shfl_sync(kFull, cb, k) + w0 + lane;
          const uint32_t ka = __shfl_sync(kFull, arc, k);
          vm[u] = 0;
          if (w0 + lane < total) {
            if constexpr (kShort) {
              const uint4 x = reinterpret_cast<const uint4*>(hs.low)[ci];
              q[u][0] = x.x, q[u][1] = x.y, q[u][2] = x.z, q[u][3] = x.w;
            } else {
              load8(g.nbr + 8ull * ci, q[u]);
            }
            sb[u] = hs.sbits[ci];
            // The chunk is its arc's last if the next one starts another.
            const bool first = (starts >> lane) & 1u;
            const bool last = (__funnelshift_r(starts, ahead, 1) >> lane) & 1u;
            vm[u] = (first ? ka & 0xFFu : 0xFFu) &
                    (last || w0 + lane + 1 == total ? (ka >> 8) & 0xFFu : 0xFFu);
            ash[u] = ka >> 16;
            ak[u] = k;
          }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
          if (vm[u] == 0) continue;
          uint32_t acc = 0;  // hits: positive in bits 0-7, negative in bits 16-23
#pragma unroll
          for (uint32_t e = 0; e < 8; e++) {
            const uint32_t x = !kShort ? q[u][e] : e & 1 ? q[u][e / 2] >> 16 : q[u][e / 2];
            const uint32_t w = bm[(x >> 4) & (kWords - 1)];
            acc = 2 * acc + (__funnelshift_r(w, w, x) & 0x10001u);
          }
          acc &= vm[u] * 0x10001u;
          const uint32_t neg = acc & (sb[u] * 0x10001u);
          const uint32_t e2 = __popc(neg >> 16);
          const uint32_t e0 = __popc((acc ^ neg) & 0xFFFFu);
          const uint32_t e1 = __popc(acc) - e0 - e2;
          const uint32_t add = (e0 + (e1 << 8) + (e2 << 16)) << ash[u];
          if (kArc) add_to_arc(add, ac + ak[u], ac + 32 + ak[u]);
          else p8.w += add;
        }
        if (!kArc && ++rounds == kDrainRounds) {
          p8.drain(tc);
          rounds = 0;
        }
      }
      if constexpr (kArc) {
        __syncwarp();
        if (c) sink.add_arc(h.asrc[h.fmt.arc(key)], ac[lane], ac[32 + lane]);
        __syncwarp();
      }
    }
    p8.drain(tc);
    p ^= 1;
    __syncthreads();
  }
  flush();
  if (!Sink::kPerVertex) flush_counts<THREADS>(tc, ctr);
}

// Device buffers of the head-side pass (allocated before any capture).
struct HeadBufs {
  uint64_t* keys = nullptr;
  uint64_t* alt = nullptr;
  uint32_t* aend = nullptr;
  uint32_t* runs = nullptr;  // end of each head's run (n)
  HeadLists lists{};         // the classes' work items
  uint8_t* need = nullptr;   // per tail: it keeps arcs for the tail side
  SortSpace sort_ws;
  HeadStream stream{};       // the arcs as the bitmap classes stream them
};

HeadBufs head_buffers(stc_ctx* c, const DeviceGraph& g) {
  HeadBufs b;
  b.keys = buffer<uint64_t>(c, B_KEYS_A, g.m_fwd);
  b.alt = buffer<uint64_t>(c, B_KEYS_B, g.m_fwd);
  b.aend = buffer<uint32_t>(c, B_HEAD_END, g.m_fwd);
  b.runs = buffer<uint32_t>(c, B_HEAD_RUNS, g.n);
  // Items: at most one per run (a head with an in-arc and a list) plus one
  // per multiple of the smallest item size.
  const size_t items = (size_t)std::min<uint64_t>(g.n, g.m_fwd) + g.m_fwd / kHeadItemMin + 1;
  b.lists.base = buffer<uint32_t>(c, B_HEAD_LIST, 3 * items + (g.n + 3) / 4);
  b.lists.cap = (uint32_t)items;
  b.need = reinterpret_cast<uint8_t*>(b.lists.base + 3 * items);
  b.sort_ws = sort_space(c, g.m_fwd);
  b.stream.low = buffer<uint16_t>(c, B_HEAD_LOW, (g.m_fwd + 7) / 8 * 8);
  b.stream.sbits = buffer<uint8_t>(c, B_SBITS, (g.m_fwd + 7) / 8);
  return b;
}

// Shared-memory limits of the head-class kernels a head-side pass with this
// tuning launches; called before the pass is enqueued (or captured).
template <class Sink, bool kTime>
void prepare_head(const Tuning& tu) {
  const size_t sb =
      block_stage_bytes(kBlockCap, fit_hash_factor(tu.hash_factor[1], kBlockCap) * kBlockCap);
  const size_t sl =
      block_stage_bytes(kLargeCap, fit_hash_factor(tu.hash_factor[2], kLargeCap) * kLargeCap);
  with_block_threads(kTime ? 256 : tu.block_threads, [&](auto T) {
    with_unroll(kTime ? kStreamUnroll : tu.unroll[1], [&](auto U) {
      constexpr int kT = decltype(T)::value, kU = decltype(U)::value;
      if constexpr (!kTime || (kT == 256 && kU == kStreamUnroll))
        STC_CUDA(cudaFuncSetAttribute(k_head_block<kT, Sink, kTime, kU>,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sb));
    });
  });
  with_unroll(kTime ? kStreamUnroll : tu.unroll[2], [&](auto U) {
    constexpr int kU = decltype(U)::value;
    if constexpr (!kTime || kU == kStreamUnroll)
      STC_CUDA(cudaFuncSetAttribute(k_head_block<512, Sink, kTime, kU>,
                                    cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sl));
  });
  if constexpr (!kTime)
    STC_CUDA(cudaFuncSetAttribute(k_head_bits<kBitsThreads, false, Sink>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(kBitsWindow / 4)));
}

// The head-side pass is enqueued on `st` (no host synchronisation) in two
// parts: the keys (before the tail side is classified, which skips the
// tails left without arcs), then the sort, runs, plan and the three
// head-class kernels.  The launch parameters of the block and large classes
// follow the tuning of the tail side's same classes.
template <class Sink>
void enqueue_head_keys(cudaStream_t st, const Csr& csr, const uint32_t* asrc,
                              const uint32_t* fdeg, uint64_t m,
                              const unsigned long long* m_dev, bool bytes, bool short_arcs,
                              const HeadBufs& b, const uint8_t* d_tables,
                              const unsigned long long* range, unsigned long long* ctr,
                              const Sink& sink, int& launches) {
  STC_CUDA(cudaMemsetAsync(ctr + C_HEAD_NKEYS, 0,
                           (C_HEAD_QUEUE + kHeadClasses - C_HEAD_NKEYS) * sizeof(unsigned long long),
                           st));
  STC_CUDA(cudaMemsetAsync(b.need, 0, csr.n, st));
  const uint32_t grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>((m + 1023) / 1024, kSMs * 8));
  const HeadKey fmt = HeadKey::of(csr.n, m);
  auto kernel = bytes ? (short_arcs ? k_head_keys<Sink, true, true> : k_head_keys<Sink, true, false>)
                      : (short_arcs ? k_head_keys<Sink, false, true> : k_head_keys<Sink, false, false>);
  kernel<<<grid, 256, 0, st>>>(csr, asrc, fdeg, m, m_dev, d_tables, range, fmt, b.keys, b.aend,
                               b.need, ctr, sink);
  launches += 1;
}

template <class Sink, bool kTime>
void enqueue_head(cudaStream_t st, const Csr& csr, const uint32_t* asrc, uint64_t m,
                  const unsigned long long* m_dev, const uint64_t* gbase, uint32_t G,
                  const HeadBufs& b, unsigned long long* ctr, const Sink& sink,
                  const ArcTimes& at, const Tuning& tu, int& launches,
                  uint32_t class_mask = 0x3F) {
  const uint32_t n = csr.n;
  const HeadKey fmt = HeadKey::of(n, m);
  const uint64_t* sorted = radix_sort(b.keys, b.alt, m, (int)fmt.ibits,
                                      (int)(fmt.ibits + fmt.vbits), b.sort_ws, ctr + C_ERROR, st, &launches,
                                      ctr + C_HEAD_NKEYS);
  uint32_t* end = b.runs;
  // The recorder times single arcs against a staged hash: no bitmap there.
  const BitsRule rule{kTime ? 0u : kBitsWindow, n, gbase, G};
  const uint32_t tiles = (uint32_t)std::max<uint64_t>(1, (m + kItemTile - 1) / kItemTile);
  k_head_items<<<std::min<uint32_t>(tiles, kSMs * 8), 256, 0, st>>>(sorted, csr.off, fmt, rule,
                                                                    b.lists, end, ctr);
  const HeadArcs h{sorted, b.aend, end, asrc, fmt, b.lists};
  launches += 1;
  const bool wide = kTime || gbase || n > kShortWindow;
  if constexpr (!kTime) {
    if (class_mask & 4u) {
      k_head_stream<<<kSMs * 8, 256, 0, st>>>(csr.nbr, csr.sgn, m, m_dev, b.stream);
      k_head_bits<kShortThreads, true, Sink>
          <<<kSMs * kShortCtas, kShortThreads, kShortWindow / 4, st>>>(csr, h, b.stream, ctr, sink);
      if (wide)
        k_head_bits<kBitsThreads, false, Sink>
            <<<kSMs * kBitsCtas, kBitsThreads, kBitsWindow / 4, st>>>(csr, h, b.stream, ctr, sink);
      launches += wide ? 3 : 2;
    }
  }
  // With every rank inside the window the bitmap takes all lists longer than
  // the warp class's.
  const bool low = kTime || gbase || n > kBitsWindow;
  // Head class c runs with class_mask bit c + 1, as the tail side's class of
  // the same tuning (the autotuner times one class at a time).
  with_unroll(kTime ? kStreamUnroll : tu.unroll[0], [&](auto U) {
    constexpr int kU = decltype(U)::value;
    if constexpr (!kTime || kU == kStreamUnroll)
      if (class_mask & 2u)
        k_head_warp<Sink, kTime, kU><<<kSMs * 4, 256, 0, st>>>(csr, h, ctr, sink, at,
                                                               tu.hash_factor[0]);
  });
  if (low && (class_mask & 4u)) {
    const uint32_t cap = kBlockCap;
    const uint32_t hf = fit_hash_factor(tu.hash_factor[1], cap);
    const uint32_t nb = hf * cap;
    const size_t smem = block_stage_bytes(cap, nb);
    with_block_threads(kTime ? 256 : tu.block_threads, [&](auto T) {
      with_unroll(kTime ? kStreamUnroll : tu.unroll[1], [&](auto U) {
        constexpr int kT = decltype(T)::value, kU = decltype(U)::value;
        if constexpr (!kTime || (kT == 256 && kU == kStreamUnroll)) {
          const uint32_t per_sm = smem <= 110 * 1024 ? 2 : 1;
          k_head_block<kT, Sink, kTime, kU><<<kSMs * per_sm, kT, smem, st>>>(
              csr, h, 1, cap, nb, hf, ctr, sink, at);
        }
      });
    });
  }
  if (low && (class_mask & 8u)) {
    const uint32_t cap = kLargeCap;
    const uint32_t hf = fit_hash_factor(tu.hash_factor[2], cap);
    const uint32_t nb = hf * cap;
    const size_t smem = block_stage_bytes(cap, nb);
    with_unroll(kTime ? kStreamUnroll : tu.unroll[2], [&](auto U) {
      constexpr int kU = decltype(U)::value;
      if constexpr (!kTime || kU == kStreamUnroll)
        k_head_block<512, Sink, kTime, kU><<<kSMs, 512, smem, st>>>(csr, h, 2, cap, nb, hf,
                                                                     ctr, sink, at);
    });
  }
  launches += low ? 3 : 1;
  STC_CUDA(cudaGetLastError());
}

// ------------------------------------------------------- persistent ----
// The persistent engine: the whole count as one sequence without host
// synchronisation, so that it can be captured once in a CUDA graph and
// replayed.  The class lists are planned on the device (k_plan); one
// persistent kernel of 256-thread CTAs then drains two device work queues:
// first the block-class lists, one per CTA at a time; then, with no further
// CTA barriers, each warp takes a warp-class list or 32 tiny lists (one per
// lane) at a time.  Large and giant lists, rare in the small graphs a batch
// holds, keep their own kernels, which read their counts from the plan.
__global__ void k_plan(unsigned long long* __restrict__ ctr, uint32_t* __restrict__ plan) {
  if (threadIdx.x != 0) return;
  uint32_t start = 0;
  for (int c = 0; c < kClasses; c++) {
    const uint32_t cnt = (uint32_t)ctr[C_WORK + c];
    plan[c] = start;
    plan[kPlanCounts + c] = cnt;
    start += cnt;
  }
  plan[kClasses] = start;
  for (int i = 0; i < 8; i++) ctr[C_WORK + i] = 0;  // fill cursors and work queues
  ctr[C_QUEUE_WARP] = 0;
}

constexpr size_t kPersistentSmem =
    StageMem::bytes(kBlockCap, 4 * kBlockCap) > 8 * kWarpStageBytes
        ? StageMem::bytes(kBlockCap, 4 * kBlockCap)
        : 8 * kWarpStageBytes;

template <class Sink>
__global__ void __launch_bounds__(256, 4) k_persistent(Csr g, const uint32_t* __restrict__ lists,
                                                       const uint32_t* __restrict__ plan,
                                                       unsigned long long* __restrict__ ctr, Sink sink,
                                                       const uint8_t* __restrict__ gtables) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint8_t tw[16][16], tb[16][16];
  __shared__ uint32_t scan_tmp[256 / 32 + 2];
  __shared__ uint32_t s_item;
  (&tw[0][0])[threadIdx.x] = gtables[256 * kTableWarp + threadIdx.x];
  (&tb[0][0])[threadIdx.x] = gtables[256 * kTableBlock + threadIdx.x];
  const uint32_t nt = plan[kPlanCounts + 0], nw = plan[kPlanCounts + 1], nb = plan[kPlanCounts + 2];
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  TypeCounts tc;
  // Phase 1: block-class lists, the whole CTA on each.
  const StageMem mb = StageMem::carve(smem, kBlockCap, 4 * kBlockCap);
  while (true) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = (uint32_t)atomicAdd(ctr + C_WORK + 5, 1ull);
    __syncthreads();
    const uint32_t item = s_item;
    if (item >= nb) break;
    block_vertex<256, Sink, false, kStreamUnroll, false>(g, lists[plan[2] + item], kBlockCap,
                                                  4 * kBlockCap, 4, mb, tb, scan_tmp, ctr, sink,
                                                  ArcTimes{nullptr, nullptr}, kTableBlock, tc);
  }
  // Phase 2: warp-granular items.  Every warp of the CTA has left phase 1
  // (the exit above is uniform), so the slices no longer alias mb in use.
  const StageMem mw = StageMem::carve(smem + w * kWarpStageBytes, kWarpCap, kWarpBuckets);
  const uint32_t total = nw + (nt + 31) / 32;
  while (true) {
    uint32_t item = 0;
    if (lane == 0) item = (uint32_t)atomicAdd(ctr + C_QUEUE_WARP, 1ull);
    item = __shfl_sync(kFull, item, 0);
    if (item >= total) break;
    if (item < nw) {
      warp_vertex<Sink, false, kStreamUnroll, false>(g, lists[plan[1] + item], lane, mw, tw, 4, ctr,
                                                     sink,
                                              ArcTimes{nullptr, nullptr}, tc);
    } else {
      const uint32_t idx = (item - nw) * 32 + lane;
      if (idx < nt) tiny_vertex<kTinyMax>(g, lists[plan[0] + idx], sink, tw, tc);
    }
  }
  if (!Sink::kPerVertex) flush_counts<256>(tc, ctr);
}

// The head-side pass of a persistent count: its buffers and the arcs.
struct HeadPlan {
  const HeadBufs* bufs = nullptr;  // null: the tables send no arc to the head side
  const uint32_t* asrc = nullptr;
  const uint32_t* fdeg = nullptr;
  uint64_t m = 0;
  bool bytes = false;       // the key pass adds up the arcs' algorithmic bytes
  bool short_arcs = false;  // ... and counts the short arcs
  const unsigned long long* m_dev = nullptr;  // arc count on the device when m is a capacity
  const uint64_t* gbase = nullptr;  // G + 1 rank boundaries of a batch
  uint32_t G = 0;
  Tuning tuning;
};

// Enqueues the persistent sequence on `st` (no host synchronisation).
template <class Sink>
void enqueue_persistent(cudaStream_t st, const Csr& csr, const ClassBounds& cb, uint32_t* lists,
                        uint32_t* plan, unsigned long long* ctr, const uint8_t* d_tables,
                        const Sink& sink, const HeadPlan& hp, int& launches) {
  const ArcTimes none{nullptr, nullptr};
  const uint8_t* need = nullptr;
  if (hp.bufs) {
    enqueue_head_keys(st, csr, hp.asrc, hp.fdeg, hp.m, hp.m_dev, hp.bytes, hp.short_arcs, *hp.bufs,
                      d_tables, nullptr, ctr, sink, launches);
    need = hp.bufs->need;
  }
  STC_CUDA(cudaMemsetAsync(ctr + C_WORK, 0, 8 * sizeof(uint64_t), st));
  k_classify_count<<<kSMs * 4, 256, 0, st>>>(csr.off, csr.n, cb, ctr, nullptr, need);
  k_plan<<<1, 32, 0, st>>>(ctr, plan);
  k_classify_fill<<<kSMs * 4, 256, 0, st>>>(csr.off, csr.n, cb, lists, plan, ctr, nullptr, need);
  k_persistent<Sink><<<kSMs * 4, 256, kPersistentSmem, st>>>(csr, lists, plan, ctr, sink,
                                                             d_tables);
  k_block<512, Sink, false, kStreamUnroll, false>
      <<<kSMs, 512, StageMem::bytes(kLargeCap, 2 * kLargeCap), st>>>(
      csr, lists, 0, kLargeCap, 2 * kLargeCap, 2, ctr + C_WORK + 6, ctr, sink,
      d_tables + 256 * kTableLarge, none, kTableLarge, plan, 3);
  k_giant<512, Sink, false><<<kSMs * 2, 512, 0, st>>>(csr, lists, 0, ctr + C_WORK + 7, ctr, sink,
                                                      d_tables + 256 * kTableGiant, none, plan, 4);
  launches += 6;
  if (hp.bufs)
    enqueue_head<Sink, false>(st, csr, hp.asrc, hp.m, hp.m_dev, hp.gbase, hp.G, *hp.bufs, ctr, sink,
                              none, hp.tuning, launches);
  STC_CUDA(cudaGetLastError());
}

// Identity of a captured persistent sequence: every pointer and size its
// kernels were given.
struct PersistentKey {
  const void* p[20];
  uint64_t v[6];
};

template <class Sink>
void count_persistent(stc_ctx* c, const Csr& csr, const ClassBounds& cb, uint32_t* lists,
                      uint32_t* plan, unsigned long long* ctr, const uint8_t* d_tables,
                      const Sink& sink, const void* s0, const void* s1, uint64_t s2,
                      const HeadPlan& hp) {
  cudaStream_t st = c->stream;
  STC_CUDA(cudaFuncSetAttribute(k_persistent<Sink>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kPersistentSmem));
  STC_CUDA(cudaFuncSetAttribute(k_block<512, Sink, false, kStreamUnroll, false>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)StageMem::bytes(kLargeCap, 2 * kLargeCap)));
  if (hp.bufs) prepare_head<Sink, false>(hp.tuning);
  // The legacy default stream cannot be captured: launch directly there.
  // So does a count that is itself being captured (a batch group's whole
  // pipeline) or that reads its arc count on the device (the one capped
  // run that sizes such a pipeline's buffers).
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (st != nullptr && st != cudaStreamLegacy && st != cudaStreamPerThread)
    STC_CUDA(cudaStreamIsCapturing(st, &cs));
  if (st == nullptr || st == cudaStreamLegacy || st == cudaStreamPerThread ||
      cs != cudaStreamCaptureStatusNone || hp.m_dev) {
    enqueue_persistent(st, csr, cb, lists, plan, ctr, d_tables, sink, hp, c->launches);
    return;
  }
  PersistentKey key{};
  const HeadBufs hb = hp.bufs ? *hp.bufs : HeadBufs{};
  const void* ptrs[20] = {csr.off, csr.nbr, csr.sgn, csr.verts, lists, plan, ctr, d_tables, s0,
                          hp.asrc, hb.keys, hb.alt, hb.aend, hb.runs, hb.lists.base, hp.fdeg, csr.nkey, hb.stream.sbits, hp.gbase,
                          hb.stream.low};
  memcpy(key.p, ptrs, sizeof(ptrs));
  key.v[0] = csr.n;
  key.v[1] = cb.tiny_max;
  key.v[2] = s2;
  key.v[3] = reinterpret_cast<uint64_t>(s1);
  key.v[4] = hp.m;
  key.v[5] = reinterpret_cast<uint64_t>(hb.sort_ws.words) ^
             ((uint64_t)hp.tuning.block_threads << 48) ^ ((uint64_t)hp.tuning.unroll[0] << 56) ^
             ((uint64_t)hp.tuning.unroll[1] << 58) ^ ((uint64_t)hp.tuning.unroll[2] << 60) ^
             ((uint64_t)hp.tuning.hash_factor[0] << 40) ^ ((uint64_t)hp.tuning.hash_factor[1] << 42) ^
             ((uint64_t)hp.tuning.hash_factor[2] << 44) ^ ((uint64_t)hp.bytes << 62) ^
             ((uint64_t)hp.short_arcs << 63);
  static_assert(sizeof(PersistentKey) <= sizeof(c->graph_key), "graph key size");
  if (c->graph_exec && memcmp(c->graph_key, &key, sizeof(key)) == 0) {
    STC_CUDA(cudaGraphLaunch(c->graph_exec, st));
    c->launches += c->graph_launches;
    return;
  }
  if (c->graph_exec) {
    STC_CUDA(cudaGraphExecDestroy(c->graph_exec));
    c->graph_exec = nullptr;
  }
  int launches = 0;
  cudaGraph_t graph = nullptr;
  STC_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
  try {
    enqueue_persistent(st, csr, cb, lists, plan, ctr, d_tables, sink, hp, launches);
  } catch (...) {
    cudaStreamEndCapture(st, &graph);
    if (graph) cudaGraphDestroy(graph);
    throw;
  }
  STC_CUDA(cudaStreamEndCapture(st, &graph));
  const cudaError_t e = cudaGraphInstantiate(&c->graph_exec, graph, 0);
  cudaGraphDestroy(graph);
  STC_CUDA(e);
  memcpy(c->graph_key, &key, sizeof(key));
  c->graph_launches = launches;
  STC_CUDA(cudaGraphLaunch(c->graph_exec, st));
  c->launches += launches;
}

// ------------------------------------------------------------- split ----
// The sign-split copy of the arc heads (the layout of
// MC/tc_merge_sign_split.cpp:20-146 and GM/signed_tc.hxx:302-396, kept beside
// the sorted heads instead of replacing them): each list's positive heads,
// then its negative heads, both ascending; psplit[u] = positive heads of u.
// Each lane takes one vertex; a list of up to 32 heads is split by its lane
// alone (count the positives, then place every head), and the warp splits
// the longer lists of its 32 vertices together, 32 heads per step, placing
// them with ballots and the popcounts of the lanes below.
constexpr uint32_t kSplitShort = 32;

__global__ void k_split_csr(const uint64_t* __restrict__ off, const uint32_t* __restrict__ nbr,
                            const int8_t* __restrict__ sgn, uint32_t n,
                            uint32_t* __restrict__ out, uint32_t* __restrict__ psplit,
                            const unsigned long long* __restrict__ err) {
  if (device_failed(err)) return;
  const uint32_t lane = lane_id();
  const uint32_t lt = lanemask_lt();
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += stride) {
    const uint32_t u = base + lane;
    const bool valid = u < n;
    const uint64_t b = valid ? off[u] : 0, e = valid ? off[u + 1] : 0;
    if (valid && e - b <= kSplitShort) {
      uint32_t pos = 0;
      for (uint64_t i = b; i < e; i++) pos += sgn[i] >= 0;
      uint32_t wp = 0, wn = 0;
      for (uint64_t i = b; i < e; i++) {
        const uint32_t x = nbr[i];
        if (sgn[i] >= 0) out[b + wp++] = x;
        else out[b + pos + wn++] = x;
      }
      psplit[u] = pos;
    }
    uint32_t longs = __ballot_sync(kFull, valid && e - b > kSplitShort);
    while (longs) {
      const int src = __ffs(longs) - 1;
      longs &= longs - 1;
      const uint64_t lb = __shfl_sync(kFull, b, src), le = __shfl_sync(kFull, e, src);
      uint32_t pos = 0;
      for (uint64_t at = lb; at < le; at += 32) {
        const uint64_t i = at + lane;
        pos += __popc(__ballot_sync(kFull, i < le && sgn[i] >= 0));
      }
      uint32_t wp = 0, wn = 0;
      for (uint64_t at = lb; at < le; at += 32) {
        const uint64_t i = at + lane;
        const bool in = i < le;
        const bool p = in && sgn[i] >= 0;
        const uint32_t bp = __ballot_sync(kFull, p), bn = __ballot_sync(kFull, in && !p);
        if (p) out[lb + wp + __popc(bp & lt)] = nbr[i];
        else if (in) out[lb + pos + wn + __popc(bn & lt)] = nbr[i];
        wp += __popc(bp);
        wn += __popc(bn);
      }
      if (lane == 0) psplit[base + src] = pos;
    }
  }
}

// ------------------------------------------------------------ shards ----
// A shard of a count is a contiguous range of source vertices in rank space
// chosen so that the shards carry about the same merge-model cost: vertex u
// costs 1 + sum over v in N+(u) of (d+(u) + d+(v)), saturated at 2^32 - 1.
// With P(r) the cost of the ranks below r, shard s of S starts at the first
// rank r with P(r) >= ceil(P(n) s / S).  Every triangle is counted by the
// shard of its lowest-ranked vertex, so the shards' counts add up to the
// whole graph's.
struct VertexCost {
  const uint64_t* off;
  const uint32_t* nbr;
  const unsigned long long* err;
  __device__ uint32_t operator()(uint64_t u) const {
    if (device_failed(err)) return 1u;
    const uint64_t b = off[u], e = off[u + 1], du = e - b;
    uint64_t cost = 1;
    for (uint64_t i = b; i < e; i++) {
      const uint32_t v = nbr[i];
      cost += du + (off[v + 1] - off[v]);
    }
    return (uint32_t)(cost < 0xFFFFFFFFull ? cost : 0xFFFFFFFFull);
  }
};
struct EmitPrefix {
  uint64_t* pre;
  __device__ void operator()(uint64_t i, uint64_t pos, uint32_t) const { pre[i] = pos; }
};

// Thread 0 writes the shard's first rank, thread 1 its end.
__global__ void k_shard_bounds(const uint64_t* __restrict__ pre, uint32_t n, uint32_t shard,
                               uint32_t shards, unsigned long long* __restrict__ ctr) {
  if (threadIdx.x > 1) return;
  const uint32_t s = shard + threadIdx.x;
  uint32_t r = 0;
  if (s >= shards) {
    r = n;
  } else if (s > 0) {
    const uint64_t target = (pre[n] * s + shards - 1) / shards;
    uint32_t lo = 0, hi = n;  // first r with pre[r] >= target (pre[n] = total)
    while (lo < hi) {
      const uint32_t mid = lo + ((hi - lo) >> 1);
      if (pre[mid] < target) lo = mid + 1; else hi = mid;
    }
    r = lo;
  }
  ctr[C_SHARD_LO + threadIdx.x] = r;
}

// Writes the rank range of cfg.shard into the counters (device side only).
void shard_range(stc_ctx* c, const DeviceGraph& g, uint32_t shard, uint32_t shards) {
  uint64_t* pre = buffer<uint64_t>(c, B_SHARD_COST, (size_t)g.n + 1);
  uint64_t* sums = buffer<uint64_t>(c, B_SCAN_SUMS, kScanSums);
  const unsigned long long* err = (unsigned long long*)counters(c) + C_ERROR;
  range_scan(VertexCost{g.off, g.nbr, err}, EmitPrefix{pre}, g.n, sums, c->stream, &c->launches);
  STC_CUDA(cudaMemcpyAsync(pre + g.n, sums + range_partition(g.n, kScanTile, kMaxSortGrid).grid,
                           sizeof(uint64_t), cudaMemcpyDeviceToDevice, c->stream));
  k_shard_bounds<<<1, 32, 0, c->stream>>>(pre, g.n, shard, shards, (unsigned long long*)counters(c));
  c->launches++;
}

}  // namespace

// Fixed degree-threshold dispatch: HEAD when A' is not the longer list
// (bucket |A'| <= bucket |B|) and |B| <= 4095 (for lists of the warp class,
// which also decides tiny lists, only when |B| >= 8: short arcs of short
// lists cost less on the tail side than an entry in the head side's sort,
// while a longer list would be staged there for a handful of them), SEARCH
// when B is at least 16x longer than A', MERGE when both are short, HASH
// otherwise (the giant class, which stages no hash, merges instead of
// hashing).  Without `head`, the tail-side table of the first version (no
// HEAD cells), which the no-allocation path uses.
void fixed_dispatch_tables(uint8_t* out, bool head) {
  for (int t = 0; t < kTableClasses; t++)
    for (int a = 0; a < 16; a++)
      for (int b = 0; b < 16; b++) {
        uint8_t s = STC_STRATEGY_HASH;
        const int bmin = t == kTableWarp ? 4 : 1;
        if (head && b >= bmin && b <= 12 && a <= b) s = STC_STRATEGY_HEAD;
        else if (b >= a + 4) s = STC_STRATEGY_SEARCH;
        else if (a <= 3 && b <= 5) s = STC_STRATEGY_MERGE;
        out[256 * t + 16 * a + b] = s;
      }
}

namespace {
// Cached tables in B_DISPATCH_FIXED: the fixed tables, and the forced-HEAD
// tables (HEAD wherever it applies, HASH elsewhere).
enum { kFixedHead = 0, kForcedHead = 1, kCachedTables = 2 };
}  // namespace

// Device copy of the dispatch tables a call uses: a forced strategy fills
// every cell (HEAD only the cells where it applies); otherwise the learned
// tables when the context holds a model and the call asks for them, else
// the fixed ones.  Per-vertex counts take the fixed tables, and no forced HEAD
// (the head side keeps an arc's counts in 16 bits, which |A'| <= 4095, as in
// the fixed tables' HEAD cells, cannot exceed).  `uses_head` (optional)
// receives whether the tables send any cell to the head side.
const uint8_t* dispatch_tables(stc_ctx* c, const CountConfig& cfg, bool* uses_head) {
  const bool totals = cfg.vertex_counts == nullptr;
  if (uses_head) *uses_head = false;
  if (!c->fixed_ready) {
    uint8_t h[kCachedTables * kTableBytes];
    fixed_dispatch_tables(h + kFixedHead * kTableBytes, true);
    for (size_t i = 0; i < kTableBytes; i++)
      h[kForcedHead * kTableBytes + i] =
          (i & 15) <= 12 ? (uint8_t)STC_STRATEGY_HEAD : (uint8_t)STC_STRATEGY_HASH;
    uint8_t* t = buffer<uint8_t>(c, B_DISPATCH_FIXED, sizeof(h));
    STC_CUDA(cudaMemcpyAsync(t, h, sizeof(h), cudaMemcpyHostToDevice, c->stream));
    STC_CUDA(cudaStreamSynchronize(c->stream));  // `h` is pageable and leaves scope
    c->fixed_ready = true;
  }
  const uint8_t* cached = buffer<uint8_t>(c, B_DISPATCH_FIXED, kCachedTables * kTableBytes);
  if (cfg.strategy == STC_STRATEGY_HEAD) {
    if (uses_head) *uses_head = totals;
    if (totals) return cached + kForcedHead * kTableBytes;
    uint8_t* t = buffer<uint8_t>(c, B_WORK2, kTableBytes);
    STC_CUDA(cudaMemsetAsync(t, (int)STC_STRATEGY_HASH, kTableBytes, c->stream));
    return t;
  }
  if (cfg.strategy != STC_STRATEGY_AUTO) {
    uint8_t* t = buffer<uint8_t>(c, B_WORK2, kTableBytes);
    STC_CUDA(cudaMemsetAsync(t, (int)cfg.strategy, kTableBytes, c->stream));
    return t;
  }
  if (totals && cfg.dispatch == STC_DISPATCH_LEARNED && c->model_loaded) {
    if (uses_head) *uses_head = c->learned_uses_head;
    return buffer<uint8_t>(c, B_DISPATCH, kTableBytes);
  }
  if (uses_head) *uses_head = true;
  return cached + kFixedHead * kTableBytes;
}

// Builds the sign-split copy of g's heads on the context's stream.
void build_split(stc_ctx* c, DeviceGraph& g) {
  g.nbr_split = buffer<uint32_t>(c, B_SPLIT_NBR, g.m_fwd + 4);
  g.psplit = buffer<uint32_t>(c, B_SPLIT_POS, g.n);
  STC_CUDA(cudaMemsetAsync(g.nbr_split + g.m_fwd, 0, 4 * sizeof(uint32_t), c->stream));
  k_split_csr<<<kSMs * 8, 256, 0, c->stream>>>(g.off, g.nbr, g.sgn, g.n, g.nbr_split, g.psplit,
                                               (unsigned long long*)counters(c) + C_ERROR);
  c->launches++;
  STC_CUDA(cudaGetLastError());
}

void count_triangles(stc_ctx* c, const DeviceGraph& gin, const CountConfig& cfg) {
  if (gin.n == 0 || gin.m_fwd == 0) return;
  if (gin.n > kMaxVertices) fail(STC_ERR_LIMIT, "counts need vertex ids below 2^31 - 2");
  cudaStream_t st = c->stream;
  DeviceGraph g = gin;
  const bool split = cfg.strategy == STC_STRATEGY_SPLIT ||
                     (cfg.strategy == STC_STRATEGY_AUTO && cfg.dispatch == STC_DISPATCH_LEARNED &&
                      c->model_loaded && c->learned_uses_split);
  if (split) build_split(c, g);
  Csr csr{g.off, g.nbr, g.sgn, g.verts, g.n, g.nbr_split, g.psplit, g.nkey};
  unsigned long long* ctr = (unsigned long long*)counters(c);
  bool uses_head = false;
  const uint8_t* d_table = dispatch_tables(c, cfg, &uses_head);
  // The head-side pass runs when the tables send arcs there.
  const bool head = uses_head && (cfg.class_mask & 0x20u) && g.asrc != nullptr &&
                    g.nkey != nullptr && g.n >= 2;
  HeadBufs hb;
  if (head) hb = head_buffers(c, g);
  else if (!g.bytes_done) algorithmic_bytes(c, g);
  const bool timed = cfg.arc_cycles != nullptr;
  const ArcTimes at{(unsigned long long*)cfg.arc_cycles, (unsigned long long*)cfg.arc_counts};
  const unsigned long long* range = nullptr;
  if (cfg.shards > 1) {
    shard_range(c, g, cfg.shard, cfg.shards);
    range = ctr + C_SHARD_LO;
  }

  // Vertex classes (a forced strategy disables the tiny class, which only
  // implements the search form; so does timing, so that every strategy's
  // timings cover the same arcs).
  const bool tiny =
      !timed && (cfg.strategy == STC_STRATEGY_AUTO || cfg.strategy == STC_STRATEGY_SEARCH);
  const ClassBounds cb{tiny ? kTinyMax : 1u, kWarpCap, kBlockCap, kLargeCap};
  // Short arcs are counted where the head side's keys are made, unless a
  // strategy is forced or arcs are timed.
  const bool short_arcs = head && !timed && cfg.strategy == STC_STRATEGY_AUTO;
  if (short_arcs) csr.short_max = kShortArc;

  // The persistent engine has no SPLIT path: counts that use SPLIT take the
  // per-class kernels.
  if (cfg.persistent && !timed && cfg.shards <= 1 && !split) {
    uint32_t* lists = buffer<uint32_t>(c, B_WORK, (size_t)g.n + kPlanWords + 8);
    uint32_t* plan = lists + g.n + 4;
    HeadPlan hp;
    if (head) {
      hp.bufs = &hb;
      hp.asrc = g.asrc;
      hp.fdeg = g.fdeg;
      hp.m = g.m_fwd;
      hp.bytes = !g.bytes_done;
      hp.short_arcs = short_arcs;
      hp.m_dev = g.m_dev;
      hp.gbase = g.G ? g.gbase : nullptr;
      hp.G = g.G;
      hp.tuning = c->tuning;
    }
    if (cfg.vertex_counts) {
      const VertexSink sink{(unsigned long long*)cfg.vertex_counts, g.verts};
      count_persistent(c, csr, cb, lists, plan, ctr, d_table, sink, sink.vcounts, nullptr, 1, hp);
    } else if (cfg.graph_counts) {
      const GraphSink sink{(unsigned long long*)cfg.graph_counts, g.gbase, g.G};
      count_persistent(c, csr, cb, lists, plan, ctr, d_table, sink, sink.gcounts, sink.gbase,
                       2 + ((uint64_t)g.G << 8), hp);
    } else {
      count_persistent(c, csr, cb, lists, plan, ctr, d_table, TotalSink{}, nullptr, nullptr, 0,
                       hp);
    }
    return;
  }
  // Runs f with the sink of this count.
  auto with_sink = [&](auto f) {
    if (cfg.vertex_counts) f(VertexSink{(unsigned long long*)cfg.vertex_counts, g.verts});
    else if (cfg.graph_counts) f(GraphSink{(unsigned long long*)cfg.graph_counts, g.gbase, g.G});
    else f(TotalSink{});
  };
  const uint8_t* need = nullptr;
  if (head) {
    with_sink([&](const auto& sink) {
      enqueue_head_keys(st, csr, g.asrc, g.fdeg, g.m_fwd, g.m_dev, !g.bytes_done, short_arcs, hb,
                        d_table, range, ctr, sink, c->launches);
    });
    need = hb.need;
  }
  k_classify_count<<<kSMs * 4, 256, 0, st>>>(g.off, g.n, cb, ctr, range, need);
  STC_CUDA(cudaMemcpyAsync(c->h_pinned + C_WORK, counters(c) + C_WORK,
                           (C_MAX_FDEG + 1 - C_WORK) * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
  STC_CUDA(cudaStreamSynchronize(st));
  const uint32_t max_fdeg = (uint32_t)c->h_pinned[C_MAX_FDEG];
  uint32_t counts[kClasses], starts[kClasses + 1];
  starts[0] = 0;
  for (int i = 0; i < kClasses; i++) {
    counts[i] = (uint32_t)c->h_pinned[C_WORK + i];
    starts[i + 1] = starts[i] + counts[i];
  }
  uint32_t* lists = buffer<uint32_t>(c, B_WORK, (size_t)starts[kClasses] + 8);
  uint32_t* d_starts = lists + starts[kClasses];
  STC_CUDA(cudaMemcpyAsync(d_starts, starts, kClasses * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  // Cursors of the fill, then the dynamic queues, live in C_WORK ...
  STC_CUDA(cudaMemsetAsync(counters(c) + C_WORK, 0, 8 * sizeof(uint64_t), st));
  k_classify_fill<<<kSMs * 4, 256, 0, st>>>(g.off, g.n, cb, lists, d_starts, ctr, range, need);
  STC_CUDA(cudaMemsetAsync(counters(c) + C_WORK, 0, 8 * sizeof(uint64_t), st));
  c->launches += 2;

  auto run = [&](const auto& sink, auto time_tag) {
    using Sink = std::decay_t<decltype(sink)>;
    constexpr bool kT = decltype(time_tag)::value;
    launch_classes<Sink, kT>(st, csr, lists, counts, starts, max_fdeg, ctr, d_table, sink, at,
                             c->tuning, cfg.class_mask, c->launches);
    if (head) {
      prepare_head<Sink, kT>(c->tuning);
      enqueue_head<Sink, kT>(st, csr, g.asrc, g.m_fwd, g.m_dev, g.G ? g.gbase : nullptr, g.G, hb,
                             ctr, sink, at, c->tuning, c->launches, cfg.class_mask);
    }
  };
  if (timed) run(TotalSink{}, std::true_type{});
  else with_sink([&](const auto& sink) { run(sink, std::false_type{}); });
  STC_CUDA(cudaGetLastError());
}

}  // namespace stc

// ===================================================== no-allocation path ===
// stc_count_oriented_csr_noalloc counts an oriented forward CSR that already
// sits in device memory without allocating anything: for callers that cannot
// call cudaMalloc (code running under a custom device allocator or inside a
// memory budget it does not control).  Its scratch (vertex worklists, the
// dispatch table, counters) lives in one file-scope device array of fixed
// size; every GPU that loads the library holds that array until exit, every
// call shares it, and calls that overlap on the GPU race on it.
namespace stc {
namespace {

constexpr uint32_t kNoAllocMaxVertices = 1u << 22;  // 16 MiB of worklists
constexpr int kNoAllocMaxDevices = 64;

struct NoAllocScratch {
  unsigned long long ctr[C_SLOTS];
  uint8_t table[kTableBytes];
  uint32_t lists[kNoAllocMaxVertices + 8];
};

static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(NoAllocScratch)];

// Input checks on the device, in two grid-stride passes with coalesced
// reads and no per-list loop, so that a long list (a hub keeps its whole
// degree under an id-ordered orientation) costs no more than other entries.
// Any violation sets ctr[C_ERROR] = kDeviceErrCsr.
// Per vertex: offsets start at 0, never decrease and end at m, and the first
// head of a non-empty list is above its tail.
__global__ void k_check_offsets(const uint64_t* __restrict__ off, const uint32_t* __restrict__ heads,
                                uint32_t n, uint64_t m, unsigned long long* __restrict__ ctr) {
  const uint32_t stride = gridDim.x * blockDim.x;
  if (blockIdx.x == 0 && threadIdx.x == 0 && (off[0] != 0 || off[n] != m))
    atomicExch(ctr + C_ERROR, (unsigned long long)kDeviceErrCsr);
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += stride) {
    const uint64_t b = off[u], e = off[u + 1];
    const bool bad = e < b || e > m || (e > b && heads[b] <= u);
    if (bad) atomicExch(ctr + C_ERROR, (unsigned long long)kDeviceErrCsr);
  }
}

// Per arc: every head is below n and above the head before it, unless it
// starts its list (then the pass above compared it with its tail).  Only a
// head not above its predecessor looks up its list, by a binary search of
// the offsets: in a valid CSR that happens at most once per list.
__global__ void k_check_heads(const uint64_t* __restrict__ off, const uint32_t* __restrict__ heads,
                              uint32_t n, uint64_t m, unsigned long long* __restrict__ ctr) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride) {
    const uint32_t h = heads[i];
    bool bad = h >= n;
    if (!bad && i > 0 && h <= heads[i - 1]) {
      uint32_t lo = 0, hi = n;  // largest u in [0, n) with off[u] <= i
      while (hi - lo > 1) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (off[mid] <= i) lo = mid; else hi = mid;
      }
      bad = off[lo] != i;  // i must start the list of u
    }
    if (bad) atomicExch(ctr + C_ERROR, (unsigned long long)kDeviceErrCsr);
  }
}

// The scratch array's device address in the current context.  It is looked
// up (cudaGetSymbolAddress) once per CUDA context: the first call in a
// context, with that context current, and again whenever the current
// context differs from the last one seen on that device, as after
// cudaDeviceReset or under a caller's own context.  Contexts are told apart
// by the driver's context id, reached through the runtime's driver entry
// points (so libstc needs no link to the driver library); without them the
// address is looked up on every call.
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long*);

std::mutex g_noalloc_mu;
struct NoAllocSlot {
  unsigned long long ctx_id = 0;
  bool valid = false;
  void* addr = nullptr;
};
NoAllocSlot g_noalloc_slot[kNoAllocMaxDevices];

bool current_context_id(unsigned long long* id) {
  static CtxGetCurrentFn get_current = nullptr;
  static CtxGetIdFn get_id = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    cudaDriverEntryPointQueryResult q1 = cudaDriverEntryPointSymbolNotFound, q2 = q1;
    void* f1 = nullptr;
    void* f2 = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f1, 12000, cudaEnableDefault, &q1) ==
            cudaSuccess &&
        cudaGetDriverEntryPointByVersion("cuCtxGetId", &f2, 12000, cudaEnableDefault, &q2) ==
            cudaSuccess &&
        q1 == cudaDriverEntryPointSuccess && q2 == cudaDriverEntryPointSuccess) {
      get_current = reinterpret_cast<CtxGetCurrentFn>(f1);
      get_id = reinterpret_cast<CtxGetIdFn>(f2);
    }
    (void)cudaGetLastError();
  }
  if (!get_current || !get_id) return false;
  CUcontext cx = nullptr;
  if (get_current(&cx) != CUDA_SUCCESS || cx == nullptr) return false;
  return get_id(cx, id) == CUDA_SUCCESS;
}

cudaError_t noalloc_scratch(int device, NoAllocScratch** out) {
  std::lock_guard<std::mutex> lock(g_noalloc_mu);
  unsigned long long id = 0;
  const bool have_id = current_context_id(&id);
  NoAllocSlot& slot = g_noalloc_slot[device];
  if (!have_id || !slot.valid || slot.ctx_id != id) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    slot.addr = p;
    slot.ctx_id = id;
    slot.valid = have_id;
  }
  *out = static_cast<NoAllocScratch*>(slot.addr);
  return cudaSuccess;
}

stc_status noalloc_cuda(cudaError_t e) {
  (void)cudaGetLastError();
  return e == cudaErrorMemoryAllocation ? STC_ERR_OUT_OF_MEMORY : STC_ERR_CUDA;
}

}  // namespace

}  // namespace stc

#define STC_NA(call)                                   \
  do {                                                 \
    const cudaError_t e_ = (call);                     \
    if (e_ != cudaSuccess) return stc::noalloc_cuda(e_); \
  } while (0)

extern "C" stc_status stc_count_oriented_csr_noalloc(const uint64_t* d_offsets,
                                                      const uint32_t* d_heads,
                                                      const int8_t* d_signs, uint32_t n,
                                                      uint64_t m, void* stream, stc_counts* out) {
  using namespace stc;
  if (!out || !d_offsets || (m && (!d_heads || !d_signs))) return STC_ERR_INVALID_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(d_heads) & 15) || (reinterpret_cast<uintptr_t>(d_signs) & 3))
    return STC_ERR_INVALID_ARGUMENT;
  if (n > kNoAllocMaxVertices || m >= (1ull << 32)) return STC_ERR_LIMIT;
  *out = stc_counts{0, 0, 0, 0};
  if (n == 0) return STC_OK;
  int device = 0;
  STC_NA(cudaGetDevice(&device));
  if (device < 0 || device >= kNoAllocMaxDevices) return STC_ERR_NO_DEVICE;
  NoAllocScratch* scr = nullptr;
  STC_NA(noalloc_scratch(device, &scr));
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned long long* ctr = scr->ctr;
  STC_NA(cudaMemsetAsync(ctr, 0, sizeof(scr->ctr), st));
  k_check_offsets<<<kSMs * 4, 256, 0, st>>>(d_offsets, d_heads, n, m, ctr);
  if (m) k_check_heads<<<kSMs * 8, 256, 0, st>>>(d_offsets, d_heads, n, m, ctr);
  STC_NA(cudaGetLastError());
  uint64_t slots[C_SLOTS];
  STC_NA(cudaMemcpyAsync(slots, ctr, sizeof(slots), cudaMemcpyDeviceToHost, st));
  STC_NA(cudaStreamSynchronize(st));
  if (slots[C_ERROR]) return STC_ERR_INVALID_ARGUMENT;
  if (m == 0) return STC_OK;

  uint8_t table[kTableBytes];
  fixed_dispatch_tables(table, false);
  STC_NA(cudaMemcpyAsync(scr->table, table, sizeof(table), cudaMemcpyHostToDevice, st));
  const ClassBounds cb{kTinyMax, kWarpCap, kBlockCap, kLargeCap};
  k_classify_count<<<kSMs * 4, 256, 0, st>>>(d_offsets, n, cb, ctr, nullptr);
  STC_NA(cudaMemcpyAsync(slots, ctr, sizeof(slots), cudaMemcpyDeviceToHost, st));
  STC_NA(cudaStreamSynchronize(st));
  const uint32_t max_fdeg = (uint32_t)slots[C_MAX_FDEG];
  uint32_t counts[kClasses], starts[kClasses + 1];
  starts[0] = 0;
  for (int i = 0; i < kClasses; i++) {
    counts[i] = (uint32_t)slots[C_WORK + i];
    starts[i + 1] = starts[i] + counts[i];
  }
  uint32_t* lists = scr->lists;
  uint32_t* d_starts = lists + starts[kClasses];
  STC_NA(cudaMemcpyAsync(d_starts, starts, kClasses * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
  STC_NA(cudaMemsetAsync(ctr + C_WORK, 0, 8 * sizeof(uint64_t), st));
  k_classify_fill<<<kSMs * 4, 256, 0, st>>>(d_offsets, n, cb, lists, d_starts, ctr, nullptr);
  STC_NA(cudaMemsetAsync(ctr + C_WORK, 0, 8 * sizeof(uint64_t), st));

  const Csr csr{d_offsets, d_heads, d_signs, nullptr, n, nullptr, nullptr};
  int launches = 0;
  try {
    launch_classes<TotalSink, false>(st, csr, lists, counts, starts, max_fdeg, ctr, scr->table,
                                     TotalSink{}, ArcTimes{nullptr, nullptr}, Tuning{}, 0x1Fu,
                                     launches);
  } catch (const Error& e) {
    (void)cudaGetLastError();
    return e.status;
  }
  STC_NA(cudaGetLastError());
  STC_NA(cudaMemcpyAsync(slots, ctr, sizeof(slots), cudaMemcpyDeviceToHost, st));
  STC_NA(cudaStreamSynchronize(st));
  if (slots[C_ERROR]) return STC_ERR_INTERNAL;
  out->t0 = slots[C_T0];
  out->t1 = slots[C_T1];
  out->t2 = slots[C_T2];
  out->t3 = slots[C_T3];
  return STC_OK;
}
