// Graph build on the GPU: ingest + dedup, degree, (degree, id) rank,
// orientation and the forward CSR with an int8 sign array.
//
// Reference: build_forward_csr (MC/graph_io.h:231-402) followed by
// sort_adj_lists (MC/tc_serial.cpp:33-93), MC = "Signed_TC/Multicore
// Implementations".  The reference sorts 12-byte structs on one thread,
// counting-sorts vertices by degree and scatters arcs with atomics into
// unsorted lists that a second pass sorts.  Here every stage is a sort or a
// streaming pass over HBM:
//
//   1. pack   (min << b | max), sign in bit 63; self-loops -> sentinel keys
//   2. stable radix sort over the 2b id bits; keep the first key of each run
//      (== the reference's "first of equal (u, v)", made deterministic)
//   3. degree = atomics over the unique keys (warp-aggregated on the min id)
//   4. rank   = stable radix sort of (deg << 32 | id) on the degree bits:
//      ties fall back to ascending id exactly like the counting sort at
//      MC/graph_io.h:270-317
//   5. orient + relabel into rank space: arc (rank lo -> rank hi); sorting
//      these keys gives every list already sorted, so no per-list sort
//   6. offsets = exclusive scan of out-degrees.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "internal.h"
#include "radix_sort.cuh"
#include "stc_device.cuh"

namespace stc {

namespace {

constexpr int kThreads = 256;

inline uint32_t grid_for(uint64_t n, uint32_t per_thread = 1) {
  uint64_t g = (n + (uint64_t)kThreads * per_thread - 1) / ((uint64_t)kThreads * per_thread);
  if (g < 1) g = 1;
  if (g > (uint64_t)kSMs * 16) g = kSMs * 16;
  return (uint32_t)g;
}

// Max kept id and self-loop count; four edges of a thread in flight.
__global__ void __launch_bounds__(256) k_scan_ids(const uint32_t* __restrict__ u,
                                                  const uint32_t* __restrict__ v, uint64_t m,
                                                  unsigned long long* __restrict__ ctr) {
  uint32_t mx = 0;
  uint32_t self = 0;
  auto add = [&](uint32_t a, uint32_t b) {
    if (a == b) self++;
    else mx = max(mx, max(a, b));
  };
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (; i + 3 * stride < m; i += 4 * stride) {
    uint32_t a[4], b[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      a[q] = __ldcs(u + i + q * stride);
      b[q] = __ldcs(v + i + q * stride);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) add(a[q], b[q]);
  }
  for (; i < m; i += stride) add(__ldcs(u + i), __ldcs(v + i));
  mx = __reduce_max_sync(kFull, mx);
  self = __reduce_add_sync(kFull, self);
  if (lane_id() == 0) {
    atomicMax(ctr + C_MAX_ID, (unsigned long long)mx);
    if (self) atomicAdd(ctr + C_SELF, (unsigned long long)self);
  }
}

// Dedup keys: (min << bits | max) with the negative flag in bit 63; a
// self-loop becomes the all-ones sentinel of the 2*bits window, which sorts
// last and can never equal a real key (real keys have min < max).
__global__ void k_pack_dedup(const uint32_t* __restrict__ u, const uint32_t* __restrict__ v,
                             const int8_t* __restrict__ s, uint64_t m, uint32_t bits,
                             uint64_t* __restrict__ keys) {
  const uint64_t sentinel = (bits * 2 >= 64) ? ~0ull >> 1 : ((1ull << (2 * bits)) - 1);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride) {
    const uint32_t a = __ldcs(u + i), b = __ldcs(v + i);
    const int8_t sg = __ldcs(s + i);
    uint64_t k;
    if (a == b) {
      k = sentinel;
    } else {
      const uint64_t lo = a < b ? a : b, hi = a < b ? b : a;
      k = (lo << bits) | hi | ((uint64_t)(sg < 0) << 63);
    }
    keys[i] = k;
  }
}

struct UniqueFlag {
  const uint64_t* keys;
  uint64_t mask;
  __device__ uint32_t operator()(uint64_t i) const {
    if (i == 0) return 1u;
    return (keys[i] & mask) != (keys[i - 1] & mask) ? 1u : 0u;
  }
};
struct UniqueEmit {
  const uint64_t* keys;
  uint64_t* out;
  __device__ void operator()(uint64_t i, uint64_t pos, uint32_t flag) const {
    if (flag) out[pos] = keys[i];
  }
};

// Undirected degree of every vertex from the sorted unique keys
// (min << bits | max).  The min endpoints of consecutive keys repeat, so a
// warp adds each run with one atomic.  The max endpoints are scattered and a
// few hubs may own millions of them, which would serialise on one address; so
// each CTA counts them in a shared-memory table that it flushes every tile of
// kDegTile keys, adding one global atomic per distinct vertex and tile (a
// vertex that finds no free slot within kDegProbes probes is added directly).
constexpr int kDegTile = 1024;
constexpr int kDegSlots = 2048;  // load <= 1/2 per tile
constexpr int kDegProbes = 8;

__global__ void __launch_bounds__(kThreads) k_degree(const uint64_t* __restrict__ keys, uint64_t mu,
                                                     uint32_t bits, uint32_t* __restrict__ deg) {
  __shared__ uint32_t tkey[kDegSlots], tcnt[kDegSlots];
  constexpr uint32_t kFree = 0xFFFFFFFFu;
  for (int i = threadIdx.x; i < kDegSlots; i += kThreads) {
    tkey[i] = kFree;
    tcnt[i] = 0;
  }
  __syncthreads();
  const uint64_t idmask = (1ull << bits) - 1;
  const uint64_t tiles = (mu + kDegTile - 1) / kDegTile;
  for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
#pragma unroll
    for (int r = 0; r < kDegTile / kThreads; r++) {
      const uint64_t i = t * kDegTile + (uint64_t)r * kThreads + threadIdx.x;
      const bool valid = i < mu;
      const uint64_t k = valid ? keys[i] : 0;
      const uint32_t a = valid ? (uint32_t)((k >> bits) & idmask) : kFree;
      const uint32_t b = valid ? (uint32_t)(k & idmask) : kFree;
      const unsigned pa = __match_any_sync(kFull, a);
      if (valid && (pa & lanemask_lt()) == 0) atomicAdd(deg + a, (uint32_t)__popc(pa));
      const unsigned pb = __match_any_sync(kFull, b);
      if (valid && (pb & lanemask_lt()) == 0) {
        const uint32_t add = (uint32_t)__popc(pb);
        uint32_t slot = (b * 0x9E3779B1u) >> (32 - 11);
        bool placed = false;
        for (int p = 0; p < kDegProbes && !placed; p++) {
          uint32_t cur = tkey[slot];
          if (cur == kFree) {  // claim the slot, or see who claimed it first
            const uint32_t old = atomicCAS(&tkey[slot], kFree, b);
            cur = old == kFree ? b : old;
          }
          if (cur == b) {
            atomicAdd(&tcnt[slot], add);
            placed = true;
          }
          slot = (slot + 1) & (kDegSlots - 1);
        }
        if (!placed) atomicAdd(deg + b, add);
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kDegSlots; i += kThreads) {
      const uint32_t v = tkey[i];
      if (v != kFree) {
        atomicAdd(deg + v, tcnt[i]);
        tkey[i] = kFree;
        tcnt[i] = 0;
      }
    }
    __syncthreads();
  }
}

// Vertex sort keys (deg << 32 | id) and the max degree.
__global__ void k_vertex_keys(const uint32_t* __restrict__ deg, uint32_t n,
                              uint64_t* __restrict__ vkeys, unsigned long long* __restrict__ ctr) {
  uint32_t mx = 0;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint32_t d = deg[i];
    vkeys[i] = ((uint64_t)d << 32) | i;
    mx = max(mx, d);
  }
  mx = __reduce_max_sync(kFull, mx);
  if (lane_id() == 0) atomicMax(ctr + C_MAX_DEG, (unsigned long long)mx);
}

__global__ void k_rank(const uint64_t* __restrict__ vkeys, uint32_t n, uint32_t* __restrict__ verts,
                       uint32_t* __restrict__ rank, const unsigned long long* __restrict__ err) {
  if (device_failed(err)) return;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += stride) {
    const uint32_t id = (uint32_t)vkeys[r];
    if (verts) verts[r] = id;
    rank[id] = r;
  }
}

// Orientation + relabelling: arc key (rank lo << bits | rank hi), sign in
// bit 63; out-degree histogram by rank.
__global__ void k_arc_keys(const uint64_t* __restrict__ ukeys, uint64_t mu, uint32_t bits,
                           const uint32_t* __restrict__ rank, uint64_t* __restrict__ akeys,
                           uint32_t* __restrict__ fdeg,
                           const unsigned long long* __restrict__ err) {
  if (device_failed(err)) return;
  const uint64_t idmask = (1ull << bits) - 1;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < mu; i += stride) {
    const uint64_t k = ukeys[i];
    const uint32_t ra = rank[(k >> bits) & idmask], rb = rank[k & idmask];
    const uint32_t lo = min(ra, rb), hi = max(ra, rb);
    akeys[i] = ((uint64_t)lo << bits) | hi | (k & (1ull << 63));
    atomicAdd(fdeg + lo, 1u);
  }
}

struct LoadU32 {
  const uint32_t* a;
  __device__ uint32_t operator()(uint64_t i) const { return a[i]; }
};
struct EmitOffset {
  uint64_t* off;
  __device__ void operator()(uint64_t i, uint64_t pos, uint32_t) const { off[i] = pos; }
};

// Algorithmic bytes of the arc at position i (tail u, head v) of a sorted
// CSR: the merge model, 5 (d+(u) + d+(v)) + 25, which a merge of both lists
// reads, and the probe model, 5 min(|A'|, |B|) + 30 (A' = the part of N+(u)
// after v, B = N+(v)), which a hash probe that streams the shorter list
// reads, with the arc's own 25 bytes and its entry staged once.
__device__ __forceinline__ void arc_bytes(uint64_t i, uint32_t u, uint32_t v,
                                          const uint64_t* __restrict__ off,
                                          const uint32_t* __restrict__ fdeg,
                                          unsigned long long& merge, unsigned long long& probe) {
  const uint64_t du = fdeg[u], dv = fdeg[v];
  merge += 5ull * (du + dv) + 25ull;
  const uint64_t alen = off[u + 1] - i - 1;
  probe += 5ull * (alen < dv ? alen : dv) + 30ull;
}

// Splits sorted arc keys into the neighbour, sign, tail and signed-head
// arrays (the last two only when given) and accumulates the merge-model and
// probe-model bytes of every arc (arc_bytes).
__global__ void k_csr_fill(const uint64_t* __restrict__ akeys, uint64_t ma, uint32_t bits,
                           const uint32_t* __restrict__ fdeg, const uint64_t* __restrict__ off,
                           uint32_t* __restrict__ nbr, int8_t* __restrict__ sgn,
                           uint32_t* __restrict__ asrc, uint32_t* __restrict__ nkey,
                           unsigned long long* __restrict__ ctr) {
  if (device_failed(ctr + C_ERROR)) return;
  const uint64_t idmask = (1ull << bits) - 1;
  unsigned long long bytes = 0, probe = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < ma; i += stride) {
    const uint64_t k = akeys[i];
    const uint32_t src = (uint32_t)((k >> bits) & idmask), dst = (uint32_t)(k & idmask);
    nbr[i] = dst;
    sgn[i] = (k >> 63) ? (int8_t)-1 : (int8_t)1;
    if (asrc) asrc[i] = src;
    if (nkey) nkey[i] = (dst << 1) | (uint32_t)(k >> 63);
    arc_bytes(i, src, dst, off, fdeg, bytes, probe);
  }
  bytes = warp_sum(bytes);
  probe = warp_sum(probe);
  if (lane_id() == 0 && bytes) {
    atomicAdd(ctr + C_ALG_BYTES, bytes);
    atomicAdd(ctr + C_PROBE_BYTES, probe);
  }
}

// Arc keys of a reference-layout CSR: one warp per vertex.  Checks the CSR on
// the way, before anything it holds is used as an index: offsets that decrease
// or pass m, ranks that are no permutation of [0, n) (`seen` starts at 0) and
// edges that leave the rank order set C_ERROR.
__global__ void k_csr_arc_keys(const uint64_t* __restrict__ off, const uint32_t* __restrict__ edges,
                               const int8_t* __restrict__ signs, const uint32_t* __restrict__ rank,
                               uint32_t n, uint64_t m, uint32_t bits, uint64_t* __restrict__ akeys,
                               uint32_t* __restrict__ fdeg, uint32_t* __restrict__ seen,
                               unsigned long long* __restrict__ ctr) {
  const uint32_t warps = gridDim.x * (blockDim.x / 32);
  for (uint32_t u = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); u < n; u += warps) {
    const uint64_t b = off[u], e = off[u + 1];
    const uint32_t ru = rank[u];
    bool bad = e < b || e > m || ru >= n;
    if (lane_id() == 0 && ru < n) bad |= atomicExch(seen + ru, 1u) != 0;
    if (__any_sync(kFull, bad)) {
      if (lane_id() == 0) atomicExch(ctr + C_ERROR, 1ull);
      continue;
    }
    for (uint64_t i = b + lane_id(); i < e; i += 32) {
      const uint32_t w = edges[i];
      const uint32_t rw = w < n ? rank[w] : 0u;
      if (rw <= ru || rw >= n) {  // ru >= 0: an id >= n fails too
        atomicExch(ctr + C_ERROR, 1ull);  // not a forward CSR of this rank order
        continue;
      }
      akeys[i] = ((uint64_t)ru << bits) | rw | ((uint64_t)(signs[i] < 0) << 63);
    }
    if (lane_id() == 0) fdeg[ru] = (uint32_t)(e - b);
  }
}

// Id-space export keys: (source id << bits | head id), sign in bit 63.
__global__ void k_export_keys(const uint64_t* __restrict__ ukeys, uint64_t mu, uint32_t bits,
                              const uint32_t* __restrict__ rank, uint64_t* __restrict__ ekeys,
                              uint32_t* __restrict__ fdeg_id) {
  const uint64_t idmask = (1ull << bits) - 1;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < mu; i += stride) {
    const uint64_t k = ukeys[i];
    const uint32_t a = (uint32_t)((k >> bits) & idmask), b = (uint32_t)(k & idmask);
    const bool fwd = rank[a] < rank[b];
    const uint32_t s = fwd ? a : b, t = fwd ? b : a;
    ekeys[i] = ((uint64_t)s << bits) | t | (k & (1ull << 63));
    atomicAdd(fdeg_id + s, 1u);
  }
}

// Where a sort reports a device-side wait that expired, and where its
// consumers look.
unsigned long long* sort_error(stc_ctx* c) { return (unsigned long long*)counters(c) + C_ERROR; }

void read_counters(stc_ctx* c, int first, int count) {
  STC_CUDA(cudaMemcpyAsync(c->h_pinned + first, counters(c) + first, count * sizeof(uint64_t),
                           cudaMemcpyDeviceToHost, c->stream));
  STC_CUDA(cudaStreamSynchronize(c->stream));
}

// The total of a range scan over sorted keys (range_reduce_scan with err),
// read to the host; fails if the sort did.
uint64_t read_total(stc_ctx* c, const uint64_t* sums, uint32_t grid) {
  STC_CUDA(cudaMemcpyAsync(c->h_pinned + C_WORK, sums + grid, 2 * sizeof(uint64_t),
                           cudaMemcpyDeviceToHost, c->stream));
  STC_CUDA(cudaStreamSynchronize(c->stream));
  check_device_error(c->h_pinned[C_WORK + 1]);
  return c->h_pinned[C_WORK];
}

// Rank-space CSR from unique keys: arc keys, sort, offsets, fill.
void finish_csr_from_arc_keys(stc_ctx* c, DeviceGraph& g, uint64_t* akeys, uint64_t* alt) {
  const SortSpace sort_ws = sort_space(c, g.m_fwd);
  uint64_t* sums = buffer<uint64_t>(c, B_SCAN_SUMS, kScanSums);
  uint64_t* sorted = radix_sort(akeys, alt, g.m_fwd, 0, 2 * (int)g.bits, sort_ws, sort_error(c), c->stream,
                                &c->launches);
  g.off = buffer<uint64_t>(c, B_OFF, (size_t)g.n + 1);
  range_scan(LoadU32{g.fdeg}, EmitOffset{g.off}, g.n, sums, c->stream, &c->launches);
  STC_CUDA(cudaMemcpyAsync(g.off + g.n, sums + range_partition(g.n, kScanTile, kMaxSortGrid).grid,
                           sizeof(uint64_t), cudaMemcpyDeviceToDevice, c->stream));
  g.nbr = buffer<uint32_t>(c, B_NBR, g.m_fwd + 8);  // + 8: the engine reads whole 32-byte chunks
  g.sgn = buffer<int8_t>(c, B_SGN, g.m_fwd + 8);
  g.asrc = buffer<uint32_t>(c, B_ASRC, g.m_fwd);
  g.nkey = buffer<uint32_t>(c, B_NKEY, g.m_fwd + 8);
  k_csr_fill<<<grid_for(g.m_fwd, 4), kThreads, 0, c->stream>>>(sorted, g.m_fwd, g.bits, g.fdeg,
                                                               g.off, g.nbr, g.sgn, g.asrc,
                                                               g.nkey,
                                                               (unsigned long long*)counters(c));
  g.bytes_done = true;
  c->launches += 1;
  STC_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------ batches ----
// A batch of G graphs is counted as one disjoint union: graph g's local id x
// becomes vbase[g] + x, where vbase is the prefix sum of the graphs' id
// spaces.  Edges (and vertices) of one graph are contiguous, so a CTA that
// owns a contiguous range finds the graph of its first element by binary
// search and then only moves a cursor forward.
__device__ __forceinline__ uint32_t first_segment(const uint64_t* __restrict__ bounds, uint32_t G,
                                                  uint64_t i) {
  uint32_t lo = 0, hi = G;  // largest g with bounds[g] <= i
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (bounds[mid] <= i) lo = mid; else hi = mid;
  }
  return lo;
}

// Id space of every graph (max endpoint + 1) and the self-loop count.  Each
// lane keeps the maximum of its current graph; a warp hands it over when one
// of its lanes moves on to another graph, which happens about once a graph
// and warp (a match of the lanes' graphs at every step took 1.2 ms for 98 M
// edges).
__global__ void __launch_bounds__(256) k_batch_ids(const uint32_t* __restrict__ u,
                                                   const uint32_t* __restrict__ v, uint64_t m,
                                                   const uint64_t* __restrict__ eoff, uint32_t G,
                                                   uint64_t per_cta, unsigned int* __restrict__ gspace,
                                                   unsigned long long* __restrict__ ctr) {
  const uint64_t begin = (uint64_t)blockIdx.x * per_cta;
  const uint64_t end = begin + per_cta < m ? begin + per_cta : m;
  if (begin >= end) return;
  uint32_t g = first_segment(eoff, G, begin);
  uint64_t gend = eoff[g + 1];
  uint32_t self = 0, space = 0;
  for (uint64_t i = begin + threadIdx.x; i < end; i += blockDim.x) {
    if (i >= gend) {
      if (space) atomicMax(gspace + g, space);
      space = 0;
      do {
        g++;
      } while (eoff[g + 1] <= i);
      gend = eoff[g + 1];
    }
    const uint32_t a = u[i], b = v[i];
    self += a == b;
    space = max(space, min(max(a, b), 0xFFFFFFFEu) + 1);  // an id of 2^32 - 1 must not wrap to 0
  }
  // The lanes of a warp mostly end in the same graph.
  const bool one = __all_sync(kFull, g == __shfl_sync(kFull, g, 0));
  const uint32_t mx = one ? __reduce_max_sync(kFull, space) : space;
  if (mx && (!one || lane_id() == 0)) atomicMax(gspace + g, mx);
  self = __reduce_add_sync(kFull, self);
  if (lane_id() == 0 && self) atomicAdd(ctr + C_SELF, (unsigned long long)self);
}

// ------------------------------------------------------- totals path ----
// A count of totals needs an acyclic orientation, not the reference's: every
// total order of the vertices counts each triangle once, from its lowest
// vertex.  So the totals path orders vertices by (degree counted over the
// input's edge copies, id) instead of (unique degree, id), which needs no
// dedup before the orientation: the arc sort that builds the CSR brings the
// copies of an edge together, and the first of each run is kept, the
// dedup's own rule (the sort is stable, so it is the first in input order).
// This removes the dedup sort of all input edges.

// Global ids of input edge i: the edge's own ids, plus the vertex base of
// its graph for a batch (found once per thread by a binary search, then by
// a cursor that only moves forward, as every thread's indices grow).
struct EdgeIds {
  const uint32_t* __restrict__ u;
  const uint32_t* __restrict__ v;
  const uint64_t* __restrict__ eoff;   // G + 1 edge offsets, or null for one graph
  const uint64_t* __restrict__ vbase;  // G + 1 vertex bases
  uint32_t G;
};

struct EdgeCursor {
  uint32_t g = 0;
  __device__ void start(const EdgeIds& e, uint64_t i) {
    if (e.eoff) g = first_segment(e.eoff, e.G, i);
  }
  __device__ void at(const EdgeIds& e, uint64_t i, uint32_t& a, uint32_t& b) {
    a = e.u[i];
    b = e.v[i];
    if (e.eoff) {
      while (e.eoff[g + 1] <= i) g++;
      const uint32_t base = (uint32_t)e.vbase[g];
      a += base;
      b += base;
    }
  }
};

// Degree of every vertex over the input's edge copies (self-loops skipped),
// or over a sample of them: with `shift` > 0, only the copies of the edges
// {a, b} whose hash has its top `shift` bits clear, 1 in 2^shift of the
// distinct edges (every copy of an edge is in or out together).  The order
// only has to be a total order for exact counts; on dense power-law graphs
// a sampled degree orders the vertices nearly as well (at RMAT scale 20 a
// 1/4 sample moves the intersection work by under 0.1%) for a quarter of
// the atomics.
// Endpoints are scattered over the degrees, so they are added there one by
// one; only the hubs, which may own millions of copies, would serialise on
// their address.  k_find_hubs names them from a sample, and a CTA counts
// those in shared memory.  (Counting every endpoint in a shared-memory table
// flushed per tile, hubs or not, took 3.1 ms at RMAT scale 24, this 0.8;
// 62 us against 20 for a million-point mesh.)

// Edges of the input are taken in chunks of kEdgeChunk, chunk c by CTA
// c mod grid: the CTAs of a launch work on neighbouring edges at any time,
// so for a batch they gather the ranks and degrees of a few neighbouring
// graphs at once, which stay in L2.  Lists too short to give every CTA such
// a chunk take smaller ones.
constexpr uint64_t kEdgeChunk = 4096;
constexpr int kEdgeItems = 4;  // edges of a thread in flight
constexpr uint32_t kEdgeGrid = kSMs * 6;
inline uint32_t edge_chunk(uint64_t m) {
  return m < kEdgeChunk * kEdgeGrid ? kEdgeItems * kThreads : (uint32_t)kEdgeChunk;
}
inline uint32_t edge_grid(uint64_t m) {
  return (uint32_t)std::min<uint64_t>((m + edge_chunk(m) - 1) / edge_chunk(m), kEdgeGrid);
}

__device__ __forceinline__ bool sampled_edge(uint32_t a, uint32_t b, uint32_t shift) {
  if (shift == 0) return true;
  const uint32_t lo = min(a, b), hi = max(a, b);
  return ((lo * 0x9E3779B1u) ^ (hi * 0x7FEB352Du) ^ ((lo ^ hi) >> 15)) >> (32 - shift) == 0;
}

// Hub table: kHubSlots ids in buckets of two.
constexpr uint32_t kHubSlots = 1024;
constexpr uint32_t kNoHub = 0xFFFFFFFFu;
// Lists and batches of fewer edges have no hub worth the sample.  (Additions
// to one address take 0.5 ns each: a shuffled star of 1,000,000 edges counts in
// 388 us with the table and took 731 without, one of 4,000,000 in a batch 0.85
// and 2.29 ms; without a hub 1,000,000 edges take 403 and 400 us, a batch of
// eight lists of 500,000 709 and 699.)
constexpr uint64_t kHubMinEdges = 1u << 19;
__device__ __forceinline__ uint32_t hub_bucket(uint32_t x) {
  return ((x * 0x9E3779B1u) >> (32 - 9)) * 2;  // of kHubSlots / 2 buckets
}
static_assert(kHubSlots == 2u << 9, "hub_bucket's shift");

// Ids that occur at least kHubHits times among `sample` (a power of two)
// endpoints taken at even distances: of 8,192, a hub with 1/1,000 of the
// endpoints is missed once in 20 lists, one with 1/500 never, and what is
// missed only costs its own serial additions.  One CTA (12 us for 2,048
// endpoints); ids that find both slots of their bucket taken are left out.
constexpr uint32_t kHubHits = 4;
inline uint32_t hub_sample(uint64_t m) { return m < (1u << 24) ? 2048 : 8192; }
inline size_t hub_smem(uint32_t sample) { return 4ull * sample * sizeof(uint32_t); }

__global__ void __launch_bounds__(1024) k_find_hubs(EdgeIds e, uint64_t m, uint32_t sample,
                                                    uint32_t* __restrict__ hubs) {
  extern __shared__ uint32_t hub_seen[];
  const uint32_t slots = 2 * sample;  // load <= 1/2
  uint32_t* id = hub_seen;
  uint32_t* hits = hub_seen + slots;
  for (uint32_t i = threadIdx.x; i < slots; i += 1024) {
    id[i] = kNoHub;
    hits[i] = 0;
  }
  for (uint32_t i = threadIdx.x; i < kHubSlots; i += 1024) hubs[i] = kNoHub;
  __syncthreads();
  const uint64_t step = m / (sample / 2);
  for (uint32_t i = threadIdx.x; i < sample; i += 1024) {
    const uint64_t at = (i >> 1) * step;
    EdgeCursor cur;
    uint32_t x, other;
    cur.start(e, at);
    if (i & 1) cur.at(e, at, other, x);
    else cur.at(e, at, x, other);
    if (x == kNoHub) continue;
    uint32_t s = (x * 0x9E3779B1u) & (slots - 1);
    while (true) {  // ends: more slots than endpoints
      const uint32_t old = atomicCAS(&id[s], kNoHub, x);
      if (old == kNoHub || old == x) break;
      s = (s + 1) & (slots - 1);
    }
    if (atomicAdd(&hits[s], 1u) == kHubHits - 1) {
      uint32_t* b = hubs + hub_bucket(x);
      if (atomicCAS(b, kNoHub, x) != kNoHub) atomicCAS(b + 1, kNoHub, x);
    }
  }
}

// The hub table of a list or batch (ids as EdgeIds gives them), or null.
const uint32_t* find_hubs(stc_ctx* c, const EdgeIds& e, uint64_t m) {
  if (m < kHubMinEdges) return nullptr;
  const uint32_t sample = hub_sample(m);
  uint32_t* hubs = buffer<uint32_t>(c, B_HUBS, kHubSlots);
  STC_CUDA(cudaFuncSetAttribute(k_find_hubs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)hub_smem(8192)));
  k_find_hubs<<<1, 1024, hub_smem(sample), c->stream>>>(e, m, sample, hubs);
  c->launches++;
  return hubs;
}

// `hubs` (kHub only): k_find_hubs's table.  Ids at or past n only reach here
// when a capped build's union outgrew its capacity (flagged by
// k_batch_bases).
template <bool kHub>
__global__ void __launch_bounds__(kThreads) k_degree_raw(EdgeIds e, uint64_t m,
                                                         uint32_t edge_chunk, uint32_t shift,
                                                         uint32_t n,
                                                         const uint32_t* __restrict__ hubs,
                                                         uint32_t* __restrict__ deg) {
  __shared__ __align__(8) uint32_t hid[kHub ? kHubSlots : 2], hcnt[kHub ? kHubSlots : 2];
  if (kHub) {
    for (uint32_t i = threadIdx.x; i < kHubSlots; i += kThreads) {
      hid[i] = hubs[i];
      hcnt[i] = 0;
    }
    __syncthreads();
  }
  auto add = [&](uint32_t x, bool valid) {
    if (kHub) {
      if (!valid) return;
      const uint32_t b = hub_bucket(x);
      const uint2 h = *reinterpret_cast<const uint2*>(hid + b);
      if (h.x == x) atomicAdd(&hcnt[b], 1u);
      else if (h.y == x) atomicAdd(&hcnt[b + 1], 1u);
      else atomicAdd(deg + x, 1u);
    } else {
      // A run of one id (a list sorted by source, a star) is added once.
      const uint32_t x0 = __shfl_sync(kFull, x, 0);
      const unsigned same = __ballot_sync(kFull, valid && x == x0);
      if (valid) {
        if (x != x0) atomicAdd(deg + x, 1u);
        else if ((same & lanemask_lt()) == 0) atomicAdd(deg + x, (uint32_t)__popc(same));
      }
    }
  };
  for (uint64_t begin = (uint64_t)blockIdx.x * edge_chunk; begin < m;
       begin += (uint64_t)gridDim.x * edge_chunk) {
    const uint64_t end = begin + edge_chunk < m ? begin + edge_chunk : m;
    EdgeCursor cur;
    cur.start(e, begin);
    for (uint64_t t = begin; t < end; t += kEdgeItems * kThreads) {
      uint32_t a[kEdgeItems], b[kEdgeItems];
#pragma unroll
      for (int r = 0; r < kEdgeItems; r++) {
        const uint64_t i = t + (uint64_t)r * kThreads + threadIdx.x;
        a[r] = b[r] = 0;  // a self-loop: skipped
        if (i < end) cur.at(e, i, a[r], b[r]);
      }
#pragma unroll
      for (int r = 0; r < kEdgeItems; r++) {
        const bool valid = a[r] != b[r] && a[r] < n && b[r] < n && sampled_edge(a[r], b[r], shift);
        add(a[r], valid);
        add(b[r], valid);
      }
    }
  }
  if (kHub) {
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < kHubSlots; i += kThreads)
      if (hcnt[i]) atomicAdd(deg + hid[i], hcnt[i]);
  }
}

// Degrees as 8-bit sort digits: exact below 16, then eight steps per power of
// two.  (degree step, id) is as good an order as (degree, id): the
// intersection work at RMAT scale 20 grows by 0.2%, on sparse graphs not at
// all, and the vertices sort in one 8-bit pass whatever the largest degree,
// which need not be known on the host.
__device__ __forceinline__ uint32_t degree_digit(uint32_t d) {
  if (d < 16) return d;
  const uint32_t bw = 32 - __clz(d);
  return 16 + 8 * (bw - 5) + ((d >> (bw - 4)) & 7u);
}

// One graph's ranks in (degree digit, id) order without moving a key: the
// counts of the digits, then one pass like the radix sort's whose output is
// each vertex's position.  ws is a sort workspace; the last CTA of the count
// turns the counts into each digit's first rank.  From 2^30 vertices on the
// tile states are 64 bits wide, as the sort's.
constexpr int kRankItems = 16;
constexpr uint32_t kRankTile = kSortThreads * kRankItems;

inline size_t rank_workspace_words(uint32_t n) {
  const uint64_t tiles = ((uint64_t)n + kRankTile - 1) / kRankTile;
  return kSortStates + (size_t)kRadix * tiles * (sort_wide(n) ? 2 : 1);
}

__global__ void __launch_bounds__(kSortThreads) k_degree_hist(const uint32_t* __restrict__ deg,
                                                              uint32_t n, uint32_t* __restrict__ ws) {
  __shared__ uint32_t hist[kRadix];
  __shared__ uint32_t scan_tmp[kSortWarps + 1];
  __shared__ bool s_last;
  const uint32_t tid = threadIdx.x;
  hist[tid] = 0;
  __syncthreads();
  for (uint64_t i = (uint64_t)blockIdx.x * kSortThreads + tid; i < n;
       i += (uint64_t)gridDim.x * kSortThreads)
    atomicAdd(&hist[degree_digit(deg[i])], 1u);
  __syncthreads();
  if (hist[tid]) atomicAdd(ws + tid, hist[tid]);
  __threadfence();
  __syncthreads();
  if (tid == 0) s_last = atomicAdd(ws + kSortDone, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  uint32_t total;
  const uint32_t c = __ldcg(ws + tid);
  ws[tid] = block_exclusive_scan<kSortThreads>(c, scan_tmp, total);
}

template <class W>
__global__ void __launch_bounds__(kSortThreads, 4) k_degree_rank(const uint32_t* __restrict__ deg,
                                                                 uint32_t n, uint32_t* __restrict__ ws,
                                                                 uint32_t* __restrict__ rank,
                                                                 unsigned long long* __restrict__ err) {
  using TS = TileState<W>;
  __shared__ uint32_t mask[2][kSortWarps][kRadix];
  __shared__ uint32_t whist[kSortWarps][kRadix];
  __shared__ uint32_t s_tile, s_abort;
  const uint32_t tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  if (tid == 0) {
    s_tile = atomicAdd(ws + kSortTickets, 1u);
    s_abort = 0;
  }
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) {
    whist[w][tid] = 0;
    mask[0][w][tid] = 0;
    mask[1][w][tid] = 0;
  }
  __syncthreads();
  const uint32_t tile = s_tile, begin = tile * kRankTile;
  if (begin >= n) return;
  const uint32_t valid = min(n - begin, kRankTile);
  const uint32_t wbase = warp * (32 * kRankItems) + lane;
  uint64_t k[kRankItems];  // digits
  uint32_t r[kRankItems / 2];
#pragma unroll
  for (int j = 0; j < kRankItems; j++)
    k[j] = wbase + 32 * j < valid ? degree_digit(deg[begin + wbase + 32 * j]) : 0u;
  if (valid == kRankTile)
    rank_keys<kRankItems, false, true>(k, wbase, valid, 0, kRadix - 1, mask, whist[warp], r);
  else
    rank_keys<kRankItems, false, false>(k, wbase, valid, 0, kRadix - 1, mask, whist[warp], r);
  __syncthreads();
  uint32_t cnt = 0, c[kSortWarps];
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) {
    c[w] = whist[w][tid];
    cnt += c[w];
  }
  if (tid == kRadix - 1) cnt -= kRankTile - valid;  // past the end: the last digit
  W* own = reinterpret_cast<W*>(ws + kSortStates) + (size_t)tile * kRadix + tid;
  TS::put(own, (tile == 0 ? TS::kPrefix : TS::kLocal) | cnt);
  uint32_t run = ws[tid] + (uint32_t)look_back(own, tile, cnt, ws, s_abort);
#pragma unroll
  for (int w = 0; w < kSortWarps; w++) {
    whist[w][tid] = run;
    run += c[w];
  }
  __syncthreads();
  if (s_abort && tid == 0) atomicExch(err, (unsigned long long)kDeviceErrTimeout);
#pragma unroll
  for (int j = 0; j < kRankItems; j++) {
    const uint32_t i = wbase + 32 * j;
    if (i < valid)  // an expired wait leaves a rank below n all the same
      rank[begin + i] = s_abort ? begin + i
                                : whist[warp][(uint32_t)k[j]] + ((r[j / 2] >> (16 * (j & 1))) & 0xFFFFu);
  }
}

// Arc keys of the input's edge copies in rank space: (rank lo << bits |
// rank hi), the negative flag in bit 63; a self-loop becomes the all-ones
// sentinel of the 2 * bits window, which sorts after every real key.  An
// endpoint at or past n (a capped build whose union outgrew its capacity)
// also becomes the sentinel and sets C_OVERFLOW.
__global__ void __launch_bounds__(kThreads) k_arc_keys_raw(
    EdgeIds e, const int8_t* __restrict__ sign, uint64_t m, uint32_t edge_chunk, uint32_t bits,
    uint32_t n, const uint32_t* __restrict__ rank, uint64_t* __restrict__ akeys,
    unsigned long long* __restrict__ ctr) {
  const uint64_t sentinel = (bits * 2 >= 64) ? ~0ull >> 1 : ((1ull << (2 * bits)) - 1);
  for (uint64_t begin = (uint64_t)blockIdx.x * edge_chunk; begin < m;
       begin += (uint64_t)gridDim.x * edge_chunk) {
    const uint64_t end = begin + edge_chunk < m ? begin + edge_chunk : m;
    EdgeCursor cur;
    cur.start(e, begin);
    for (uint64_t t = begin + threadIdx.x; t < end; t += kEdgeItems * kThreads) {
      uint32_t a[kEdgeItems], b[kEdgeItems], neg = 0;
#pragma unroll
      for (int r = 0; r < kEdgeItems; r++) {
        const uint64_t i = t + (uint64_t)r * kThreads;
        a[r] = b[r] = 0;
        if (i < end) {
          cur.at(e, i, a[r], b[r]);
          neg |= (uint32_t)(sign[i] < 0) << r;
        }
      }
      uint32_t ra[kEdgeItems], rb[kEdgeItems];
#pragma unroll
      for (int r = 0; r < kEdgeItems; r++) {
        const bool in = a[r] != b[r] && a[r] < n && b[r] < n;
        ra[r] = in ? rank[a[r]] : 0u;
        rb[r] = in ? rank[b[r]] : 0u;  // equal: no key
      }
#pragma unroll
      for (int r = 0; r < kEdgeItems; r++) {
        const uint64_t i = t + (uint64_t)r * kThreads;
        if (i >= end) break;
        if (a[r] >= n || b[r] >= n) atomicExch(ctr + C_OVERFLOW, 1ull);
        akeys[i] = ra[r] == rb[r] ? sentinel
                                  : ((uint64_t)min(ra[r], rb[r]) << bits) | max(ra[r], rb[r]) |
                                        ((uint64_t)((neg >> r) & 1u) << 63);
      }
    }
  }
}

// The first key of each run of equal (lo, hi) in the sorted arc keys becomes
// arc `pos` of the CSR: head, sign, tail and signed head.
struct EmitArc {
  const uint64_t* keys;
  uint32_t bits;
  uint32_t* nbr;
  int8_t* sgn;
  uint32_t* asrc;
  uint32_t* nkey;
  __device__ void operator()(uint64_t i, uint64_t pos, uint32_t flag) const {
    if (!flag) return;
    const uint64_t k = keys[i];
    const uint64_t idmask = (1ull << bits) - 1;
    const uint32_t head = (uint32_t)(k & idmask);
    nbr[pos] = head;
    sgn[pos] = (k >> 63) ? (int8_t)-1 : (int8_t)1;
    asrc[pos] = (uint32_t)((k >> bits) & idmask);
    nkey[pos] = (head << 1) | (uint32_t)(k >> 63);
  }
};

// Out-degree of every tail from the sorted arcs: lanes take consecutive
// arcs, so a warp adds each run of equal tails with one atomic.  With m_dev,
// m is a capacity and *m_dev the arc count.
__global__ void k_fdeg_count(const uint32_t* __restrict__ asrc, uint64_t m,
                             const unsigned long long* __restrict__ m_dev,
                             uint32_t* __restrict__ fdeg) {
  if (m_dev) m = min(m, (uint64_t)*m_dev);
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < m;
       base += stride) {
    const uint64_t p = base + lane_id();
    const uint32_t t = p < m ? asrc[p] : 0xFFFFFFFFu;
    const unsigned peers = __match_any_sync(kFull, t);
    if (p < m && (peers & lanemask_lt()) == 0) atomicAdd(fdeg + t, (uint32_t)__popc(peers));
  }
}

// The merge-model and probe-model bytes of every arc (arc_bytes); m_dev as
// in k_fdeg_count.
__global__ void k_alg_bytes(const uint32_t* __restrict__ asrc, const uint32_t* __restrict__ nbr,
                            uint64_t m, const unsigned long long* __restrict__ m_dev,
                            const uint64_t* __restrict__ off, const uint32_t* __restrict__ fdeg,
                            unsigned long long* __restrict__ ctr) {
  if (device_failed(ctr + C_ERROR)) return;
  if (m_dev) m = min(m, (uint64_t)*m_dev);
  unsigned long long bytes = 0, probe = 0;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride)
    arc_bytes(i, asrc[i], nbr[i], off, fdeg, bytes, probe);
  bytes = warp_sum(bytes);
  probe = warp_sum(probe);
  if (lane_id() == 0 && bytes) {
    atomicAdd(ctr + C_ALG_BYTES, bytes);
    atomicAdd(ctr + C_PROBE_BYTES, probe);
  }
}

// Vertex bases of a capped batch build, on the device: vbase = exclusive
// prefix of the graphs' id spaces, vbase[G] = vertices of the union (also
// written to C_BATCH_N); a union larger than the capacity n sets C_OVERFLOW.
// One CTA of 1,024 threads, 1,024 graphs per step.
__global__ void __launch_bounds__(1024) k_batch_bases(const unsigned int* __restrict__ space,
                                                      uint32_t G, uint32_t n,
                                                      uint64_t* __restrict__ vbase,
                                                      unsigned long long* __restrict__ ctr) {
  __shared__ uint64_t warp_incl[32];
  __shared__ uint64_t carry;
  const uint32_t lane = lane_id(), w = threadIdx.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t b0 = 0; b0 < G; b0 += 1024) {
    const uint32_t i = b0 + threadIdx.x;
    const uint64_t x = i < G ? space[i] : 0;
    uint64_t v = x;  // inclusive scan within the warp
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint64_t y = __shfl_up_sync(kFull, v, d);
      if (lane >= (uint32_t)d) v += y;
    }
    if (lane == 31) warp_incl[w] = v;
    __syncthreads();
    if (w == 0) {
      uint64_t t = warp_incl[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint64_t y = __shfl_up_sync(kFull, t, d);
        if (lane >= (uint32_t)d) t += y;
      }
      warp_incl[lane] = t;
    }
    __syncthreads();
    const uint64_t before = carry + (w ? warp_incl[w - 1] : 0) + v - x;
    if (i < G) vbase[i] = before;
    __syncthreads();
    if (threadIdx.x == 1023) carry = before + x;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    vbase[G] = carry;
    ctr[C_BATCH_N] = carry;
    if (carry > n) ctr[C_OVERFLOW] = 1;
  }
}

// Vertex sort keys of a batch's totals build: graph << (32 + dbits) | degree
// digit (its top dbits bits) << 32 | id; vertices past the union (vbase[G] <=
// i < n, a capped build) take all-ones graph and degree bits and so rank
// last.
__global__ void k_batch_vertex_keys(const uint32_t* __restrict__ deg, uint32_t n,
                                    const uint64_t* __restrict__ vbase, uint32_t G,
                                    uint64_t per_cta, uint32_t dbits, uint32_t gbits,
                                    uint64_t* __restrict__ vkeys) {
  const uint64_t begin = (uint64_t)blockIdx.x * per_cta;
  const uint64_t end = begin + per_cta < n ? begin + per_cta : n;
  if (begin >= end) return;
  const uint64_t nreal = vbase[G];
  const uint64_t pad = ((1ull << (dbits + gbits)) - 1) << 32;
  uint32_t g = begin < nreal ? first_segment(vbase, G, begin) : 0;
  for (uint64_t i = begin + threadIdx.x; i < end; i += blockDim.x) {
    if (i >= nreal) {
      vkeys[i] = pad | i;
      continue;
    }
    while (vbase[g + 1] <= i) g++;
    const uint64_t d = degree_digit(deg[i]) >> (8 - dbits);
    vkeys[i] = (gbits ? (uint64_t)g << (32 + dbits) : 0ull) | (d << 32) | i;
  }
}

// UniqueFlag over all m sorted arc keys, the self-loop sentinels (sorted
// last, all ones in the 2 * bits window) excluded: a capped build does not
// know m_valid on the host.
struct UniqueArcFlag {
  const uint64_t* keys;
  uint64_t mask;
  __device__ uint32_t operator()(uint64_t i) const {
    const uint64_t k = keys[i] & mask;
    if (k == mask) return 0u;
    if (i == 0) return 1u;
    return k != (keys[i - 1] & mask) ? 1u : 0u;
  }
};

// Steps 2-6 of the totals path, after the ids (g.n, g.bits, g.m_valid set):
// degrees over the edge copies (sampled on dense graphs; `hubs` is
// k_find_hubs's table or null), (degree digit, id) rank (graph-major for a
// batch with vertex bases d_vbase), arc keys of every copy, their sort, the
// first of each run of equal arcs, offsets.  g.ukeys and g.verts stay null.
// With `caps` (a batch whose sizes stay on the device) nothing is read back:
// g.n is the vertex capacity, the sample shift comes from caps, and g.m_fwd
// is the arc capacity (m) with the arc count in C_BATCH_MU (g.m_dev).
void build_totals(stc_ctx* c, const EdgeIds& e, const int8_t* d_sign, uint64_t m, DeviceGraph& g,
                  const uint64_t* d_vbase, uint32_t G, const uint32_t* hubs = nullptr,
                  const BatchCaps* caps = nullptr) {
  cudaStream_t st = c->stream;
  unsigned long long* ctr = (unsigned long long*)counters(c);
  const SortSpace sort_ws =
      sort_space(c, std::max<uint64_t>(m, g.n), rank_workspace_words(g.n));
  uint64_t* sums = buffer<uint64_t>(c, B_SCAN_SUMS, kScanSums);
  g.ukeys = nullptr;
  g.deg = buffer<uint32_t>(c, B_DEG, g.n);
  g.rank = buffer<uint32_t>(c, B_RANK, g.n);
  g.fdeg = buffer<uint32_t>(c, B_FDEG, g.n);
  if (g.n) {
    STC_CUDA(cudaMemsetAsync(g.deg, 0, (size_t)g.n * sizeof(uint32_t), st));
    STC_CUDA(cudaMemsetAsync(g.fdeg, 0, (size_t)g.n * sizeof(uint32_t), st));
  }
  if (g.m_valid) {
    // Sample 1 in 2^shift edges once the average degree reaches 8 (2 m / n
    // >= 8): shift = bit width of m / n, less 2, at most 3.  (From degree 16
    // on the 1,024-graph batch counted 6 ms slower and built 17 ms faster;
    // RMAT scale 24 moved by under 0.5 ms either way.)  Degrees that outgrow
    // L2 cost a DRAM access each, which outweighs a sparse graph's better
    // order: with 2^26 vertices and 2^27 edges, shift 0 / 1 / 2 / 3 took 6.7 /
    // 3.6 / 2.0 / 1.2 ms here and 5.0 / 5.6 / 5.7 / 5.8 ms to count.
    const uint64_t ratio = g.m_valid / std::max<uint64_t>(1, g.n);
    const uint32_t bw = bit_width64(ratio);
    g.shift = bw > 2 ? std::min<uint32_t>(3, bw - 2) : 0;
    if (g.n > 1u << 24) g.shift = std::max<uint32_t>(g.shift, g.n > 1u << 25 ? 3 : 2);
    if (caps) g.shift = caps->shift;
    auto kernel = hubs ? k_degree_raw<true> : k_degree_raw<false>;
    kernel<<<edge_grid(m), kThreads, 0, st>>>(e, m, edge_chunk(m), g.shift, g.n, hubs, g.deg);
    c->launches++;
  }
  STC_CUDA(cudaGetLastError());
  mark(c, 2);

  if (g.n && !d_vbase) {
    const uint32_t tiles = (uint32_t)(((uint64_t)g.n + kRankTile - 1) / kRankTile);
    STC_CUDA(cudaMemsetAsync(sort_ws.words, 0, rank_workspace_words(g.n) * sizeof(uint32_t), st));
    k_degree_hist<<<grid_for(g.n, 16), kSortThreads, 0, st>>>(g.deg, g.n, sort_ws.words);
    auto rank = sort_wide(g.n) ? k_degree_rank<uint64_t> : k_degree_rank<uint32_t>;
    rank<<<tiles, kSortThreads, 0, st>>>(g.deg, g.n, sort_ws.words, g.rank, sort_error(c));
    c->launches += 2;
  } else if (g.n) {
    uint64_t* va = buffer<uint64_t>(c, B_VKEYS_A, g.n);
    uint64_t* vb = buffer<uint64_t>(c, B_VKEYS_B, g.n);
    const uint32_t gbits = bit_width64(G > 1 ? G - 1 : 0);
    const uint32_t dbits = std::min<uint32_t>(8, 32 - gbits);
    const RangePartition vp = range_partition(g.n, kSortTile, kMaxSortGrid);
    k_batch_vertex_keys<<<vp.grid, kThreads, 0, st>>>(g.deg, g.n, d_vbase, G, vp.per_cta, dbits,
                                                      gbits, va);
    uint64_t* vs = radix_sort(va, vb, g.n, 32, (int)(32 + dbits + gbits), sort_ws, sort_error(c), st,
                              &c->launches);
    k_rank<<<grid_for(g.n, 4), kThreads, 0, st>>>(vs, g.n, nullptr, g.rank, sort_error(c));
    c->launches += 2;
  }
  STC_CUDA(cudaGetLastError());
  mark(c, 3);

  g.m_unique = g.m_fwd = 0;
  if (g.m_valid) {
    uint64_t* ka = buffer<uint64_t>(c, B_KEYS_A, m);
    uint64_t* kb = buffer<uint64_t>(c, B_KEYS_B, m);
    wait_sign(c);  // a host sign array may still be on its way (stc_count)
    k_arc_keys_raw<<<edge_grid(m), kThreads, 0, st>>>(e, d_sign, m, edge_chunk(m), g.bits, g.n,
                                                      g.rank, ka, ctr);
    c->launches++;
    uint64_t* sorted = radix_sort(ka, kb, m, 0, 2 * (int)g.bits, sort_ws, sort_error(c), st, &c->launches);
    const uint64_t mask = (1ull << (2 * g.bits)) - 1;
    if (caps) {
      const UniqueArcFlag flag{sorted, mask};
      // No arcs after an expired wait: the kernels below are bounded by their number.
      const uint32_t grid = range_reduce_scan(flag, m, sums, st, &c->launches, sort_error(c));
      STC_CUDA(cudaMemcpyAsync(ctr + C_BATCH_MU, sums + grid, sizeof(uint64_t),
                               cudaMemcpyDeviceToDevice, st));
      g.m_unique = g.m_fwd = m;
      g.m_dev = ctr + C_BATCH_MU;
      g.nbr = buffer<uint32_t>(c, B_NBR, m + 8);
      g.sgn = buffer<int8_t>(c, B_SGN, m + 8);
      g.asrc = buffer<uint32_t>(c, B_ASRC, m);
      g.nkey = buffer<uint32_t>(c, B_NKEY, m + 8);
      range_apply(flag, EmitArc{sorted, g.bits, g.nbr, g.sgn, g.asrc, g.nkey}, m, sums, st,
                  &c->launches);
    } else {
      // Self-loops sorted last: the first m_valid keys are the real arcs.
      const UniqueFlag flag{sorted, mask};
      const uint32_t grid =
          range_reduce_scan(flag, g.m_valid, sums, st, &c->launches, sort_error(c));
      g.m_unique = g.m_fwd = read_total(c, sums, grid);
      g.nbr = buffer<uint32_t>(c, B_NBR, g.m_fwd + 8);  // + 8: the engine reads whole 32-byte chunks
      g.sgn = buffer<int8_t>(c, B_SGN, g.m_fwd + 8);
      g.asrc = buffer<uint32_t>(c, B_ASRC, g.m_fwd);
      g.nkey = buffer<uint32_t>(c, B_NKEY, g.m_fwd + 8);
      range_apply(flag, EmitArc{sorted, g.bits, g.nbr, g.sgn, g.asrc, g.nkey}, g.m_valid, sums,
                  st, &c->launches);
    }
    k_fdeg_count<<<grid_for(g.m_fwd, 4), kThreads, 0, st>>>(g.asrc, g.m_fwd, g.m_dev, g.fdeg);
    c->launches++;
  }
  g.off = buffer<uint64_t>(c, B_OFF, (size_t)g.n + 1);
  if (g.n) {
    range_scan(LoadU32{g.fdeg}, EmitOffset{g.off}, g.n, sums, st, &c->launches);
    STC_CUDA(cudaMemcpyAsync(g.off + g.n, sums + range_partition(g.n, kScanTile, kMaxSortGrid).grid,
                             sizeof(uint64_t), cudaMemcpyDeviceToDevice, st));
  } else {
    STC_CUDA(cudaMemsetAsync(g.off, 0, sizeof(uint64_t), st));
  }
  if (!g.m_fwd) {
    g.nbr = buffer<uint32_t>(c, B_NBR, 4);
    g.sgn = buffer<int8_t>(c, B_SGN, 4);
  }
  STC_CUDA(cudaGetLastError());
  mark(c, 4);
}

// ---------------------------------------------------- dense relabel ----
// Counts of totals accept any 32-bit id: an edge list whose largest id
// reaches 2^31 - 2 (the engine's signed keys and ranks stay below it)
// is relabelled to dense ids first, the index of each id among the list's
// distinct ids.  The relabelling keeps the ids' order, so the graph, its
// (degree, id) order and its counts are those of the original list.

// Both endpoints of every edge as 64-bit sort keys.
__global__ void k_endpoint_keys(const uint32_t* __restrict__ u, const uint32_t* __restrict__ v,
                                uint64_t m, uint64_t* __restrict__ keys) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride) {
    keys[2 * i] = u[i];
    keys[2 * i + 1] = v[i];
  }
}

struct DistinctEmit {
  const uint64_t* keys;
  uint32_t* out;
  __device__ void operator()(uint64_t i, uint64_t pos, uint32_t flag) const {
    if (flag) out[pos] = (uint32_t)keys[i];
  }
};

__device__ __forceinline__ uint32_t dense_id(const uint32_t* __restrict__ ids, uint32_t nd,
                                             uint32_t x) {
  uint32_t lo = 0, hi = nd;  // first index with ids[index] >= x (x is present)
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (ids[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo;
}

__global__ void k_relabel(const uint32_t* __restrict__ u, const uint32_t* __restrict__ v,
                          uint64_t m, const uint32_t* __restrict__ ids, uint32_t nd,
                          uint32_t* __restrict__ ou, uint32_t* __restrict__ ov) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += stride) {
    ou[i] = dense_id(ids, nd, u[i]);
    ov[i] = dense_id(ids, nd, v[i]);
  }
}

// Relabels the m edges at (*src, *dst) to dense ids in context buffers and
// points *src / *dst at them; returns the number of distinct ids.
uint64_t relabel_dense(stc_ctx* c, const uint32_t** src, const uint32_t** dst, uint64_t m) {
  cudaStream_t st = c->stream;
  if (2 * m >= (1ull << 32))  // both endpoints of every edge in one sort
    fail(STC_ERR_LIMIT, "an edge list with ids from 2^31 - 2 on has 2^31 or more elements");
  const SortSpace sort_ws = sort_space(c, 2 * m);
  uint64_t* sums = buffer<uint64_t>(c, B_SCAN_SUMS, kScanSums);
  uint64_t* ka = buffer<uint64_t>(c, B_KEYS_A, 2 * m);
  uint64_t* kb = buffer<uint64_t>(c, B_KEYS_B, 2 * m);
  k_endpoint_keys<<<grid_for(m, 4), kThreads, 0, st>>>(*src, *dst, m, ka);
  c->launches++;
  const uint64_t* sorted = radix_sort(ka, kb, 2 * m, 0, 32, sort_ws, sort_error(c), st, &c->launches);
  const UniqueFlag flag{sorted, 0xFFFFFFFFull};
  const uint32_t grid = range_reduce_scan(flag, 2 * m, sums, st, &c->launches, sort_error(c));
  const uint64_t nd = read_total(c, sums, grid);
  if (nd > kMaxVertices)
    fail(STC_ERR_LIMIT, std::to_string(nd) + " distinct vertex ids >= 2^31 - 1");
  uint32_t* ids = buffer<uint32_t>(c, B_DISTINCT, nd);
  range_apply(flag, DistinctEmit{sorted, ids}, 2 * m, sums, st, &c->launches);
  uint32_t* out = buffer<uint32_t>(c, B_RELABEL, 2 * m);
  k_relabel<<<grid_for(m, 4), kThreads, 0, st>>>(*src, *dst, m, ids, (uint32_t)nd, out, out + m);
  c->launches++;
  STC_CUDA(cudaGetLastError());
  *src = out;
  *dst = out + m;
  return nd;
}

}  // namespace

void algorithmic_bytes(stc_ctx* c, const DeviceGraph& g) {
  k_alg_bytes<<<grid_for(g.m_fwd, 4), kThreads, 0, c->stream>>>(
      g.asrc, g.nbr, g.m_fwd, g.m_dev, g.off, g.fdeg, (unsigned long long*)counters(c));
  c->launches++;
  STC_CUDA(cudaGetLastError());
}

void build_graph(stc_ctx* c, const uint32_t* d_src, const uint32_t* d_dst, const int8_t* d_sign,
                 uint64_t m, DeviceGraph& g, bool totals) {
  cudaStream_t st = c->stream;
  unsigned long long* ctr = (unsigned long long*)counters(c);
  g = DeviceGraph{};
  g.m_input = m;
  if (m >= (1ull << 32)) fail(STC_ERR_LIMIT, "edge list has 2^32 or more elements");

  // 1. ids: max kept id and self-loops.
  mark(c, 1);
  if (m) {
    k_scan_ids<<<grid_for(m, 4), kThreads, 0, st>>>(d_src, d_dst, m, ctr);
    c->launches++;
  }
  // The hubs are found while the host waits for the ids.
  STC_CUDA(cudaMemcpyAsync(c->h_pinned + C_MAX_ID, counters(c) + C_MAX_ID, 2 * sizeof(uint64_t),
                           cudaMemcpyDeviceToHost, st));
  STC_CUDA(cudaEventRecord(c->ev_read, st));
  const uint32_t* hubs =
      totals ? find_hubs(c, EdgeIds{d_src, d_dst, nullptr, nullptr, 0}, m) : nullptr;
  STC_CUDA(cudaEventSynchronize(c->ev_read));
  uint64_t max_id = c->h_pinned[C_MAX_ID];
  const uint64_t self = c->h_pinned[C_SELF];
  // Ranks stay below 2^31 - 2 where triangles are counted (kMaxVertices).
  // Counts of totals relabel larger ids to dense ones; the other paths report
  // by id and refuse them, 2^31 - 2 itself only where they count (a forward
  // CSR may hold it).
  if (!totals && max_id > kMaxVertices)
    fail(STC_ERR_LIMIT, "vertex id " + std::to_string(max_id) + " >= 2^31 - 1");
  if (max_id >= kMaxVertices && totals) {
    max_id = relabel_dense(c, &d_src, &d_dst, m) - 1;
    hubs = nullptr;  // named by the ids of the list as given
  }
  g.n = m ? (uint32_t)max_id + 1 : 0;
  g.m_valid = m - self;
  g.bits = std::max<uint32_t>(1, bit_width64(max_id));
  if (totals) {
    build_totals(c, EdgeIds{d_src, d_dst, nullptr, nullptr, 0}, d_sign, m, g, nullptr, 0, hubs);
    return;
  }
  const SortSpace sort_ws = sort_space(c, std::max<uint64_t>(m, g.n));
  uint64_t* sums = buffer<uint64_t>(c, B_SCAN_SUMS, kScanSums);

  // 2. dedup.
  uint64_t* ka = buffer<uint64_t>(c, B_KEYS_A, m);
  uint64_t* kb = buffer<uint64_t>(c, B_KEYS_B, m);
  g.ukeys = buffer<uint64_t>(c, B_UKEYS, g.m_valid);
  if (g.m_valid) {
    wait_sign(c);
    k_pack_dedup<<<grid_for(m, 4), kThreads, 0, st>>>(d_src, d_dst, d_sign, m, g.bits, ka);
    c->launches++;
    uint64_t* sorted = radix_sort(ka, kb, m, 0, 2 * (int)g.bits, sort_ws, sort_error(c), st, &c->launches);
    const uint64_t mask = (1ull << (2 * g.bits)) - 1;
    const UniqueFlag flag{sorted, mask};
    const uint32_t grid =
        range_reduce_scan(flag, g.m_valid, sums, st, &c->launches, sort_error(c));
    range_apply(flag, UniqueEmit{sorted, g.ukeys}, g.m_valid, sums, st, &c->launches);
    g.m_unique = read_total(c, sums, grid);
  }
  STC_CUDA(cudaGetLastError());
  mark(c, 2);

  // 3-4. degree and (degree, id) rank.
  g.deg = buffer<uint32_t>(c, B_DEG, g.n);
  g.rank = buffer<uint32_t>(c, B_RANK, g.n);
  g.verts = buffer<uint32_t>(c, B_VERTS, g.n);
  g.fdeg = buffer<uint32_t>(c, B_FDEG, g.n);
  if (g.n) {
    STC_CUDA(cudaMemsetAsync(g.deg, 0, (size_t)g.n * sizeof(uint32_t), st));
    STC_CUDA(cudaMemsetAsync(g.fdeg, 0, (size_t)g.n * sizeof(uint32_t), st));
    if (g.m_unique) {
      k_degree<<<grid_for(g.m_unique, 16), kThreads, 0, st>>>(g.ukeys, g.m_unique, g.bits, g.deg);
      c->launches++;
    }
    uint64_t* va = buffer<uint64_t>(c, B_VKEYS_A, g.n);
    uint64_t* vb = buffer<uint64_t>(c, B_VKEYS_B, g.n);
    k_vertex_keys<<<grid_for(g.n, 4), kThreads, 0, st>>>(g.deg, g.n, va, ctr);
    c->launches++;
    read_counters(c, C_MAX_DEG, 1);
    g.max_deg = (uint32_t)c->h_pinned[C_MAX_DEG];
    uint64_t* vs = radix_sort(va, vb, g.n, 32, 32 + (int)bit_width64(g.max_deg), sort_ws, sort_error(c), st,
                              &c->launches);
    k_rank<<<grid_for(g.n, 4), kThreads, 0, st>>>(vs, g.n, g.verts, g.rank, sort_error(c));
    c->launches++;
  }
  STC_CUDA(cudaGetLastError());
  mark(c, 3);

  // 5-6. orientation into rank space and the forward CSR.
  g.m_fwd = g.m_unique;
  if (g.m_fwd) {
    k_arc_keys<<<grid_for(g.m_fwd, 4), kThreads, 0, st>>>(g.ukeys, g.m_fwd, g.bits, g.rank, ka,
                                                          g.fdeg, sort_error(c));
    c->launches++;
    finish_csr_from_arc_keys(c, g, ka, kb);
  } else {
    g.off = buffer<uint64_t>(c, B_OFF, (size_t)g.n + 1);
    STC_CUDA(cudaMemsetAsync(g.off, 0, ((size_t)g.n + 1) * sizeof(uint64_t), st));
    g.nbr = buffer<uint32_t>(c, B_NBR, 1);
    g.sgn = buffer<int8_t>(c, B_SGN, 1);
  }
  mark(c, 4);
}

void graph_from_forward_csr(stc_ctx* c, uint32_t n, uint64_t m, const uint64_t* d_off,
                            const uint32_t* d_edges, const int8_t* d_signs, const uint32_t* d_rank,
                            DeviceGraph& g) {
  cudaStream_t st = c->stream;
  unsigned long long* ctr = (unsigned long long*)counters(c);
  g = DeviceGraph{};
  g.n = n;
  g.m_input = g.m_valid = g.m_unique = g.m_fwd = m;
  if (m >= (1ull << 32)) fail(STC_ERR_LIMIT, "forward CSR has 2^32 or more edges");
  if (n > kMaxVertices) fail(STC_ERR_LIMIT, "forward CSR has 2^31 - 1 or more vertices");
  g.bits = std::max<uint32_t>(1, bit_width64(n ? n - 1 : 0));
  g.rank = const_cast<uint32_t*>(d_rank);
  g.fdeg = buffer<uint32_t>(c, B_FDEG, n);
  mark(c, 1);
  mark(c, 2);
  mark(c, 3);
  uint64_t* ka = buffer<uint64_t>(c, B_KEYS_A, m);
  uint64_t* kb = buffer<uint64_t>(c, B_KEYS_B, m);
  if (n) {
    uint32_t* seen = buffer<uint32_t>(c, B_DEG, n);
    STC_CUDA(cudaMemsetAsync(seen, 0, (size_t)n * sizeof(uint32_t), st));
    k_csr_arc_keys<<<kSMs * 8, kThreads, 0, st>>>(d_off, d_edges, d_signs, d_rank, n, m, g.bits, ka,
                                                  g.fdeg, seen, ctr);
    c->launches++;
    read_counters(c, C_ERROR, 1);
    if (c->h_pinned[C_ERROR] == kDeviceErrCsr) {
      fail(STC_ERR_INVALID_ARGUMENT,
           "not a forward CSR: offsets decrease, rank is not a permutation of [0, n), an edge does "
           "not go from lower to higher rank, or an id is >= n");
    }
    check_device_error(c->h_pinned[C_ERROR]);
  }
  if (m) {
    finish_csr_from_arc_keys(c, g, ka, kb);
  } else {
    g.off = buffer<uint64_t>(c, B_OFF, (size_t)n + 1);
    STC_CUDA(cudaMemsetAsync(g.off, 0, ((size_t)n + 1) * sizeof(uint64_t), st));
    g.nbr = buffer<uint32_t>(c, B_NBR, 1);
    g.sgn = buffer<int8_t>(c, B_SGN, 1);
  }
  mark(c, 4);
}

void build_graph_batch(stc_ctx* c, const uint32_t* d_src, const uint32_t* d_dst,
                       const int8_t* d_sign, uint64_t m, const uint64_t* h_eoff, uint32_t G,
                       DeviceGraph& g) {
  cudaStream_t st = c->stream;
  unsigned long long* ctr = (unsigned long long*)counters(c);
  g = DeviceGraph{};
  g.m_input = m;
  g.G = G;
  if (m >= (1ull << 32)) fail(STC_ERR_LIMIT, "batch has 2^32 or more edges");
  uint64_t* d_eoff = buffer<uint64_t>(c, B_BATCH_META, 2ull * (G + 1));
  uint64_t* d_vbase = d_eoff + (G + 1);
  unsigned int* d_space = reinterpret_cast<unsigned int*>(buffer<uint32_t>(c, B_BATCH_SPACE, G));
  STC_CUDA(cudaMemcpyAsync(d_eoff, h_eoff, (G + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice, st));
  STC_CUDA(cudaMemsetAsync(d_space, 0, G * sizeof(uint32_t), st));

  // 1. id space per graph -> vertex bases of the union.
  mark(c, 1);
  const RangePartition ep = range_partition(m, kSortTile, kMaxSortGrid);
  if (m) {
    k_batch_ids<<<ep.grid, kThreads, 0, st>>>(d_src, d_dst, m, d_eoff, G, ep.per_cta, d_space, ctr);
    c->launches++;
  }
  std::vector<uint32_t> space(G);
  STC_CUDA(cudaMemcpyAsync(space.data(), d_space, G * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  read_counters(c, C_SELF, 1);
  std::vector<uint64_t> vbase(G + 1, 0);
  for (uint32_t i = 0; i < G; i++) vbase[i + 1] = vbase[i] + space[i];
  const uint64_t ntot = vbase[G];
  if (ntot > kMaxVertices)
    fail(STC_ERR_LIMIT, "batch has 2^31 - 1 or more vertices in total");
  STC_CUDA(cudaMemcpyAsync(d_vbase, vbase.data(), (G + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice,
                           st));
  g.n = (uint32_t)ntot;
  g.m_valid = m - c->h_pinned[C_SELF];
  g.bits = std::max<uint32_t>(1, bit_width64(ntot ? ntot - 1 : 0));
  g.gbase = d_vbase;
  const EdgeIds e{d_src, d_dst, d_eoff, d_vbase, G};
  build_totals(c, e, d_sign, m, g, d_vbase, G, find_hubs(c, e, m));
}

void build_graph_batch_capped(stc_ctx* c, const uint32_t* d_src, const uint32_t* d_dst,
                              const int8_t* d_sign, uint64_t m, uint32_t G, const BatchCaps& caps,
                              DeviceGraph& g) {
  cudaStream_t st = c->stream;
  unsigned long long* ctr = (unsigned long long*)counters(c);
  g = DeviceGraph{};
  g.m_input = m;
  g.G = G;
  if (m >= (1ull << 32)) fail(STC_ERR_LIMIT, "batch has 2^32 or more edges");
  if (caps.n == 0 || caps.n >= (1u << 31) - 1 || caps.bits != std::max<uint32_t>(1, bit_width64(caps.n - 1)))
    fail(STC_ERR_INTERNAL, "inconsistent batch capacities");
  if (!c->h_eoff || c->h_eoff_cap < (size_t)G + 1) fail(STC_ERR_INTERNAL, "edge offsets not staged");
  uint64_t* d_eoff = buffer<uint64_t>(c, B_BATCH_META, 2ull * (G + 1));
  uint64_t* d_vbase = d_eoff + (G + 1);
  unsigned int* d_space = reinterpret_cast<unsigned int*>(buffer<uint32_t>(c, B_BATCH_SPACE, G));
  STC_CUDA(cudaMemcpyAsync(d_eoff, c->h_eoff, (G + 1) * sizeof(uint64_t), cudaMemcpyHostToDevice,
                           st));
  STC_CUDA(cudaMemsetAsync(d_space, 0, G * sizeof(uint32_t), st));

  // 1. id space per graph -> vertex bases of the union, on the device.
  mark(c, 1);
  const RangePartition ep = range_partition(m, kSortTile, kMaxSortGrid);
  if (m) {
    k_batch_ids<<<ep.grid, kThreads, 0, st>>>(d_src, d_dst, m, d_eoff, G, ep.per_cta, d_space, ctr);
    c->launches++;
  }
  k_batch_bases<<<1, 1024, 0, st>>>(d_space, G, caps.n, d_vbase, ctr);
  c->launches++;
  STC_CUDA(cudaGetLastError());
  g.n = caps.n;
  g.m_valid = m;
  g.bits = caps.bits;
  g.gbase = d_vbase;
  const EdgeIds e{d_src, d_dst, d_eoff, d_vbase, G};
  build_totals(c, e, d_sign, m, g, d_vbase, G, find_hubs(c, e, m), &caps);
}

void export_forward_csr(stc_ctx* c, const DeviceGraph& g, stc_forward_csr* out) {
  cudaStream_t st = c->stream;
  const uint32_t n = g.n;
  const uint64_t mu = g.m_unique;
  uint32_t* fdeg_id = buffer<uint32_t>(c, B_EXPORT_FDEG, n);
  uint64_t* off_id = buffer<uint64_t>(c, B_EXPORT_OFF, (size_t)n + 1);
  uint64_t* ka = buffer<uint64_t>(c, B_KEYS_A, mu);
  uint64_t* kb = buffer<uint64_t>(c, B_KEYS_B, mu);
  const SortSpace sort_ws = sort_space(c, mu);
  uint64_t* sums = buffer<uint64_t>(c, B_SCAN_SUMS, kScanSums);
  uint32_t* edges = buffer<uint32_t>(c, B_NBR, mu);
  int8_t* signs = buffer<int8_t>(c, B_SGN, mu);
  if (n) STC_CUDA(cudaMemsetAsync(fdeg_id, 0, (size_t)n * sizeof(uint32_t), st));
  uint64_t* sorted = ka;
  if (mu) {
    k_export_keys<<<grid_for(mu, 4), kThreads, 0, st>>>(g.ukeys, mu, g.bits, g.rank, ka, fdeg_id);
    sorted = radix_sort(ka, kb, mu, 0, 2 * (int)g.bits, sort_ws, sort_error(c), st, &c->launches);
  }
  if (n) {
    range_scan(LoadU32{fdeg_id}, EmitOffset{off_id}, n, sums, st, &c->launches);
    STC_CUDA(cudaMemcpyAsync(off_id + n, sums + range_partition(n, kScanTile, kMaxSortGrid).grid,
                             sizeof(uint64_t), cudaMemcpyDeviceToDevice, st));
  }
  if (mu) {
    k_csr_fill<<<grid_for(mu, 4), kThreads, 0, st>>>(sorted, mu, g.bits, fdeg_id, off_id, edges,
                                                     signs, nullptr, nullptr,
                                                     (unsigned long long*)counters(c));
  }
  STC_CUDA(cudaGetLastError());
  out->n = n;
  out->m = mu;
  out->offsets = (uint64_t*)host_alloc(((size_t)n + 1) * sizeof(uint64_t));
  out->edges = (uint32_t*)host_alloc(mu * sizeof(uint32_t));
  out->signs = (int8_t*)host_alloc(mu);
  out->fdeg = (uint32_t*)host_alloc((size_t)n * sizeof(uint32_t));
  out->rank = (uint32_t*)host_alloc((size_t)n * sizeof(uint32_t));
  if (!out->offsets || !out->edges || !out->signs || !out->fdeg || !out->rank) {
    stc_free_forward_csr(out);
    fail(STC_ERR_OUT_OF_MEMORY, "host allocation for the forward CSR failed");
  }
  if (n == 0) out->offsets[0] = 0;
  download(c, {piece(off_id, out->offsets, n ? (size_t)n + 1 : 0), piece(fdeg_id, out->fdeg, n),
               piece(g.rank, out->rank, n), piece(edges, out->edges, mu),
               piece(signs, out->signs, mu)});
}

}  // namespace stc
