// Self-collision kernels: area-weighted normals, the spatial-hash counting
// sort (vertex and edge-midpoint keys), vertex-vertex / vertex-triangle
// contacts, multi-layer untangling, edge-edge contacts and the apply pass.
//
// Contacts accumulate into a per-vertex 16 x int32 record with integer
// atomics (fixed point x1e6), so results do not depend on thread order.
// The one order-dependent piece of the reference, the in-bucket order of the
// counting sort (atomic scatter, shaders/spatial_grid_sort.wgsl:182-194), is
// made canonical here: each bucket is sorted by ascending element index.
#pragma once
#include "solver_kernels.cuh"
#include "vmath.cuh"

namespace tcloth {

enum : int {
  A_DX, A_DY, A_DZ, A_CNT, A_PDX, A_PDY, A_PDZ, A_PCNT,
  A_CPX, A_CPY, A_CPZ, A_CNX, A_CNY, A_CNZ, A_UT, A_EEC, A_N
};

struct SCArgs {
  uint32_t n, ne, table;
  float cell;
  float relief;
  int enable_relief;
  float max_disp_ratio;
  int exclude_neighbors;
  int untangle;  // effective: option && multiple layers
  uint32_t max_search;
  const float4* x4;
  const float4* p4;
  const float4* v4;  // layer bits in .w
  const float* local_len;
  const uint32_t* adj_off;
  const uint32_t* adj_idx;
  const uint32_t* th_off;
  const uint32_t* th_idx;
  const float* th_rest;
  const uint32_t* star_off;
  const uint2* star_idx;
  const uint2* edges;
  const uint32_t* edge_bits;
  const uint32_t* cs;    // vertex cell starts (table + 1)
  const uint32_t* srt;   // vertex sorted indices
  const uint32_t* ecs;   // edge cell starts
  const uint32_t* esrt;  // edge sorted indices
  const float4* nrm;
  int32_t* acc;
  // per-substep caches written by the hash pass (same float operations as
  // the reference performs per candidate, done once per element)
  // per vertex j: bounding box of p over j and its star triangles' vertices,
  // and the range of their motion p - x: (lo, mlo.x), (hi, mlo.y), (mhi, mlo.z)
  const float4* sbox;
  // per star entry (j; v0, v1), aligned with star_idx: the triangle's box over
  // p and its mean motion as seen from j: (min, motion.x), (max, motion.y),
  // motion.z
  const float4* st_lo;
  const float4* st_hi;
  const float* st_mz;
  // vertices (edges) in Morton order of their initial positions (midpoints):
  // the order in which k_sc_solve (k_ee) works them
  const uint32_t* order;
  const uint32_t* eorder;
  const int4* vcell;    // floor(p / cell) per vertex
  const float* mlen;    // |p - x| per vertex
  const int4* ecell;    // floor(midpoint / cell) per edge
  const float4* eamin;  // min of both endpoints' p and x per edge
  const float4* eamax;
  // candidate records in hash-sorted order (slot k of the sorted arrays)
  const float4* vs_p;   // p, thickness of vertex srt[k]
  const int4* vs_c;     // cell, index of vertex srt[k]
  const float4* vs_q;   // local edge length, layer bits, inverse mass, |p - x| of vertex srt[k]
  const int4* es_c;     // cell, index of edge esrt[k]
  const uint2* es_v;    // endpoints of edge esrt[k]
  const float4* es_lo;  // swept AABB of edge esrt[k]; .w: bits of its first endpoint
  const float4* es_hi;  // .w: bits of its second endpoint
  // pairs that need the continuous (CCD) search are deferred to k_ee_ccd
  uint2* ccd_q;
  uint32_t* ccd_n;
  uint32_t ccd_cap;
  // (edge, edge) pairs counted by k_ee_cluster, worked one lane each by k_ee_pairs.
  // The list is split into kEeSeg segments of ee_cap / kEeSeg entries with a
  // counter each (ee_n[kEeSeg]); block b of k_ee_cluster appends to
  // segment b % kEeSeg, so that no one counter takes every warp's atomic.  A counter
  // may run past its segment's capacity (k_ee_pairs reads min(count, cap));
  // the pairs past it are worked inside the filter.
  uint2* ee_q;
  uint32_t* ee_n;
  uint32_t ee_cap;
  // optional record of the narrow-phase input (null when off): the
  // (vertex, triangle) pairs that pass the cheap tests of sc_solve and the
  // (edge, edge) pairs counted within max_search; rec_n[0] / rec_n[1] count
  // them, entries past the capacities are dropped
  uint4* rec_vt;
  uint2* rec_ee;
  uint32_t* rec_n;
  uint32_t rec_vt_cap, rec_ee_cap;
};

__device__ __forceinline__ void record_vt(const SCArgs& s, uint32_t i, uint32_t a, uint32_t b, uint32_t c) {
  const uint32_t k = atomicAdd(&s.rec_n[0], 1u);
  if (k < s.rec_vt_cap) s.rec_vt[k] = make_uint4(i, a, b, c);
}
__device__ __forceinline__ void record_ee(const SCArgs& s, uint32_t ea, uint32_t eb) {
  const uint32_t k = atomicAdd(&s.rec_n[1], 1u);
  if (k < s.rec_ee_cap) s.rec_ee[k] = make_uint2(ea, eb);
}

// A vertex's sorted two-hop list (and rest lengths), in shared memory when it
// fits, else in global memory; binary search as in
// shaders/self_collision.wgsl:243-293.
struct TwoHop {
  const uint32_t* idx;
  const float* rest;
  uint32_t n;
};
__device__ __forceinline__ bool th_find(const TwoHop& t, uint32_t b, uint32_t& pos) {
  uint32_t lo = 0, hi = t.n;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2u;
    const uint32_t v = t.idx[mid];
    if (v == b) { pos = mid; return true; }
    if (v < b) lo = mid + 1u; else hi = mid;
  }
  return false;
}
__device__ __forceinline__ bool near_folded_sq_t(const TwoHop& t, uint32_t a, uint32_t b, float d2) {
  uint32_t q;
  if (a == b) return true;
  if (!th_find(t, b, q)) return false;
  const float l0 = t.rest[q];
  return !(d2 < (l0 * l0) * 0.25f);
}
constexpr uint32_t kTwoHopCache = 64;
constexpr uint32_t kRounds = 4;  // candidates per warp chunk = 32 * kRounds
constexpr uint32_t kEeSeg = 256;       // segments of the E-E pair list
constexpr uint32_t kEePairBlocks = 4;  // k_ee_pairs blocks per segment
// Stage vertex v's two-hop list in shared memory (whole warp participates).
__device__ __forceinline__ TwoHop stage_two_hop(const uint32_t* th_off, const uint32_t* th_idx, const float* th_rest,
                                               uint32_t v, uint32_t* sh_idx, float* sh_rest, int lane) {
  const uint32_t b = th_off[v], e = th_off[v + 1];
  TwoHop t;
  t.n = e - b;
  if (t.n <= kTwoHopCache) {
    for (uint32_t k = lane; k < t.n; k += 32u) {
      sh_idx[k] = th_idx[b + k];
      sh_rest[k] = th_rest[b + k];
    }
    __syncwarp();
    t.idx = sh_idx;
    t.rest = sh_rest;
  } else {
    t.idx = th_idx + b;
    t.rest = th_rest + b;
  }
  return t;
}

__device__ __forceinline__ uint32_t layer_of(const float4* v4, uint32_t i) { return __float_as_uint(v4[i].w); }

// Star boxes and star-entry records for the vertex-triangle pass (see
// SCArgs::sbox, st_lo), and with nrm the area-weighted normals (k_normals, which
// reads the same positions): one thread per vertex over its star pairs.
__global__ void k_star_box(uint32_t n, const uint32_t* __restrict__ star_off, const uint2* __restrict__ star_idx,
                           const float4* __restrict__ x4, const float4* __restrict__ p4, float4* __restrict__ sbox,
                           float4* __restrict__ st_lo, float4* __restrict__ st_hi, float* __restrict__ st_mz,
                           float4* __restrict__ nrm) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const V3 pj = mk(p4[j]), pjo = mk(x4[j]);
  V3 lo = pj, hi = pj, mlo = pj - pjo, mhi = mlo, ns = mk(0.f, 0.f, 0.f);
  for (uint32_t k = star_off[j]; k < star_off[j + 1]; ++k) {
    const uint2 pr = star_idx[k];
    const V3 a = mk(p4[pr.x]), b = mk(p4[pr.y]);
    const V3 ao = mk(x4[pr.x]), bo = mk(x4[pr.y]), ma = a - ao, mb = b - bo;
    ns = ns + cross(ao - pjo, bo - pjo);
    lo = vmin(lo, vmin(a, b));
    hi = vmax(hi, vmax(a, b));
    mlo = vmin(mlo, vmin(ma, mb));
    mhi = vmax(mhi, vmax(ma, mb));
    const V3 tmin = vmin(vmin(pj, a), b), tmax = vmax(vmax(pj, a), b);
    const V3 tmove = (((pj - pjo) + ma) + mb) / 3.0f;
    st_lo[k] = make_float4(tmin.x, tmin.y, tmin.z, tmove.x);
    st_hi[k] = make_float4(tmax.x, tmax.y, tmax.z, tmove.y);
    st_mz[k] = tmove.z;
  }
  sbox[3 * size_t(j)] = make_float4(lo.x, lo.y, lo.z, mlo.x);
  sbox[3 * size_t(j) + 1] = make_float4(hi.x, hi.y, hi.z, mlo.y);
  sbox[3 * size_t(j) + 2] = make_float4(mhi.x, mhi.y, mhi.z, mlo.z);
  if (nrm) {
    const float l = length(ns);
    const V3 r = l > kEps ? ns / l : mk(0.f, 0.f, 0.f);
    nrm[j] = make_float4(r.x, r.y, r.z, 0.f);
  }
}

// ---------------- normals: shaders/compute_normals.wgsl:25-58
__global__ void k_normals(uint32_t n, const float4* __restrict__ x4, const uint32_t* __restrict__ star_off,
                          const uint2* __restrict__ star_idx, float4* __restrict__ nrm) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const V3 pi = mk(x4[i]);
  V3 s = mk(0.f, 0.f, 0.f);
  for (uint32_t k = star_off[i]; k < star_off[i + 1]; ++k) {
    const uint2 pr = star_idx[k];
    s = s + cross(mk(x4[pr.x]) - pi, mk(x4[pr.y]) - pi);
  }
  const float l = length(s);
  V3 r = l > kEps ? s / l : mk(0.f, 0.f, 0.f);
  nrm[i] = make_float4(r.x, r.y, r.z, 0.f);
}

// ---------------- spatial hash (spatial_hash.rs:158-247, spatial_grid_sort*.wgsl)
// which == 0: key of vertex i is its predicted position; which == 1: key of
// edge i is the midpoint of its two predicted endpoints.
__global__ void k_hash_count(uint32_t cnt, int which, const float4* __restrict__ x4, const float4* __restrict__ p4,
                             const uint2* __restrict__ edges, float cell, uint32_t table, uint32_t* __restrict__ keys,
                             uint32_t* __restrict__ counts, int4* __restrict__ cells, float* __restrict__ mlen,
                             float4* __restrict__ amin, float4* __restrict__ amax) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt) return;
  V3 q;
  if (which == 0) {
    q = mk(p4[i]);
    mlen[i] = length(q - mk(x4[i]));
  } else {
    const uint2 e = edges[i];
    const V3 p0 = mk(p4[e.x]), p1 = mk(p4[e.y]);
    q = (p0 + p1) * 0.5f;
    const V3 lo = vmin(vmin(p0, p1), vmin(mk(x4[e.x]), mk(x4[e.y])));
    const V3 hi = vmax(vmax(p0, p1), vmax(mk(x4[e.x]), mk(x4[e.y])));
    amin[i] = make_float4(lo.x, lo.y, lo.z, 0.f);
    amax[i] = make_float4(hi.x, hi.y, hi.z, 0.f);
  }
  const I3 c = cell_of(q, cell);
  cells[i] = make_int4(c.x, c.y, c.z, 0);
  const uint32_t h = hash3(c.x, c.y, c.z, table);
  keys[i] = h;
  // warp-aggregated increment: lanes with the same bucket share one atomic
  const uint32_t active = __activemask();
  const uint32_t peers = __match_any_sync(active, h);
  const int leader = __ffs(peers) - 1;
  const int lane = threadIdx.x & 31;
  if (lane == leader) atomicAdd(&counts[h], __popc(peers));
}

// Exclusive scan of counts[table] into starts[table + 1] in two launches:
// k_scan_blocks scans 1024-entry tiles (coalesced loads, warp-shuffle scans)
// and writes tile totals; k_scan_finish adds the scanned tile totals.
__device__ __forceinline__ uint32_t block_incl_scan_1024(uint32_t v, uint32_t* warp_tot, uint32_t& total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += t;
  }
  if (lane == 31) warp_tot[wid] = v;
  __syncthreads();
  if (wid == 0) {
    uint32_t w = warp_tot[lane];
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += t;
    }
    warp_tot[lane] = w;
  }
  __syncthreads();
  total = warp_tot[31];
  return v + (wid > 0 ? warp_tot[wid - 1] : 0u);
}
__global__ void __launch_bounds__(1024) k_scan_blocks(uint32_t table, const uint32_t* __restrict__ counts,
                                                      uint32_t* __restrict__ starts, uint32_t* __restrict__ tile_sum) {
  __shared__ uint32_t warp_tot[32];
  const uint32_t i = blockIdx.x * 1024u + threadIdx.x;
  const uint32_t c = i < table ? counts[i] : 0u;
  uint32_t total;
  const uint32_t incl = block_incl_scan_1024(c, warp_tot, total);
  if (i < table) starts[i] = incl - c;
  if (threadIdx.x == 0) tile_sum[blockIdx.x] = total;
}
__global__ void __launch_bounds__(1024) k_scan_finish(uint32_t table, uint32_t ntiles, const uint32_t* __restrict__ tile_sum,
                                                      uint32_t* __restrict__ starts) {
  __shared__ uint32_t tile_off[64];
  if (threadIdx.x < 64) {
    // ntiles <= 64 (table <= 65536): scan of tile sums by the first warp pair
    uint32_t v = threadIdx.x < ntiles ? tile_sum[threadIdx.x] : 0u;
    tile_off[threadIdx.x] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t acc = 0;
    for (uint32_t t = 0; t < ntiles; ++t) { const uint32_t v = tile_off[t]; tile_off[t] = acc; acc += v; }
    starts[table] = acc;
  }
  __syncthreads();
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < table; i += gridDim.x * blockDim.x)
    starts[i] += tile_off[i >> 10];
}

// The same scan in one launch: a block sums the counts before its 1,024-entry
// tile itself (at most 63 tiles, from L2) instead of waiting for another
// launch's tile totals.
__global__ void __launch_bounds__(1024) k_hash_scan(uint32_t table, const uint32_t* __restrict__ counts,
                                                    uint32_t* __restrict__ starts) {
  __shared__ uint32_t warp_tot[32], before[32];
  const uint32_t i = blockIdx.x * 1024u + threadIdx.x;
  uint32_t b = 0;
  for (uint32_t k = threadIdx.x; k < blockIdx.x * 1024u; k += 1024u) b += counts[k];
  b = __reduce_add_sync(0xffffffffu, b);
  if ((threadIdx.x & 31u) == 0) before[threadIdx.x >> 5] = b;
  const uint32_t c = i < table ? counts[i] : 0u;
  uint32_t total;
  const uint32_t incl = block_incl_scan_1024(c, warp_tot, total);  // (synchronises the block)
  const uint32_t base = __reduce_add_sync(0xffffffffu, before[threadIdx.x & 31u]);
  if (i < table) starts[i] = base + incl - c;
  if (i == table - 1u) starts[table] = base + incl;
}
// Scatter that takes the counts down again: they are zero for the next build
// without a clear, and no cursors are needed (the in-bucket order is made
// canonical afterwards).
__global__ void k_hash_place(uint32_t cnt, const uint32_t* __restrict__ keys, const uint32_t* __restrict__ starts,
                             uint32_t* __restrict__ counts, uint32_t* __restrict__ sorted) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt) return;
  const uint32_t h = keys[i];
  sorted[starts[h] + atomicSub(&counts[h], 1u) - 1u] = i;
}

__global__ void k_hash_scatter(uint32_t cnt, const uint32_t* __restrict__ keys, const uint32_t* __restrict__ starts,
                               uint32_t* __restrict__ cursor, uint32_t* __restrict__ sorted) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt) return;
  const uint32_t h = keys[i];
  sorted[starts[h] + atomicAdd(&cursor[h], 1u)] = i;
}

// Candidate records in sorted order, so a warp scanning one bucket reads
// consecutive slots instead of chasing sorted index -> element -> data.
__global__ void k_gather_vertices(uint32_t n, const uint32_t* __restrict__ srt, const float4* __restrict__ x4,
                                  const float4* __restrict__ p4, const float4* __restrict__ v4,
                                  const float* __restrict__ local_len, const float* __restrict__ mlen,
                                  const int4* __restrict__ vcell, float4* __restrict__ vs_p, int4* __restrict__ vs_c,
                                  float4* __restrict__ vs_q) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const uint32_t j = srt[k];
  vs_p[k] = p4[j];
  const int4 c = vcell[j];
  vs_c[k] = make_int4(c.x, c.y, c.z, (int)j);
  vs_q[k] = make_float4(local_len[j], v4[j].w, x4[j].w, mlen[j]);
}
__global__ void k_gather_edges(uint32_t ne, const uint32_t* __restrict__ esrt, const uint2* __restrict__ edges,
                               const int4* __restrict__ ecell, const float4* __restrict__ amin,
                               const float4* __restrict__ amax, int4* __restrict__ es_c, uint2* __restrict__ es_v,
                               float4* __restrict__ es_lo, float4* __restrict__ es_hi) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= ne) return;
  const uint32_t e = esrt[k];
  const int4 c = ecell[e];
  es_c[k] = make_int4(c.x, c.y, c.z, (int)e);
  const uint2 v = edges[e];
  es_v[k] = v;
  // the box records also carry the endpoints (bits in .w), so the E-E
  // filter needs no separate endpoint load
  float4 lo = amin[e], hi = amax[e];
  lo.w = __uint_as_float(v.x);
  hi.w = __uint_as_float(v.y);
  es_lo[k] = lo;
  es_hi[k] = hi;
}

// Canonical in-bucket order: ascending index.  Buckets hold a few to a few
// dozen entries; each thread sorts one bucket in a local array (registers /
// L1) and writes it back; larger buckets fall back to in-place insertion.
__global__ void k_hash_sort_buckets(uint32_t table, const uint32_t* __restrict__ starts, uint32_t* __restrict__ sorted) {
  const uint32_t h = blockIdx.x * blockDim.x + threadIdx.x;
  if (h >= table) return;
  const uint32_t b = starts[h], e = starts[h + 1];
  const uint32_t n = e - b;
  if (n < 2) return;
  constexpr uint32_t kLocal = 64;
  if (n <= kLocal) {
    uint32_t a[kLocal];
    for (uint32_t k = 0; k < n; ++k) a[k] = sorted[b + k];
    for (uint32_t k = 1; k < n; ++k) {
      const uint32_t v = a[k];
      uint32_t j = k;
      while (j > 0 && a[j - 1] > v) { a[j] = a[j - 1]; --j; }
      a[j] = v;
    }
    for (uint32_t k = 0; k < n; ++k) sorted[b + k] = a[k];
    return;
  }
  for (uint32_t k = b + 1; k < e; ++k) {
    const uint32_t v = sorted[k];
    uint32_t j = k;
    while (j > b && sorted[j - 1] > v) { sorted[j] = sorted[j - 1]; --j; }
    sorted[j] = v;
  }
}

// The same canonical order (each bucket ascending), one warp per 32 buckets,
// most of which hold nothing to sort (a warp per bucket spent 22 us on 65,536
// buckets, 10 us of it on empty ones): a bucket of up to 64 entries is sorted in
// registers by a bitonic network (two per lane, padding 0xFFFFFFFF, which no
// index reaches); up to kSortRankCap entries by rank in shared memory; longer
// buckets fall back to the serial insertion sort on lane 0.  Blocks of 4 warps.
constexpr uint32_t kSortRankCap = 1024;
__device__ __forceinline__ void sort_bucket(uint32_t b, uint32_t e, uint32_t lane, uint32_t* buf,
                                            uint32_t* __restrict__ sorted) {
  const uint32_t n = e - b;
  if (n > 64 && n <= kSortRankCap) {
    // rank sort in shared memory: the entries are distinct indices, so the
    // rank of v (the number of smaller entries) is its sorted position
    for (uint32_t i = lane; i < n; i += 32u) buf[i] = sorted[b + i];
    __syncwarp();
    for (uint32_t i = lane; i < n; i += 32u) {
      const uint32_t v = buf[i];
      uint32_t r = 0;
      for (uint32_t k = 0; k < n; ++k) r += buf[k] < v ? 1u : 0u;
      sorted[b + r] = v;
    }
    return;
  }
  if (n > 64) {  // larger than kSortRankCap: insertion sort by one lane
    if (lane == 0)
      for (uint32_t k = b + 1; k < e; ++k) {
        const uint32_t v = sorted[k];
        uint32_t j = k;
        while (j > b && sorted[j - 1] > v) { sorted[j] = sorted[j - 1]; --j; }
        sorted[j] = v;
      }
    return;
  }
  uint32_t a0 = lane < n ? sorted[b + lane] : 0xFFFFFFFFu;
  uint32_t a1 = lane + 32u < n ? sorted[b + lane + 32u] : 0xFFFFFFFFu;
  // (entries past n are padding: networks of 8, 16, 32 or 64)
  const uint32_t kmax = n > 32 ? 64u : n > 16 ? 32u : n > 8 ? 16u : 8u;
  for (uint32_t k = 2; k <= kmax; k <<= 1) {
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      if (j == 32u) {  // partners lane and lane + 32 live in one lane
        const uint32_t lo = min(a0, a1), hi = max(a0, a1);
        const bool up = (lane & k) == 0u;
        a0 = up ? lo : hi;
        a1 = up ? hi : lo;
      } else {
        const uint32_t o0 = __shfl_xor_sync(0xffffffffu, a0, j);
        const uint32_t o1 = __shfl_xor_sync(0xffffffffu, a1, j);
        const bool lower = (lane & j) == 0u;
        const bool up0 = (lane & k) == 0u, up1 = ((lane + 32u) & k) == 0u;
        a0 = (lower == up0) ? min(a0, o0) : max(a0, o0);
        a1 = (lower == up1) ? min(a1, o1) : max(a1, o1);
      }
    }
  }
  if (lane < n) sorted[b + lane] = a0;
  if (lane + 32u < n) sorted[b + lane + 32u] = a1;
}
__global__ void __launch_bounds__(128) k_hash_sort_buckets_warp(uint32_t table, const uint32_t* __restrict__ starts,
                                                                uint32_t* __restrict__ sorted) {
  __shared__ uint32_t sh_sort[4][kSortRankCap];
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t h = (blockIdx.x * 4u + (threadIdx.x >> 5)) * 32u + lane;
  uint32_t b = 0, e = 0;
  if (h < table) {
    b = starts[h];
    e = starts[h + 1];
  }
  for (uint32_t todo = __ballot_sync(0xffffffffu, e - b >= 2u); todo; todo &= todo - 1u) {
    const int k = __ffs(todo) - 1;
    sort_bucket(__shfl_sync(0xffffffffu, b, k), __shfl_sync(0xffffffffu, e, k), lane, sh_sort[threadIdx.x >> 5], sorted);
    __syncwarp();
  }
}

// ---------------- accumulation helpers (shaders/self_collision.wgsl:77-118)
__device__ __forceinline__ int32_t to_fixed(float x) { return f2i(clampf(x * 1000000.0f, -50000000.0f, 50000000.0f)); }
__device__ __forceinline__ void add_disp(int32_t* acc, uint32_t v, V3 d) {
  int32_t* a = acc + (size_t)v * A_N;
  atomicAdd(&a[A_DX], to_fixed(d.x));
  atomicAdd(&a[A_DY], to_fixed(d.y));
  atomicAdd(&a[A_DZ], to_fixed(d.z));
  atomicAdd((uint32_t*)&a[A_CNT], 1u);
}
__device__ __forceinline__ void add_pin(int32_t* acc, uint32_t v, V3 d) {
  int32_t* a = acc + (size_t)v * A_N;
  atomicAdd(&a[A_PDX], to_fixed(d.x));
  atomicAdd(&a[A_PDY], to_fixed(d.y));
  atomicAdd(&a[A_PDZ], to_fixed(d.z));
  atomicAdd((uint32_t*)&a[A_PCNT], 1u);
}
__device__ __forceinline__ void add_ccd(int32_t* acc, uint32_t v, V3 d, bool count_ee) {
  int32_t* a = acc + (size_t)v * A_N;
  const int32_t ix = to_fixed(d.x), iy = to_fixed(d.y), iz = to_fixed(d.z);
  if (ix > 0) atomicMax(&a[A_CPX], ix); else if (ix < 0) atomicMin(&a[A_CNX], ix);
  if (iy > 0) atomicMax(&a[A_CPY], iy); else if (iy < 0) atomicMin(&a[A_CNY], iy);
  if (iz > 0) atomicMax(&a[A_CPZ], iz); else if (iz < 0) atomicMin(&a[A_CNZ], iz);
  if (count_ee) {
    const float lf = clampf(length(d) * 1000000.0f, 0.0f, 2000000000.0f);
    const uint32_t u = lf != lf ? 0u : (uint32_t)lf;
    if (u > 0u) atomicAdd((uint32_t*)&a[A_EEC], 1u);
  }
}

__device__ __forceinline__ bool th_search(const SCArgs& s, uint32_t a, uint32_t b, uint32_t& pos) {
  uint32_t lo = s.th_off[a], hi = s.th_off[a + 1];
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2u;
    const uint32_t v = s.th_idx[mid];
    if (v == b) { pos = mid; return true; }
    if (v < b) lo = mid + 1u; else hi = mid;
  }
  return false;
}
// is_within_two_hops (shaders/self_collision.wgsl:243-264)
__device__ __forceinline__ bool within2(const SCArgs& s, uint32_t a, uint32_t b) {
  uint32_t q;
  if (a == b) return true;
  return th_search(s, a, b, q);
}
// is_topologically_near_folded (:268-293)
__device__ __forceinline__ bool near_folded(const SCArgs& s, uint32_t a, uint32_t b, float d) {
  uint32_t q;
  if (a == b) return true;
  if (!th_search(s, a, b, q)) return false;
  return !(d < s.th_rest[q] * 0.5f);
}
// is_topologically_near_folded_sq (shaders/self_collision_ee_direct.wgsl:237-262)
__device__ __forceinline__ bool near_folded_sq(const SCArgs& s, uint32_t a, uint32_t b, float d2) {
  uint32_t q;
  if (a == b) return true;
  if (!th_search(s, a, b, q)) return false;
  const float l0 = s.th_rest[q];
  return !(d2 < (l0 * l0) * 0.25f);
}

// ---------------- sc_solve: shaders/self_collision.wgsl:317-681
// A warp works a cluster of kScV (1 to 8) vertices that are neighbours in space.  Their
// 27-cell neighbourhoods overlap, so the union of the buckets is scanned once:
// the candidates are staged in shared memory, 32 / kScV of them are tested
// against all the vertices at a time, a shared load and a dozen operations for
// 32 pairs.  The (vertex, candidate) pairs that may matter go
// through four more phases, each on full batches of 32 fed through queues in
// shared memory (per vertex on config 2, 131,072 vertices):
//   1 scan     distance against conservative reaches     (about 230 candidates
//              a cluster)
//   2 gate     exact bounds, two-hop exclusion, star box (48 pairs)
//   3 box      swept box against each star triangle      (160)
//   4 owner    ownership, two-hop exclusion              (70)
//   5 contact  the contact math                          (20; vertex-vertex
//              contacts, 1.5, and untangle candidates likewise)
// One loop picks the furthest phase whose queue holds a full batch, so that
// each phase's code exists once: inlined wherever a queue fills, the contact
// math outgrows the instruction cache (1.25 against 0.99 ms).  Contacts
// accumulate with integer atomics and every other outcome is independent of
// order too; the untangle candidate, which the reference picks with a
// first-strict-minimum scan in its visiting order (cx outer, cz inner, bucket
// order inside a cell), is the minimum of (distance^2, that order).
//
// A warp per vertex with its own bucket walk, compaction and batches of a few
// lanes spent 6,500 warp instructions a vertex: 1.20 ms per pass on config 2,
// now 3,250 and 0.79 ms, bound by instruction issue and the latency of the
// gathers (7 blocks of 4 warps per SM; 8 spill, 6 leave latency uncovered).
struct VertCtx {
  uint32_t index;
  bool pin_i;
  V3 xi, pi;
  float mli, thi, lli;
  I3 cell;
};
constexpr int kScWarps = 4;            // warps per block
constexpr uint32_t kScCells = 96;      // cells of a union
constexpr uint32_t kScSlotBits = 27;   // queue entries: vertex << 27 | slot
constexpr uint32_t kScSlotMask = (1u << kScSlotBits) - 1u;
template <uint32_t kScV>
struct ScWarp {
  // the cluster's vertices
  uint32_t index[kScV], pin[kScV], th_b[kScV], th_n[kScV], th_first[kScV], th_last[kScV];
  float px[kScV], py[kScV], pz[kScV], xx[kScV], xy[kScV], xz[kScV], ml[kScV], th[kScV], ll[kScV];
  int32_t cx[kScV], cy[kScV], cz[kScV];
  unsigned long long best[kScV];         // untangle candidate: distance^2 bits, order
  // the union's candidates (union_ranges)
  uint32_t end[kScCells], beg[kScCells];
  uint8_t box[kScCells];
  // staged candidates: p and reach, layer, slot
  float4 cp[32u + 32u / kScV];
  uint32_t clayer[32u + 32u / kScV], cslot[32u + 32u / kScV];
  uint32_t q[64];                       // past the scan
  uint32_t uq[64];                      // untangle candidates past the scan
  uint4 vq[36];                         // past the gate: pair, star range, contact thickness
  uint2 bq[64];                         // past the box test: pair, star entry
  uint2 tq[64];                         // past the owner test
  uint32_t vv[64];                      // vertex-vertex contacts
  __device__ __forceinline__ VertCtx ctx(uint32_t i) const {
    return VertCtx{index[i], pin[i] != 0u, mk(xx[i], xy[i], xz[i]), mk(px[i], py[i], pz[i]), ml[i], th[i], ll[i],
                   I3{cx[i], cy[i], cz[i]}};
  }
};
// two-hop list of the cluster's vertex i (see th_find)
template <class W>
__device__ __forceinline__ bool sc_th_find(const SCArgs& s, const W& m, uint32_t i, uint32_t b, uint32_t& pos) {
  // most vertices met in contact belong to another part of the mesh
  if (b < m.th_first[i] || b > m.th_last[i]) return false;
  uint32_t at = m.th_b[i];
  for (uint32_t len = m.th_n[i]; len > 1u;) {
    const uint32_t half = len >> 1;
    at += s.th_idx[at + half - 1u] < b ? half : 0u;
    len -= half;
  }
  pos = at;
  return s.th_idx[at] == b;
}
template <class W>
__device__ __forceinline__ bool sc_within2(const SCArgs& s, const W& m, uint32_t i, uint32_t b) {
  uint32_t q;
  return m.index[i] == b || sc_th_find(s, m, i, b, q);
}
__device__ __forceinline__ bool near_cell(const I3& a, const int4& b) {
  return abs(b.x - a.x) <= 1 && abs(b.y - a.y) <= 1 && abs(b.z - a.z) <= 1;
}
// The box of cells around the 27-cell neighbourhoods of a cluster, at most
// kScCells of them: cells [o, o + e).
struct UnionBox {
  int32_t ox, oy, oz;
  uint32_t ex, ey, ez;
  // place of a cell in the box, ~0 outside
  __device__ __forceinline__ uint32_t at(const int4& c) const {
    const uint32_t bx = uint32_t(c.x) - uint32_t(ox), by = uint32_t(c.y) - uint32_t(oy), bz = uint32_t(c.z) - uint32_t(oz);
    return bx < ex && by < ey && bz < ez ? (bx * ey + by) * ez + bz : ~0u;
  }
};
// The box for all elements of the cluster in `todo` (lanes; element v of lane),
// or, where that is more than kScCells, for as many as fit; mine: this lane's
// element is in it.
template <uint32_t kV>
__device__ __forceinline__ UnionBox union_box(const I3& cell, uint32_t todo, uint32_t v, uint32_t lane, bool& mine) {
  const bool in = (todo >> lane) & 1u;
  int32_t ox = __reduce_min_sync(0xffffffffu, in ? cell.x : INT32_MAX);
  int32_t oy = __reduce_min_sync(0xffffffffu, in ? cell.y : INT32_MAX);
  int32_t oz = __reduce_min_sync(0xffffffffu, in ? cell.z : INT32_MAX);
  int32_t hx = __reduce_max_sync(0xffffffffu, in ? cell.x : INT32_MIN);
  int32_t hy = __reduce_max_sync(0xffffffffu, in ? cell.y : INT32_MIN);
  int32_t hz = __reduce_max_sync(0xffffffffu, in ? cell.z : INT32_MIN);
  mine = in;
  // (cells at both ends of the range, of positions that have run away: the
  // difference + 3 would wrap to a small extent)
  auto extent = [](int32_t lo, int32_t hi) {
    const uint32_t d = uint32_t(hi) - uint32_t(lo);
    return d <= kScCells ? d + 3u : kScCells + 1u;
  };
  uint32_t ex = extent(ox, hx), ey = extent(oy, hy), ez = extent(oz, hz);
  if (ex > kScCells || ey > kScCells || ez > kScCells || ex * ey * ez > kScCells) {
    const int lead = __ffs(todo) - 1;
    ox = hx = __shfl_sync(0xffffffffu, cell.x, lead);
    oy = hy = __shfl_sync(0xffffffffu, cell.y, lead);
    oz = hz = __shfl_sync(0xffffffffu, cell.z, lead);
    ex = ey = ez = 3u;
    mine = false;
    for (uint32_t w = 0; w < kV; ++w) {
      const int32_t wx = __shfl_sync(0xffffffffu, cell.x, w), wy = __shfl_sync(0xffffffffu, cell.y, w),
                    wz = __shfl_sync(0xffffffffu, cell.z, w);
      if (!((todo >> w) & 1u)) continue;
      const int32_t nx = min(ox, wx), ny = min(oy, wy), nz = min(oz, wz);
      const int32_t mx = max(hx, wx), my = max(hy, wy), mz = max(hz, wz);
      const uint32_t fx = extent(nx, mx), fy = extent(ny, my), fz = extent(nz, mz);
      if (fx > kScCells || fy > kScCells || fz > kScCells || fx * fy * fz > kScCells) continue;
      ox = nx; oy = ny; oz = nz;
      hx = mx; hy = my; hz = mz;
      ex = fx; ey = fy; ez = fz;
      mine = mine || v == w;
    }
  }
  return UnionBox{int32_t(uint32_t(ox) - 1u), int32_t(uint32_t(oy) - 1u), int32_t(uint32_t(oz) - 1u), ex, ey, ez};
}
// The candidates of a box's cells, flattened over its non-empty buckets: for
// the r-th, end[r] = candidates up to and including it, beg[r] = slot of its
// first minus the candidates before it, box[r] = the cell's place in the box
// (a bucket may hold other cells' elements too, and may come up for several
// cells; an element counts where its own cell is the bucket's).  skip(begin,
// end) returns where a bucket's candidates start.  Returns their number.
template <class F>
__device__ __forceinline__ uint32_t union_ranges(const UnionBox& ub, uint32_t table, const uint32_t* starts,
                                                 uint32_t* end, uint32_t* beg_out, uint8_t* box, uint32_t lane,
                                                 F&& skip) {
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint32_t total = 0, kept = 0;
  const uint32_t eyz = ub.ey * ub.ez, vol = ub.ex * eyz;
  __syncwarp();
  for (uint32_t q0 = 0; q0 < vol; q0 += 32u) {
    const uint32_t q = q0 + lane;
    uint32_t beg = 0, cnt = 0;
    if (q < vol) {
      const uint32_t qx = q / eyz, r = q - qx * eyz, qy = r / ub.ez;
      const uint32_t h = hash3(int32_t(uint32_t(ub.ox) + qx), int32_t(uint32_t(ub.oy) + qy),
                               int32_t(uint32_t(ub.oz) + r - qy * ub.ez), table);
      const uint32_t en = starts[h + 1];
      beg = skip(starts[h], en);
      cnt = en - beg;
    }
    uint32_t incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
      if (int(lane) >= o) incl += u;
    }
    const uint32_t some = __ballot_sync(0xffffffffu, cnt != 0u);
    if (cnt) {
      const uint32_t r = kept + __popc(some & lt_mask);
      end[r] = total + incl;
      beg_out[r] = beg - (total + incl - cnt);
      box[r] = uint8_t(q);
    }
    kept += __popc(some);
    total += __shfl_sync(0xffffffffu, incl, 31);
  }
  __syncwarp();
  return total;
}

// Reach of a vertex in the scan.  A pair matters only within
// max(eth, vtb) <= vtb = eth + 1.3 llj + mli + mlj (the tests of sc_gate) with
// eth <= thi + thj + 0.06 lli, so within reach_i + reach_j; a slack of 1e-5
// covers the rounding on both sides.  Not finite: within reach of everything.
__device__ __forceinline__ float sc_reach(float th, float ll_part, float ml) {
  const float r = (fmaxf(th, 0.f) + ll_part + ml) * 1.00001f + 1e-9f;
  return r < 1e18f ? r : 1e18f;
}

// Exact tests of one pair (shaders/self_collision.wgsl:356-470): the cluster's
// vertex i, candidate slot.  vv: the vertex-vertex contact math must run
// (vv_contact); true with the star range of the candidate and the contact
// thickness when its incident triangles must be tested.
template <class W>
__device__ __forceinline__ bool sc_gate(const SCArgs& s, const W& m, uint32_t i, uint32_t slot, bool& vv,
                                        uint32_t& st_b, uint32_t& st_n, float& out_eth) {
  vv = false;
  const VertCtx c = m.ctx(i);
  const int4 jc = s.vs_c[slot];
  const uint32_t j = (uint32_t)jc.w;
  const float4 pj4 = s.vs_p[slot];
  const float4 q = s.vs_q[slot];
  if (j == c.index || !near_cell(c.cell, jc)) return false;
  const V3 dvv = c.pi - mk(pj4);
  const float d2 = dot(dvv, dvv);
  const float llj = q.x;
  const float eth = fmaxf(c.thi + pj4.w, fminf(c.lli, llj) * 0.06f);
  const float mgd = eth + (c.lli + llj) * 1.3f;
  const float vtb = eth + llj * 1.3f + c.mli + q.w;
  const bool near_v = d2 < eth * eth, near_t = d2 <= vtb * vtb;
  if (!(d2 <= mgd * mgd && (near_v || near_t))) return false;
  // one search of i's two-hop list serves both tests on j: near_folded
  // (:268-293) and, below, within_two_hops (:243-264); j != index here
  uint32_t thq = 0;
  const bool j_in2 = sc_th_find(s, m, i, j, thq);
  if (j_in2 && !(sqrtf(fmaxf(d2, 0.0f)) < s.th_rest[thq] * 0.5f)) return false;
  vv = !c.pin_i && (!(q.z > 0.0f) || c.index < j) && near_v && d2 > kEps * kEps;
  if (!near_t || j_in2) return false;
  // Every triangle of j's star is skipped by its own swept-box test
  // (smin > tmax or smax < tmin on an axis) when the widest possible swept
  // box of i, over the star's motion range plus a 10 um rounding margin,
  // misses the star's box: skipping the whole star is then exact.
  const float4 b0 = s.sbox[3 * size_t(j)], b1 = s.sbox[3 * size_t(j) + 1], b2 = s.sbox[3 * size_t(j) + 2];
  const V3 xi = c.xi, pi = c.pi;
  const float sl = 1e-5f;
  const float rl[3] = {xi.x + b0.w - sl, xi.y + b1.w - sl, xi.z + b2.w - sl};
  const float rh[3] = {xi.x + b2.x + sl, xi.y + b2.y + sl, xi.z + b2.z + sl};
  const float pa[3] = {pi.x, pi.y, pi.z};
  const float lo[3] = {b0.x, b0.y, b0.z}, hi[3] = {b1.x, b1.y, b1.z};
#pragma unroll
  for (int ax = 0; ax < 3; ++ax) {
    const float smin_lb = fminf(rl[ax], pa[ax]) - eth - sl;
    const float smax_ub = fmaxf(rh[ax], pa[ax]) + eth + sl;
    if (smin_lb > hi[ax] || smax_ub < lo[ax]) return false;
  }
  st_b = s.star_off[j];
  st_n = s.star_off[j + 1] - st_b;
  out_eth = eth;
  return st_n > 0u;
}
// One untangle candidate of the cluster's vertex i (:377-383): its key
// (distance^2 bits, visiting order), or all ones.
template <class W>
__device__ __forceinline__ unsigned long long sc_untangle_key(const SCArgs& s, const W& m, uint32_t i,
                                                              uint32_t slot) {
  const int4 jc = s.vs_c[slot];
  const float4 pj4 = s.vs_p[slot];
  const float llj = s.vs_q[slot].x;
  const I3 cell{m.cx[i], m.cy[i], m.cz[i]};
  const V3 dvv = mk(m.px[i], m.py[i], m.pz[i]) - mk(pj4);
  const float d2 = dot(dvv, dvv);
  const float eth = fmaxf(m.th[i] + pj4.w, fminf(m.ll[i], llj) * 0.06f);
  const float ur = eth * 2.5f + llj * 1.3f;
  if (!near_cell(cell, jc) || !(d2 < 1e20f) || !(d2 <= ur * ur) || sc_within2(s, m, i, (uint32_t)jc.w)) return ~0ull;
  const uint32_t k = uint32_t((jc.x - cell.x + 1) * 9 + (jc.y - cell.y + 1) * 3 + (jc.z - cell.z + 1));
  return (unsigned long long)__float_as_uint(d2) << 32 | (k << kScSlotBits | slot);
}

// Sum of d into vertex v's displacement (add_disp) for the lanes with `on`,
// called by the whole warp.  The lanes of a batch mostly share a few v, whose
// contributions are summed in the warp first: integer sums, so the order is
// free.
__device__ __forceinline__ void add_disp_shared(int32_t* acc, uint32_t v, V3 d, bool on) {
  const uint32_t peers = __match_any_sync(0xffffffffu, on ? v : 0xFFFFFFFFu);
  if (!on) return;
  const int32_t x = __reduce_add_sync(peers, to_fixed(d.x));
  const int32_t y = __reduce_add_sync(peers, to_fixed(d.y));
  const int32_t z = __reduce_add_sync(peers, to_fixed(d.z));
  if (int(threadIdx.x & 31u) == __ffs(peers) - 1) {
    int32_t* a = acc + (size_t)v * A_N;
    atomicAdd(&a[A_DX], x);
    atomicAdd(&a[A_DY], y);
    atomicAdd(&a[A_DZ], z);
    atomicAdd((uint32_t*)&a[A_CNT], uint32_t(__popc(peers)));
  }
}

// The vertex-vertex contact (shaders/self_collision.wgsl:405-460) of vertex
// `index` (not pinned) and candidate slot `slot`, which are closer than their
// contact thickness.
__device__ __forceinline__ void vv_contact(const SCArgs& s, uint32_t index, uint32_t slot) {
  const float4 pi4 = s.p4[index];
  const float wi = s.x4[index].w;
  const uint32_t j = (uint32_t)s.vs_c[slot].w;
  const float4 pj4 = s.vs_p[slot];
  const float4 q = s.vs_q[slot];
  const V3 pj = mk(pj4), dvv = mk(pi4) - pj;
  const float eth = fmaxf(pi4.w + pj4.w, fminf(s.local_len[index], q.x) * 0.06f);
  const float dvl = sqrtf(fmaxf(dot(dvv, dvv), 0.0f));
  const float wj = q.z;
  const bool both = wj > 0.0f;
  int32_t* acc = s.acc;
  bool utv = false;
  if (s.untangle != 0) {
    const uint32_t li = layer_of(s.v4, index), lj = __float_as_uint(q.y);
    if (li != lj) {
      const V3 ni = mk(s.nrm[index]), nj = mk(s.nrm[j]);
      const float nil = length(ni), njl = length(nj);
      if (li > lj) {
        if (njl > 0.5f) {
          const V3 nju = nj / njl;
          const bool allow = (wj <= 0.0f) || (nil <= 0.5f) || (dot(ni / fmaxf(nil, kEps), nju) > 0.0f);
          utv = allow && (dot(dvv, nju) < 0.0f);
        }
      } else if (both && nil > 0.5f) {
        const V3 niu = ni / nil;
        const bool allow = (njl <= 0.5f) || (dot(nj / fmaxf(njl, kEps), niu) > 0.0f);
        utv = allow && (dot(-dvv, niu) < 0.0f);
      }
    }
  }
  if (utv) return;
  const V3 nn = dvv / dvl;
  const float pen = eth - dvl;
  const float ws = wi + wj;
  if (ws > kEps) {
    if (wj <= 0.0f) {
      add_pin(acc, index, nn * pen + (pj - mk(s.x4[j])) * 0.5f);
    } else {
      const V3 disp = nn * (pen * 0.5f);
      add_disp(acc, index, disp * (wi / ws));
      add_disp(acc, j, (-disp) * (wj / ws));
    }
  }
}

// One (candidate j, incident triangle) pair, star entry `st` of j
// (shaders/self_collision.wgsl:477-667).  The cheap tests (swept bounds,
// ownership, two-hop exclusion; any order gives the same outcome) come first,
// in vt_box and vt_owner; a pair that passes both needs the contact math,
// vt_contact.  Each pair is independent (its output goes through the
// order-free integer accumulators).
//
// vt_box: the swept box of the vertex against the triangle's, on the star
// entry's record and the contact thickness eth of (i, j)
template <class W>
__device__ __forceinline__ bool vt_box(const SCArgs& s, const W& m, uint32_t i, float eth, uint32_t st) {
  const float4 tlo = s.st_lo[st], thi = s.st_hi[st];
  const float mz = s.st_mz[st];
  const V3 pi = mk(m.px[i], m.py[i], m.pz[i]);
  const V3 rel = mk(m.xx[i], m.xy[i], m.xz[i]) + mk(tlo.w, thi.w, mz);
  const V3 E = mk(eth, eth, eth);
  const V3 smin = vmin(rel, pi) - E, smax = vmax(rel, pi) + E;
  return !(smin.x > thi.x || smin.y > thi.y || smin.z > thi.z || smax.x < tlo.x || smax.y < tlo.y || smax.z < tlo.z);
}
// ownership (:486-500): the triangle is tested from its in-range vertex of
// smallest index, so only a vertex below j can take it away; then the two-hop
// exclusion
template <class W>
__device__ __forceinline__ bool vt_owner(const SCArgs& s, const W& m, uint32_t i, uint32_t j, uint32_t st) {
  const uint2 pr = s.star_idx[st];
  const uint32_t index = m.index[i];
  if (pr.x == index || pr.y == index) return false;
  const V3 pi = mk(m.px[i], m.py[i], m.pz[i]);
  const float thi = m.th[i], lli = m.ll[i], mli = m.ml[i];
  const I3 cell{m.cx[i], m.cy[i], m.cz[i]};
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const uint32_t v = e ? pr.y : pr.x;
    if (j > v) {
      const float4 q = s.p4[v];
      const V3 d = pi - mk(q);
      const float ll = s.local_len[v];
      const float et = fmaxf(thi + q.w, fminf(lli, ll) * 0.06f);
      const float b = et + ll * 1.3f + mli + s.mlen[v];
      if (dot(d, d) <= b * b && near_cell(cell, s.vcell[v])) return false;
    }
  }
  return !sc_within2(s, m, i, pr.x) && !sc_within2(s, m, i, pr.y);
}

// The contact math of a pair that passed the cheap tests: vertex `index`,
// candidate slot `slot`, star entry `st`; called by the whole warp, `on` lanes
// work.  What both contact forms end in, a displacement tp shared by the four
// vertices, is added after the branches.
__device__ __forceinline__ void vt_contact(const SCArgs& s, bool on, uint32_t index, uint32_t slot, uint32_t st) {
  int32_t* acc = s.acc;
  bool push = false;
  V3 tp = mk(0.f, 0.f, 0.f), bw = mk(0.f, 0.f, 0.f);
  float wi = 0.f, wj = 0.f, wv0 = 0.f, wv1 = 0.f, wtot = 1.f;
  uint32_t j = 0, v0 = 0, v1 = 0;
  if (on) {
  const float4 xi4 = s.x4[index], pi4 = s.p4[index];
  wi = xi4.w;
  const bool pin_i = wi <= 0.0f;
  const V3 xi = mk(xi4), pi = mk(pi4);
  const uint32_t li = layer_of(s.v4, index);
  const bool untangle = s.untangle != 0;
  j = (uint32_t)s.vs_c[slot].w;
  const float4 pj4 = s.vs_p[slot];
  const float4 q = s.vs_q[slot];
  const uint2 pr = s.star_idx[st];
  v0 = pr.x;
  v1 = pr.y;
  const V3 tmove = mk(s.st_lo[st].w, s.st_hi[st].w, s.st_mz[st]);
  const V3 pj = mk(pj4);
  const float eth = fmaxf(pi4.w + pj4.w, fminf(s.local_len[index], q.x) * 0.06f);
  const uint32_t lj = __float_as_uint(q.y);
  wj = q.z;
  const float eth2 = eth * eth;
  const V3 pv0 = mk(s.p4[v0]), pv1 = mk(s.p4[v1]);
  wv0 = s.x4[v0].w;
  wv1 = s.x4[v1].w;
  const bool tpin = (wj <= 0.0f) || (wv0 <= 0.0f) || (wv1 <= 0.0f);
  const V3 rel = xi + tmove;
  const V3 mv = pi - rel;
  const float msq = dot(mv, mv);
  float ht = 1.0f, hu = 0.0f, hv = 0.0f;
  bool hit = false;
  if (msq > 1e-12f) hit = seg_tri(rel, pi, pj, pv0, pv1, ht, hu, hv);
  if (hit) {
    const V3 hp = rel + mv * ht;
    const V3 tc = cross(pv0 - pj, pv1 - pj);
    const float tl = length(tc);
    const V3 tn = tl > 1e-12f ? tc / tl : mk(0.0f, 1.0f, 0.0f);
    const float hor = dot(rel - pj, tn);
    bool utc = false;
    if (untangle && !pin_i && (li > lj) && tl > 1e-12f) {
      const V3 ni = mk(s.nrm[index]);
      const float nil = length(ni);
      const bool allow = tpin || (nil <= 0.5f) || (dot(ni / fmaxf(nil, kEps), tn) > 0.0f);
      const bool ret = (hor < 0.0f) && (dot(mv, tn) > 0.0f);
      utc = allow && ret;
    }
    if (!utc) {
      const float ss = fabsf(hor) > 1e-6f ? hor : dot(-mv, tn);
      const V3 ns = ss >= 0.0f ? tn : -tn;
      const float ho = fmaxf(dot(rel - hp, ns), 0.0f);
      const float hs = fmaxf(ho, eth * 0.25f);
      const V3 psafe = hp + ns * hs;
      const V3 tccd = psafe - pi;
      const float pcs = fmaxf(0.0f, eth - hs);
      if (tpin) {
        if (!pin_i) add_ccd(acc, index, tccd + ns * pcs, false);
      } else if (pin_i) {
        const V3 bc = mk(clampf(1.0f - hu - hv, 0.0f, 1.0f), clampf(hu, 0.0f, 1.0f), clampf(hv, 0.0f, 1.0f));
        const float wt = bc.x * bc.x * wj + bc.y * bc.y * wv0 + bc.z * bc.z * wv1;
        if (wt > kEps) {
          const V3 full = tccd + ns * pcs;
          if (wj > 0.0f) add_ccd(acc, j, (-full) * (bc.x * wj / wt), false);
          if (wv0 > 0.0f) add_ccd(acc, v0, (-full) * (bc.y * wv0 / wt), false);
          if (wv1 > 0.0f) add_ccd(acc, v1, (-full) * (bc.z * wv1 / wt), false);
        }
      } else {
        const V3 bc = mk(clampf(1.0f - hu - hv, 0.0f, 1.0f), clampf(hu, 0.0f, 1.0f), clampf(hv, 0.0f, 1.0f));
        const float wt = bc.x * bc.x * wj + bc.y * bc.y * wv0 + bc.z * bc.z * wv1;
        wtot = wi + wt;
        if (wtot > kEps) {
          add_ccd(acc, index, tccd * (wi / wtot), false);
          if (wj > 0.0f) add_ccd(acc, j, (-tccd) * (bc.x * wj / wtot), false);
          if (wv0 > 0.0f) add_ccd(acc, v0, (-tccd) * (bc.y * wv0 / wtot), false);
          if (wv1 > 0.0f) add_ccd(acc, v1, (-tccd) * (bc.z * wv1 / wtot), false);
          if (pcs > kEps) {
            tp = ns * (pcs * 0.6f);
            bw = bc;
            push = true;
          }
        }
      }
    }
  } else {
    bool isf;
    V3 bary;
    const V3 cp = closest_tri(pi, pj, pv0, pv1, isf, bary);
    const V3 dvt = pi - cp;
    const float d2vt = dot(dvt, dvt);
    if (!pin_i && d2vt < eth2 && d2vt > kEps * kEps) {
      const float dvtl = sqrtf(d2vt);
      bool utv = false;
      if (untangle && li > lj) {
        const V3 tc = cross(pv0 - pj, pv1 - pj);
        const float tl = length(tc);
        if (tl > kEps) {
          const V3 tn = tc / tl;
          if (dot(dvt, tn) < 0.0f) {
            const V3 ni = mk(s.nrm[index]);
            const float nil = length(ni);
            utv = tpin || (nil <= 0.5f) || (dot(ni / fmaxf(nil, kEps), tn) > 0.0f);
          }
        }
      }
      if (!utv) {
        const V3 nvt = dvt / dvtl;
        const float pvt = eth - dvtl;
        if (tpin) {
          add_pin(acc, index, nvt * pvt + tmove * 0.5f);
        } else {
          const float wt = bary.x * bary.x * wj + bary.y * bary.y * wv0 + bary.z * bary.z * wv1;
          wtot = wi + wt;
          if (wtot > kEps) {
            tp = nvt * (pvt * 0.6f);
            bw = bary;
            push = true;
          }
        }
      }
    }
  }
  }
  add_disp_shared(acc, index, tp * (wi / wtot), push);
  if (push) {
    if (wj > 0.0f) add_disp(acc, j, (-tp) * (bw.x * wj / wtot));
    if (wv0 > 0.0f) add_disp(acc, v0, (-tp) * (bw.y * wv0 / wtot));
    if (wv1 > 0.0f) add_disp(acc, v1, (-tp) * (bw.z * wv1 / wtot));
  }
}

template <uint32_t kScV>
__global__ void __launch_bounds__(32 * kScWarps, 7) k_sc_solve(const __grid_constant__ SCArgs s) {
  __shared__ ScWarp<kScV> sh[kScWarps];
  const uint32_t lane = threadIdx.x & 31u;
  ScWarp<kScV>& m = sh[threadIdx.x >> 5];
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t at = (blockIdx.x * kScWarps + (threadIdx.x >> 5)) * kScV;
  if (at >= s.n) return;  // whole warp
  // a lane's vertex, and which of the 32 / kScV candidates at a time it tests
  const uint32_t v = lane % kScV, sub = lane / kScV;
  constexpr uint32_t kSub = 32u / kScV;
  // ---- the cluster
  const uint32_t index = at + v < s.n ? s.order[at + v] : 0xFFFFFFFFu;
  bool live = index != 0xFFFFFFFFu;
  V3 pi = mk(0.f, 0.f, 0.f);
  float reach = 0.f, treach = 0.f, best_in = -1.f;
  uint32_t layer = 0;
  I3 cell{0, 0, 0};
  if (live) {
    const float4 xi4 = s.x4[index], pi4 = s.p4[index];
    const float ml = s.mlen[index], ll = s.local_len[index];
    const bool pin = xi4.w <= 0.0f;
    live = !(pin && ml < kEps);
    const int4 vc = s.vcell[index];
    cell = I3{vc.x, vc.y, vc.z};
    pi = mk(pi4);
    reach = sc_reach(pi4.w, 0.06f * ll, ml);
    treach = sc_reach(2.5f * pi4.w, 2.5f * 0.06f * ll, 0.f);
    layer = layer_of(s.v4, index);
    if (s.untangle && !pin && layer > 0u) best_in = 1e20f;  // tracks an untangle candidate
    const uint32_t tb = s.th_off[index], tn = s.th_off[index + 1] - tb;
    m.index[v] = index;
    m.pin[v] = pin ? 1u : 0u;
    m.th_b[v] = tb;
    m.th_n[v] = tn;
    m.th_first[v] = tn ? s.th_idx[tb] : 1u;
    m.th_last[v] = tn ? s.th_idx[tb + tn - 1u] : 0u;
    m.px[v] = pi.x; m.py[v] = pi.y; m.pz[v] = pi.z;
    m.xx[v] = xi4.x; m.xy[v] = xi4.y; m.xz[v] = xi4.z;
    m.ml[v] = ml; m.th[v] = pi4.w; m.ll[v] = ll;
    m.cx[v] = cell.x; m.cy[v] = cell.y; m.cz[v] = cell.z;
  }
  m.best[v] = ~0ull;
  uint32_t todo = __ballot_sync(0xffffffffu, live);
  uint32_t max_layer = 0;  // of the tracking lanes: candidates of this layer or above interest none of them
  {
    const uint32_t l = live && best_in > 0.f ? layer : 0u;
    max_layer = __reduce_max_sync(0xffffffffu, l);
  }
  uint32_t qn = 0, uqn = 0, vqn = 0, bqn = 0, tqn = 0, vvn = 0;  // queue lengths
  uint32_t pos = 0, total = 0, cn = 0, k = 0;                      // scan position, staged candidates
  bool mine = false, drain = false;
  UnionBox ub{0, 0, 0, 0, 0, 0};
  float4 blo = make_float4(0.f, 0.f, 0.f, 0.f);
  V3 bhi = pi;
  for (;;) {
    __syncwarp();
    if (tqn >= 32u || (drain && tqn && !bqn && !vqn && !qn)) {  // 5
      const uint32_t nb = min(tqn, 32u);
      tqn -= nb;
      const bool on = lane < nb;
      const uint2 e = on ? m.tq[tqn + lane] : make_uint2(0u, 0u);
      vt_contact(s, on, on ? m.index[e.x >> kScSlotBits] : 0u, e.x & kScSlotMask, e.y);
      continue;
    }
    if (vvn >= 32u || (drain && vvn && !qn)) {
      const uint32_t nb = min(vvn, 32u);
      vvn -= nb;
      if (lane < nb) {
        const uint32_t e = m.vv[vvn + lane];
        vv_contact(s, m.index[e >> kScSlotBits], e & kScSlotMask);
      }
      continue;
    }
    if (bqn >= 32u || (drain && bqn && !vqn && !qn)) {  // 4
      const uint32_t nb = min(bqn, 32u);
      bqn -= nb;
      bool pass = false;
      uint2 e = make_uint2(0u, 0u);
      if (lane < nb) {
        e = m.bq[bqn + lane];
        const uint32_t j = (uint32_t)s.vs_c[e.x & kScSlotMask].w;
        pass = vt_owner(s, m, e.x >> kScSlotBits, j, e.y);
        if (pass && s.rec_vt) {
          const uint2 tv = s.star_idx[e.y];
          record_vt(s, m.index[e.x >> kScSlotBits], j, tv.x, tv.y);
        }
      }
      const uint32_t b = __ballot_sync(0xffffffffu, pass);
      if (pass) m.tq[tqn + __popc(b & lt_mask)] = e;
      tqn += __popc(b);
      continue;
    }
    if (vqn >= 4u || (drain && vqn && !qn)) {  // 3: 4 pairs x 8 star entries a round
      do {
        const uint32_t nb = min(vqn, 4u), g = lane >> 3, ei = lane & 7u;
        const uint32_t w = vqn - nb + min(g, nb - 1u);
        const uint4 e = m.vq[w];
        const uint32_t sn = g < nb ? e.z : 0u;
        const uint32_t st = e.y + ei;
        const bool pass = ei < sn && vt_box(s, m, e.x >> kScSlotBits, __uint_as_float(e.w), st);
        const uint32_t b = __ballot_sync(0xffffffffu, pass);
        if (pass) m.bq[bqn + __popc(b & lt_mask)] = make_uint2(e.x, st);
        bqn += __popc(b);
        // a star of more than 8 entries keeps its pair queued with the rest
        // of its range; the others' entries are used up
        if (!__any_sync(0xffffffffu, sn > 8u)) {
          vqn -= nb;
        } else {
          __syncwarp();
          if (ei == 0 && g < nb) m.vq[w] = make_uint4(e.x, e.y + 8u, sn > 8u ? sn - 8u : 0u, e.w);
          __syncwarp();
        }
      } while (bqn < 32u && vqn >= 4u);
      continue;
    }
    if (qn >= 32u || (drain && qn)) {  // 2
      const uint32_t nb = min(qn, 32u);
      qn -= nb;
      uint32_t e = 0, sb = 0, sn = 0;
      float eth = 0.f;
      bool vv = false, vt = false;
      if (lane < nb) {
        e = m.q[qn + lane];
        vt = sc_gate(s, m, e >> kScSlotBits, e & kScSlotMask, vv, sb, sn, eth);
      }
      const uint32_t bv = __ballot_sync(0xffffffffu, vv), b = __ballot_sync(0xffffffffu, vt);
      if (vv) m.vv[vvn + __popc(bv & lt_mask)] = e;
      vvn += __popc(bv);
      if (vt) m.vq[vqn + __popc(b & lt_mask)] = make_uint4(e, sb, sn, __float_as_uint(eth));
      vqn += __popc(b);
      continue;
    }
    if (uqn >= 32u || (drain && uqn)) {
      const uint32_t nb = min(uqn, 32u);
      uqn -= nb;
      if (lane < nb) {
        const uint32_t e = m.uq[uqn + lane];
        const unsigned long long key = sc_untangle_key(s, m, e >> kScSlotBits, e & kScSlotMask);
        if (key != ~0ull) atomicMin(&m.best[e >> kScSlotBits], key);
      }
      __syncwarp();
      if (best_in > 0.f) best_in = fminf(best_in, __uint_as_float(min(uint32_t(m.best[v] >> 32), 0x60AD78ECu)));
      continue;
    }
    if (drain) break;
    if (cn >= kSub || (cn && pos >= total)) {  // 1: the staged candidates against the cluster
      do {
        const uint32_t nb = min(cn, kSub);
        cn -= nb;
        const uint32_t c = cn + min(sub, nb - 1u);
        const bool on = mine && sub < nb;
        const float4 a = m.cp[c];
        const V3 d = pi - mk(a);
        const float d2 = dot(d, d), r = reach + a.w;
        const bool pass = on && d2 <= r * r;
        const uint32_t b = __ballot_sync(0xffffffffu, pass);
        const uint32_t e = v << kScSlotBits | m.cslot[c];
        if (pass) m.q[qn + __popc(b & lt_mask)] = e;
        qn += __popc(b);
        if (max_layer) {
          const bool track = on && m.clayer[c] < layer && d2 <= best_in;
          const uint32_t bt = __ballot_sync(0xffffffffu, track);
          if (track) m.uq[uqn + __popc(bt & lt_mask)] = e;
          uqn += __popc(bt);
        }
      } while (cn >= kSub && qn < 32u && uqn < 32u);
      continue;
    }
    if (pos < total) {  // stage candidates that come near the cluster
      {
        const uint32_t t = pos + lane;
        pos += 32u;
        bool keep = false;
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t slot = 0, cl = 0;
        if (t < total) {
          while (t >= m.end[k]) ++k;
          slot = m.beg[k] + t;
          const float4 p = s.vs_p[slot], q = s.vs_q[slot];
          cl = __float_as_uint(q.y);
          a = make_float4(p.x, p.y, p.z, sc_reach(p.w, 1.3f * q.x, q.w));
          const float r = blo.w + fmaxf(a.w, max_layer ? sc_reach(2.5f * p.w, 1.3f * q.x, 0.f) : 0.f);
          const V3 d = mk(fmaxf(fmaxf(blo.x - p.x, p.x - bhi.x), 0.f), fmaxf(fmaxf(blo.y - p.y, p.y - bhi.y), 0.f),
                          fmaxf(fmaxf(blo.z - p.z, p.z - bhi.z), 0.f));
          keep = dot(d, d) <= r * r && ub.at(s.vs_c[slot]) == uint32_t(m.box[k]);
        }
        const uint32_t b = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const uint32_t q = cn + __popc(b & lt_mask);
          m.cp[q] = a;
          m.clayer[q] = cl;
          m.cslot[q] = slot;
        }
        cn += __popc(b);
      }
      continue;
    }
    if (!todo) {
      drain = true;
      continue;
    }
    ub = union_box<kScV>(cell, todo, v, lane, mine);
    todo &= ~__ballot_sync(0xffffffffu, mine);
    total = union_ranges(ub, s.table, s.cs, m.end, m.beg, m.box, lane, [](uint32_t beg, uint32_t) { return beg; });
    // the box around the vertices, and in blo.w the largest reach among them
    // (an untangle candidate, within eth * 2.5 + 1.3 llj, included)
    const float inf = __int_as_float(0x7F800000);
    blo = mine ? make_float4(pi.x, pi.y, pi.z, best_in > 0.f ? fmaxf(reach, treach) : reach)
               : make_float4(inf, inf, inf, 0.f);
    bhi = mine ? pi : mk(-inf, -inf, -inf);
    for (int o = 1; o < int(kScV); o <<= 1) {
      blo.x = fminf(blo.x, __shfl_xor_sync(0xffffffffu, blo.x, o));
      blo.y = fminf(blo.y, __shfl_xor_sync(0xffffffffu, blo.y, o));
      blo.z = fminf(blo.z, __shfl_xor_sync(0xffffffffu, blo.z, o));
      blo.w = fmaxf(blo.w, __shfl_xor_sync(0xffffffffu, blo.w, o));
      bhi = vmax(bhi, mk(__shfl_xor_sync(0xffffffffu, bhi.x, o), __shfl_xor_sync(0xffffffffu, bhi.y, o),
                         __shfl_xor_sync(0xffffffffu, bhi.z, o)));
    }
    pos = cn = k = 0;
  }
  if (best_in >= 0.f && live && sub == 0u) {
    const unsigned long long key = m.best[v];
    if (key != ~0ull) {
      const uint32_t j = (uint32_t)s.vs_c[uint32_t(key) & kScSlotMask].w;
      if (j < 0x3FFFFEu) s.acc[(size_t)index * A_N + A_UT] = (int32_t)(j + 1u);
    }
  }
}

// ---------------- sc_untangle: shaders/self_collision_untangle.wgsl:199-394
__device__ __forceinline__ bool th_range_has(const SCArgs& s, uint32_t b0, uint32_t e0, uint32_t v) {
  if (b0 >= e0) return false;
  uint32_t lo = b0, hi = e0;
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2u;
    const uint32_t x = s.th_idx[mid];
    if (x == v) return true;
    if (x < v) lo = mid + 1u; else hi = mid;
  }
  return false;
}

__global__ void k_untangle(SCArgs s) {
  const uint32_t index = blockIdx.x * blockDim.x + threadIdx.x;
  if (index >= s.n || !s.untangle) return;
  int32_t* ai = s.acc + (size_t)index * A_N;
  const uint32_t cand = (uint32_t)ai[A_UT];
  if (cand == 0u) return;
  ai[A_UT] = 0;
  const float wi = s.x4[index].w;
  const uint32_t li = layer_of(s.v4, index);
  if (wi <= 0.0f || li == 0u) return;
  const uint32_t j1e = cand & 0x3FFFFFu;
  if (j1e == 0u) return;
  const uint32_t j1 = j1e - 1u;
  if (j1 >= s.n || j1 == index) return;
  const float4 pi4 = s.p4[index];
  const V3 pi = mk(pi4);
  const float thi = pi4.w, lli = s.local_len[index];
  const uint32_t ts = s.th_off[index], te = s.th_off[index + 1];
  uint32_t j2 = 0xFFFFFFFFu;
  float bnd = 1e20f;
  for (uint32_t a = s.adj_off[j1]; a < s.adj_off[j1 + 1]; ++a) {
    const uint32_t nb = s.adj_idx[a];
    if (nb < s.n && nb != index && layer_of(s.v4, nb) < li) {
      const V3 dn = pi - mk(s.p4[nb]);
      const float dns = dot(dn, dn);
      if (dns < bnd && !th_range_has(s, ts, te, nb)) { bnd = dns; j2 = nb; }
    }
  }
  float bd2 = 1e20f, bh = 0.0f;
  uint32_t bj = 0xFFFFFFFFu, bv0 = 0, bv1 = 0;
  for (int ci = 0; ci < 2; ++ci) {
    const uint32_t j = ci == 0 ? j1 : j2;
    if (j == 0xFFFFFFFFu) continue;
    const float4 pj4 = s.p4[j];
    const V3 pj = mk(pj4);
    const float eth = fmaxf(thi + pj4.w, fminf(lli, s.local_len[j]) * 0.06f);
    const float capt = eth * 2.5f;
    const float capsq = capt * capt;
    for (uint32_t st = s.star_off[j]; st < s.star_off[j + 1]; ++st) {
      const uint2 pr = s.star_idx[st];
      const uint32_t v0 = pr.x, v1 = pr.y;
      if (v0 == index || v1 == index) continue;
      if (ci == 1 && (v0 == j1 || v1 == j1)) continue;
      const V3 pv0 = mk(s.p4[v0]), pv1 = mk(s.p4[v1]);
      const V3 tmin = vmin(vmin(pj, pv0), pv1), tmax = vmax(vmax(pj, pv0), pv1);
      const V3 z = mk(0.f, 0.f, 0.f);
      const V3 ad = vmax(tmin - pi, z) + vmax(pi - tmax, z);
      const float lim = fminf(capsq, bd2 + 1e-10f);
      if (dot(ad, ad) >= lim) continue;
      bool isf;
      V3 bary;
      const V3 pt = closest_tri(pi, pj, pv0, pv1, isf, bary);
      const V3 du = pi - pt;
      const float dsu = dot(du, du);
      if (dsu >= capsq) continue;
      if (bj != 0xFFFFFFFFu && dsu > bd2 + 1e-10f) continue;
      const V3 tc = cross(pv0 - pj, pv1 - pj);
      const float tl = length(tc);
      if (tl <= kEps) continue;
      const float hu = dot(du, tc / tl);
      const bool same = fabsf(dsu - bd2) <= 1e-10f;
      const bool better = (hu >= 0.0f && bh < 0.0f) || (((hu >= 0.0f) == (bh >= 0.0f)) && fabsf(hu) > fabsf(bh));
      if (bj == 0xFFFFFFFFu || dsu < bd2 - 1e-10f || (same && better)) {
        if (th_range_has(s, ts, te, j) || th_range_has(s, ts, te, v0) || th_range_has(s, ts, te, v1)) continue;
        bd2 = dsu; bh = hu; bj = j; bv0 = v0; bv1 = v1;
      }
    }
  }
  if (bj != 0xFFFFFFFFu && bh < 0.0f) {
    const float4 qj = s.p4[bj], q0 = s.p4[bv0], q1 = s.p4[bv1];
    const V3 upj = mk(qj), up0 = mk(q0), up1 = mk(q1);
    const float wj = s.x4[bj].w, w0 = s.x4[bv0].w, w1 = s.x4[bv1].w;
    bool isf;
    V3 bary;
    const V3 pt = closest_tri(pi, upj, up0, up1, isf, bary);
    const V3 du = pi - pt;
    const float dl = length(du);
    const V3 tc = cross(up0 - upj, up1 - upj);
    const float tl = length(tc);
    if (tl > kEps && dl > kEps) {
      const V3 tn = tc / tl;
      const float hu = dot(du, tn);
      if (hu < 0.0f) {
        const V3 ni = mk(s.nrm[index]);
        const float nil = length(ni);
        const bool tpin = (wj <= 0.0f) || (w0 <= 0.0f) || (w1 <= 0.0f);
        const bool allow = tpin || (nil <= 0.5f) || (dot(ni / fmaxf(nil, kEps), tn) > 0.0f);
        const float etu = fmaxf(thi + qj.w, fminf(lli, s.local_len[bj]) * 0.06f);
        const float cb = -hu / dl;
        const float rt = sqrtf(fmaxf(dl * dl - hu * hu, 0.0f));
        const float rl = fmaxf(etu * 0.5f, kEps);
        if (allow && cb > 0.707f && rt < rl) {
          const V3 ni2 = (mk(s.nrm[bj]) * bary.x + mk(s.nrm[bv0]) * bary.y) + mk(s.nrm[bv1]) * bary.z;
          const float nl = length(ni2);
          const bool behind = (nl <= 0.5f) || (dot(du, ni2) < 0.0f);
          if (behind) {
            const float cw = clampf((cb - 0.707f) / 0.2f, 0.0f, 1.0f);
            const float rw = clampf(1.0f - rt / rl, 0.0f, 1.0f);
            const float pen = fminf(etu - hu, etu * 2.0f) * cw * rw;
            if (pen > kEps) {
              if (tpin) {
                add_disp(s.acc, index, tn * pen);
              } else {
                const float wt = bary.x * bary.x * wj + bary.y * bary.y * w0 + bary.z * bary.z * w1;
                const float wtot = wi + wt;
                if (wtot > kEps) {
                  const V3 disp = tn * (pen * 0.5f);
                  add_disp(s.acc, index, disp * (wi / wtot));
                  if (wj > 0.0f) add_disp(s.acc, bj, (-disp) * (bary.x * wj / wtot));
                  if (w0 > 0.0f) add_disp(s.acc, bv0, (-disp) * (bary.y * w0 / wtot));
                  if (w1 > 0.0f) add_disp(s.acc, bv1, (-disp) * (bary.z * w1 / wtot));
                }
              }
            }
          }
        }
      }
    }
  }
}

// ---------------- sc_solve_ee: shaders/self_collision_ee_direct.wgsl:266-776
__device__ __forceinline__ float seg_eval(V3 a0o, V3 a0, V3 a1o, V3 a1, V3 b0o, V3 b0, V3 b1o, V3 b1, float tau,
                                          float& so, float& to) {
  const V3 A0 = vmix(a0o, a0, tau), A1 = vmix(a1o, a1, tau), B0 = vmix(b0o, b0, tau), B1 = vmix(b1o, b1, tau);
  seg_seg(A0, A1, B0, B1, so, to);
  const V3 d = vmix(A0, A1, so) - vmix(B0, B1, to);
  return dot(d, d);
}
__device__ __forceinline__ float seg_vol(V3 a0o, V3 a0, V3 a1o, V3 a1, V3 b0o, V3 b0, V3 b1o, V3 b1, float tau) {
  const V3 A0 = vmix(a0o, a0, tau), A1 = vmix(a1o, a1, tau), B0 = vmix(b0o, b0, tau), B1 = vmix(b1o, b1, tau);
  return dot(cross(A1 - A0, B1 - B0), B0 - A0);
}
__device__ __forceinline__ bool outer_behind(const SCArgs& s, uint32_t la, uint32_t lb, uint32_t a0, uint32_t a1,
                                             uint32_t b0, uint32_t b1, bool afix, bool bfix, V3 dab) {
  if (la == lb) return false;
  const V3 na = mk(s.nrm[a0]) + mk(s.nrm[a1]), nb = mk(s.nrm[b0]) + mk(s.nrm[b1]);
  const float nal = length(na), nbl = length(nb);
  if (la > lb) {
    if (nbl <= 0.5f) return false;
    const V3 ni = nb / nbl;
    const bool allow = bfix || (nal <= 0.5f) || (dot(na / fmaxf(nal, kEps), ni) > 0.0f);
    return allow && (dot(dab, ni) < 0.0f);
  }
  if (nal <= 0.5f) return false;
  const V3 ni = na / nal;
  const bool allow = afix || (nbl <= 0.5f) || (dot(nb / fmaxf(nbl, kEps), ni) > 0.0f);
  return allow && (dot(-dab, ni) < 0.0f);
}

// The continuous search of a moving edge pair
// (shaders/self_collision_ee_direct.wgsl:404-470): nine samples of the squared
// distance over the substep, one more where the pair's volume first changes
// sign, then six ternary steps around the best.
struct CcdMotion {
  V3 a0o, a0, a1o, a1, b0o, b0, b1o, b1;
  __device__ __forceinline__ float eval(float tau, float& so, float& to) const {
    return seg_eval(a0o, a0, a1o, a1, b0o, b0, b1o, b1, tau, so, to);
  }
  __device__ __forceinline__ float vol(float tau) const { return seg_vol(a0o, a0, a1o, a1, b0o, b0, b1o, b1, tau); }
};
struct CcdBest {
  float tau, d2, s, t;
};
__device__ __forceinline__ CcdBest ccd_search(const CcdMotion& m) {
  float msd = 1e20f, btau = 0.0f, hs = 0.125f, ms = 0.f, mt = 0.f;
  float pv = m.vol(0.0f);
  float zc = -1.0f;
  for (uint32_t k = 0; k <= 8u; ++k) {
    const float tk = (float)k * 0.125f;
    float es, et;
    const float ed = m.eval(tk, es, et);
    if (ed < msd) { msd = ed; btau = tk; ms = es; mt = et; }
    if (k > 0u) {
      const float vol = m.vol(tk);
      if (pv * vol <= 0.0f && zc < 0.0f) zc = tk - 0.0625f;
      pv = vol;
    }
  }
  if (zc >= 0.0f) {
    float es, et;
    const float ed = m.eval(zc, es, et);
    if (ed < msd) { msd = ed; btau = zc; hs = 0.0625f; ms = es; mt = et; }
  }
  float tlo = fmaxf(0.0f, btau - hs), thi = fminf(1.0f, btau + hs);
  CcdBest r{btau, msd, ms, mt};
  for (int it = 0; it < 6; ++it) {
    const float m1 = tlo + (thi - tlo) * (1.0f / 3.0f);
    const float mm2 = thi - (thi - tlo) * (1.0f / 3.0f);
    float e1s, e1t, e2s, e2t;
    const float e1 = m.eval(m1, e1s, e1t);
    const float e2 = m.eval(mm2, e2s, e2t);
    if (e1 < r.d2) r = CcdBest{m1, e1, e1s, e1t};
    if (e2 < r.d2) r = CcdBest{mm2, e2, e2s, e2t};
    if (e1 < e2) thi = mm2; else tlo = m1;
  }
  return r;
}
// The same by 8 lanes (all of the warp call it, groups of 8 with one pair
// each): the samples one per lane, the two ends of a ternary step on the even
// and odd lanes; 9 evaluations in a row instead of 22.  The same samples and
// the same choices, so the same result, on every lane of the group.
__device__ __forceinline__ CcdBest ccd_search8(const CcdMotion& m, uint32_t lane) {
  const uint32_t r = lane & 7u, base = lane & 24u;
  const float tk = (float)(r + 1u) * 0.125f;  // samples 1 to 8; sample 0 by every lane
  float es, et, es0, et0;
  const float ed0 = m.eval(0.0f, es0, et0), v0 = m.vol(0.0f);
  const float ed = m.eval(tk, es, et), vk = m.vol(tk);
  CcdBest best{0.0f, 1e20f, 0.f, 0.f};
  if (ed0 < best.d2) best = CcdBest{0.0f, ed0, es0, et0};
  float pv = v0, zc = -1.0f;
#pragma unroll
  for (uint32_t k = 0; k < 8u; ++k) {
    const float d = __shfl_sync(0xffffffffu, ed, base + k), vol = __shfl_sync(0xffffffffu, vk, base + k);
    const float qs = __shfl_sync(0xffffffffu, es, base + k), qt = __shfl_sync(0xffffffffu, et, base + k);
    const float t = (float)(k + 1u) * 0.125f;
    if (d < best.d2) best = CcdBest{t, d, qs, qt};
    if (pv * vol <= 0.0f && zc < 0.0f) zc = t - 0.0625f;
    pv = vol;
  }
  float hs = 0.125f;
  if (zc >= 0.0f) {
    const float d = m.eval(zc, es, et);
    if (d < best.d2) { best = CcdBest{zc, d, es, et}; hs = 0.0625f; }
  }
  float tlo = fmaxf(0.0f, best.tau - hs), thi = fminf(1.0f, best.tau + hs);
  for (int it = 0; it < 6; ++it) {
    const float m1 = tlo + (thi - tlo) * (1.0f / 3.0f);
    const float mm2 = thi - (thi - tlo) * (1.0f / 3.0f);
    const float e = m.eval((r & 1u) ? mm2 : m1, es, et);
    const float e1 = __shfl_sync(0xffffffffu, e, base), e2 = __shfl_sync(0xffffffffu, e, base + 1u);
    const float s1 = __shfl_sync(0xffffffffu, es, base), s2 = __shfl_sync(0xffffffffu, es, base + 1u);
    const float t1 = __shfl_sync(0xffffffffu, et, base), t2 = __shfl_sync(0xffffffffu, et, base + 1u);
    if (e1 < best.d2) best = CcdBest{m1, e1, s1, t1};
    if (e2 < best.d2) best = CcdBest{mm2, e2, s2, t2};
    if (e1 < e2) thi = mm2; else tlo = m1;
  }
  return best;
}

struct EdgeCtx {
  uint32_t ei, u0, u1;
  float w_u0, w_u1;
  bool apin, bnda;
  V3 p_u0, p_u1, p_u0o, p_u1o;
  float thu0, thu1, mta;
  V3 amin, amax;
  uint32_t la;
  bool untangle;
};

// Contact work for one counted edge pair (shaders/self_collision_ee_direct.wgsl:356-774).
// defer_ccd: the warp pass hands pairs that need the CCD search to the
// one-thread-per-pair k_ee_ccd (inline when the queue is full).  pre: the
// result of the pair's CCD search where it has run already.
__device__ __forceinline__ void ee_pair(const SCArgs& s, const EdgeCtx& c, const TwoHop& th0, const TwoHop& th1,
                                        uint32_t eb, uint32_t j, uint32_t vj, const float4& qj, const float4& qvj,
                                        const float4& xj, const float4& xvj, bool defer_ccd,
                                        const CcdBest* pre = nullptr) {
  const uint32_t u0 = c.u0, u1 = c.u1;
  const float w_u0 = c.w_u0, w_u1 = c.w_u1;
  const bool apin = c.apin, bnda = c.bnda;
  const V3 p_u0 = c.p_u0, p_u1 = c.p_u1, p_u0o = c.p_u0o, p_u1o = c.p_u1o;
  const float thu0 = c.thu0, thu1 = c.thu1, mta = c.mta;
  const uint32_t la = c.la;
  const bool untangle = c.untangle;
  int32_t* acc = s.acc;
  const V3 p_j = mk(qj), p_vj = mk(qvj), p_jo = mk(xj), p_vjo = mk(xvj);
  const float w_j = xj.w, w_vj = xvj.w;
  const float thj = qj.w, thvj = qvj.w;
  const uint32_t lb = layer_of(s.v4, j);
  const bool bndb = ((s.edge_bits[eb >> 5] >> (eb & 31u)) & 1u) != 0u;
  const bool bpair = bnda || bndb;
  bool run_ccd = bpair, has1 = false;
  float s1 = 0.f, t1 = 0.f, d2c = 0.f, ethc = 0.f;
  V3 dl1 = mk(0.f, 0.f, 0.f);
  if (!run_ccd) {
    seg_seg(p_u0, p_u1, p_j, p_vj, s1, t1);
    dl1 = vmix(p_u0, p_u1, s1) - vmix(p_j, p_vj, t1);
    d2c = dot(dl1, dl1);
    ethc = mixf(thu0, thu1, s1) + mixf(thj, thvj, t1);
    const float meg = mta + fmaxf(thj, thvj);
    const V3 dv0 = p_u0 - p_u0o, dv1 = p_u1 - p_u1o, dvj = p_j - p_jo, dvvj = p_vj - p_vjo;
    const V3 va = (dv0 + dv1) * 0.5f, vb = (dvj + dvvj) * 0.5f;
    const float rdg = length(va - vb) + 0.5f * (length(dv1 - dv0) + length(dvvj - dvj));
    const float reach = meg + rdg;
    if (d2c > reach * reach) return;
    has1 = true;
    const V3 d0g = vmix(p_u0o, p_u1o, s1) - vmix(p_jo, p_vjo, t1);
    run_ccd = (rdg > ethc * 0.5f) || (dot(d0g, dl1) <= 0.0f);
  }
  if (run_ccd && defer_ccd) {
    const uint32_t q = atomicAdd(s.ccd_n, 1u);
    if (q < s.ccd_cap) {
      s.ccd_q[q] = make_uint2(c.ei, eb);
      return;
    }
  }
  if (run_ccd) {
    const CcdMotion mo{p_u0o, p_u0, p_u1o, p_u1, p_jo, p_j, p_vjo, p_vj};
    const CcdBest best = pre ? *pre : ccd_search(mo);
    const float tstar = best.tau, dstar = best.d2, ss = best.s, ts = best.t;
    const float ets = mixf(thu0, thu1, ss) + mixf(thj, thvj, ts);
    if (dstar >= ets * ets) return;
    if (s.exclude_neighbors) {
      const V3 a0s = vmix(p_u0o, p_u0, tstar), a1s = vmix(p_u1o, p_u1, tstar);
      const V3 b0s = vmix(p_jo, p_j, tstar), b1s = vmix(p_vjo, p_vj, tstar);
      const V3 t0 = a0s - b0s, t1v = a0s - b1s, t2 = a1s - b0s, t3 = a1s - b1s;
      if (near_folded_sq_t(th0, u0, j, dot(t0, t0)) || near_folded_sq_t(th0, u0, vj, dot(t1v, t1v)) ||
          near_folded_sq_t(th1, u1, j, dot(t2, t2)) || near_folded_sq_t(th1, u1, vj, dot(t3, t3)))
        return;
    }
    bool utc = false;
    if (untangle && la != lb) {
      const bool afx = (w_u0 == 0.0f) && (w_u1 == 0.0f);
      const bool bfx = (w_j == 0.0f) && (w_vj == 0.0f);
      const V3 d0u = ((p_u0o + p_u1o) - (p_jo + p_vjo)) * 0.5f;
      const V3 d1u = ((p_u0 + p_u1) - (p_j + p_vj)) * 0.5f;
      const V3 mu = d1u - d0u;
      if (la > lb && !afx) {
        const V3 ni = mk(s.nrm[j]), no = mk(s.nrm[u0]);
        const bool allow = bfx || (dot(no, no) <= 0.25f);
        utc = allow && (dot(ni, ni) > 0.25f) && (dot(d0u, ni) < 0.0f) && (dot(mu, ni) > 0.0f);
      } else if (lb > la && !bfx) {
        const V3 ni = mk(s.nrm[u0]), no = mk(s.nrm[j]);
        const bool allow = afx || (dot(no, no) <= 0.25f);
        utc = allow && (dot(ni, ni) > 0.25f) && (dot(-d0u, ni) < 0.0f) && (dot(-mu, ni) > 0.0f);
      }
    }
    if (utc) return;
    float s0, t0p;
    seg_seg(p_u0o, p_u1o, p_jo, p_vjo, s0, t0p);
    const V3 d0 = vmix(p_u0o, p_u1o, s0) - vmix(p_jo, p_vjo, t0p);
    const float dist0 = length(d0);
    if (dist0 > kEps) {
      const V3 n0 = d0 / dist0;
      float s1b, t1b;
      seg_seg(p_u0, p_u1, p_j, p_vj, s1b, t1b);
      const V3 d1 = vmix(p_u0, p_u1, s1b) - vmix(p_j, p_vj, t1b);
      const float dist1 = length(d1);
      const V3 de = vmix(p_u0, p_u1, ss) - vmix(p_j, p_vj, ts);
      const float he = dot(de, n0);
      const bool crossed = (he <= 0.0f) || (dot(d1, n0) <= 0.0f) || (bpair && dist1 >= ets && tstar < 1.0f);
      if (he < ets && crossed) {
        const float pc = ets - he;
        const bool bpin = (w_j <= 0.0f) || (w_vj <= 0.0f);
        if (apin && bpin) return;
        const bool aall = (w_u0 == 0.0f) && (w_u1 == 0.0f);
        const bool ball = (w_j == 0.0f) && (w_vj == 0.0f);
        const bool cpe = !(aall || ball);
        if (bpin) {
          const V3 em = ((p_j - p_jo) + (p_vj - p_vjo)) * 0.5f;
          const float a = 1.0f - ss, b = ss;
          const float den = a * a * w_u0 + b * b * w_u1;
          if (den > kEps) {
            const V3 pb = n0 * pc + em * 0.5f;
            if (w_u0 > 0.0f) add_ccd(acc, u0, pb * fminf((a * w_u0) / den, 2.0f), cpe);
            if (w_u1 > 0.0f) add_ccd(acc, u1, pb * fminf((b * w_u1) / den, 2.0f), cpe);
          }
        } else if (apin) {
          const V3 em = ((p_u0 - p_u0o) + (p_u1 - p_u1o)) * 0.5f;
          const float a = 1.0f - ts, b = ts;
          const float den = a * a * w_j + b * b * w_vj;
          if (den > kEps) {
            const V3 pb = (-n0) * pc + em * 0.5f;
            if (w_j > 0.0f) add_ccd(acc, j, pb * fminf((a * w_j) / den, 2.0f), cpe);
            if (w_vj > 0.0f) add_ccd(acc, vj, pb * fminf((b * w_vj) / den, 2.0f), cpe);
          }
        } else {
          const float we1 = (1.0f - ss) * (1.0f - ss) * w_u0 + ss * ss * w_u1;
          const float we2 = (1.0f - ts) * (1.0f - ts) * w_j + ts * ts * w_vj;
          const float wtot = we1 + we2;
          if (wtot > kEps) {
            const V3 tcc = n0 * pc;
            if (w_u0 > 0.0f) add_ccd(acc, u0, tcc * ((1.0f - ss) * w_u0 / wtot), true);
            if (w_u1 > 0.0f) add_ccd(acc, u1, tcc * (ss * w_u1 / wtot), true);
            if (w_j > 0.0f) add_ccd(acc, j, (-tcc) * ((1.0f - ts) * w_j / wtot), true);
            if (w_vj > 0.0f) add_ccd(acc, vj, (-tcc) * (ts * w_vj / wtot), true);
          }
        }
        return;
      }
    }
  }
  {
    float sst, tst, d2e, eth;
    V3 de;
    if (has1) {
      sst = s1; tst = t1; de = dl1; d2e = d2c; eth = ethc;
    } else {
      seg_seg(p_u0, p_u1, p_j, p_vj, sst, tst);
      de = (p_u0 + (p_u1 - p_u0) * sst) - (p_j + (p_vj - p_j) * tst);
      d2e = dot(de, de);
      eth = mixf(thu0, thu1, sst) + mixf(thj, thvj, tst);
    }
    if (d2e >= eth * eth || d2e <= kEps * kEps) return;
    if (s.exclude_neighbors) {
      const V3 e0 = p_u0 - p_j, e1 = p_u0 - p_vj, e2 = p_u1 - p_j, e3 = p_u1 - p_vj;
      if (near_folded_sq_t(th0, u0, j, dot(e0, e0)) || near_folded_sq_t(th0, u0, vj, dot(e1, e1)) ||
          near_folded_sq_t(th1, u1, j, dot(e2, e2)) || near_folded_sq_t(th1, u1, vj, dot(e3, e3)))
        return;
    }
    const float del = sqrtf(d2e);
    bool ute = false;
    if (untangle) {
      const bool afx = (w_u0 <= 0.0f) && (w_u1 <= 0.0f);
      const bool bfx = (w_j <= 0.0f) && (w_vj <= 0.0f);
      ute = outer_behind(s, la, lb, u0, u1, j, vj, afx, bfx, de);
    }
    if (!ute) {
      const V3 ne = de / del;
      const float pe = eth - del;
      const bool bpin = (w_j <= 0.0f) || (w_vj <= 0.0f);
      if (apin && bpin) return;
      if (bpin) {
        const V3 em = ((p_j - p_jo) + (p_vj - p_vjo)) * 0.5f;
        const float a = 1.0f - sst, b = sst;
        const float den = a * a * w_u0 + b * b * w_u1;
        if (den > kEps) {
          const V3 pb = ne * pe + em * 0.5f;
          if (w_u0 > 0.0f) add_pin(acc, u0, pb * fminf((a * w_u0) / den, 2.0f));
          if (w_u1 > 0.0f) add_pin(acc, u1, pb * fminf((b * w_u1) / den, 2.0f));
        }
      } else if (apin) {
        const V3 em = ((p_u0 - p_u0o) + (p_u1 - p_u1o)) * 0.5f;
        const float a = 1.0f - tst, b = tst;
        const float den = a * a * w_j + b * b * w_vj;
        if (den > kEps) {
          const V3 pb = (-ne) * pe + em * 0.5f;
          if (w_j > 0.0f) add_pin(acc, j, pb * fminf((a * w_j) / den, 2.0f));
          if (w_vj > 0.0f) add_pin(acc, vj, pb * fminf((b * w_vj) / den, 2.0f));
        }
      } else {
        const float we1 = (1.0f - sst) * (1.0f - sst) * w_u0 + sst * sst * w_u1;
        const float we2 = (1.0f - tst) * (1.0f - tst) * w_j + tst * tst * w_vj;
        const float wtot = we1 + we2;
        if (wtot > kEps) {
          const V3 td = ne * (pe * 0.6f);
          if (w_u0 > 0.0f) add_disp(acc, u0, td * ((1.0f - sst) * w_u0 / wtot));
          if (w_u1 > 0.0f) add_disp(acc, u1, td * (sst * w_u1 / wtot));
          if (w_j > 0.0f) add_disp(acc, j, (-td) * ((1.0f - tst) * w_j / wtot));
          if (w_vj > 0.0f) add_disp(acc, vj, (-td) * (tst * w_vj / wtot));
        }
      }
    }
  }
}

__device__ __forceinline__ EdgeCtx edge_ctx(const SCArgs& s, uint32_t ei) {
  EdgeCtx c;
  c.ei = ei;
  const uint2 ea = s.edges[ei];
  c.u0 = ea.x;
  c.u1 = ea.y;
  const float4 xu0 = s.x4[c.u0], xu1 = s.x4[c.u1], qu0 = s.p4[c.u0], qu1 = s.p4[c.u1];
  c.w_u0 = xu0.w;
  c.w_u1 = xu1.w;
  c.apin = (c.w_u0 <= 0.0f) || (c.w_u1 <= 0.0f);
  c.p_u0 = mk(qu0); c.p_u1 = mk(qu1); c.p_u0o = mk(xu0); c.p_u1o = mk(xu1);
  c.thu0 = qu0.w;
  c.thu1 = qu1.w;
  c.mta = fmaxf(c.thu0, c.thu1);
  c.bnda = ((s.edge_bits[ei >> 5] >> (ei & 31u)) & 1u) != 0u;
  const V3 m2 = mk(c.mta * 2.0f, c.mta * 2.0f, c.mta * 2.0f);
  c.amin = vmin(vmin(c.p_u0, c.p_u1), vmin(c.p_u0o, c.p_u1o)) - m2;
  c.amax = vmax(vmax(c.p_u0, c.p_u1), vmax(c.p_u0o, c.p_u1o)) + m2;
  c.la = layer_of(s.v4, c.u0);
  c.untangle = s.untangle != 0;
  return c;
}

// Contact work for a listed (edge, edge) pair, with the two-hop lists of
// the first edge's endpoints read from global memory.
__device__ __forceinline__ void ee_listed_pair(const SCArgs& s, uint2 pr, bool defer_ccd,
                                               const CcdBest* pre = nullptr) {
  const EdgeCtx c = edge_ctx(s, pr.x);
  TwoHop th0, th1;
  th0.idx = s.th_idx + s.th_off[c.u0];
  th0.rest = s.th_rest + s.th_off[c.u0];
  th0.n = s.th_off[c.u0 + 1] - s.th_off[c.u0];
  th1.idx = s.th_idx + s.th_off[c.u1];
  th1.rest = s.th_rest + s.th_off[c.u1];
  th1.n = s.th_off[c.u1 + 1] - s.th_off[c.u1];
  const uint2 ebv = s.edges[pr.y];
  ee_pair(s, c, th0, th1, pr.y, ebv.x, ebv.y, s.p4[ebv.x], s.p4[ebv.y], s.x4[ebv.x], s.x4[ebv.y], defer_ccd, pre);
}

// ee_listed_pair outside the caller's register allocation, for the rare
// pairs that do not fit the pair list.
__device__ __noinline__ void ee_listed_pair_call(const SCArgs& s, uint2 pr) { ee_listed_pair(s, pr, true); }

// Counted pairs listed by k_ee_cluster, one thread each: the CCD gate of
// shaders/self_collision_ee_direct.wgsl:361-403 and the discrete contact
// from :632 on; pairs that need the CCD search go on to k_ee_ccd.
// Grid: kEeSeg * kEePairBlocks blocks of 256 threads.
__global__ void __launch_bounds__(256, 4) k_ee_pairs(SCArgs s) {
  const uint32_t seg = blockIdx.x / kEePairBlocks, segcap = s.ee_cap / kEeSeg;
  const uint32_t total = min(s.ee_n[seg], segcap);
  const uint2* list = s.ee_q + size_t(seg) * segcap;
  for (uint32_t q = (blockIdx.x % kEePairBlocks) * blockDim.x + threadIdx.x; q < total;
       q += kEePairBlocks * blockDim.x) {
    const uint2 pr = list[q];
    if (s.rec_ee) record_ee(s, pr.x, pr.y);
    ee_listed_pair(s, pr, true);
  }
}

// Deferred CCD pairs (the CCD search plus the discrete fall-through of
// shaders/self_collision_ee_direct.wgsl:404-774): one thread each when they
// fill the launch, else 8 lanes each for the search, whose chain of evaluations
// is then the launch's time.
__global__ void __launch_bounds__(256, 3) k_ee_ccd(SCArgs s) {
  const uint32_t total = min(*s.ccd_n, s.ccd_cap);
  const uint32_t lane = threadIdx.x & 31u, width = total * 8u <= gridDim.x * blockDim.x ? 8u : 1u;
  const uint32_t step = gridDim.x * blockDim.x / width;
  const uint32_t first = (blockIdx.x * blockDim.x + threadIdx.x) / width;
  for (uint32_t q = first; __any_sync(0xffffffffu, q < total); q += step) {
    const bool on = q < total;
    const uint2 pr = on ? s.ccd_q[q] : make_uint2(0u, 0u);
    const uint2 a = on ? s.edges[pr.x] : make_uint2(0u, 0u), b = on ? s.edges[pr.y] : make_uint2(0u, 0u);
    const CcdMotion m{mk(s.x4[a.x]), mk(s.p4[a.x]), mk(s.x4[a.y]), mk(s.p4[a.y]),
                      mk(s.x4[b.x]), mk(s.p4[b.x]), mk(s.x4[b.y]), mk(s.p4[b.y])};
    const CcdBest best = width == 8u ? ccd_search8(m, lane) : ccd_search(m);
    if (on && (width == 1u || (lane & 7u) == 0u)) ee_listed_pair(s, pr, false, &best);
    __syncwarp();
  }
}

// One edge, searched by a warp in the reference's order: candidates of the 27
// cells around the edge midpoint are flattened (dz outer, dx inner) and visited
// 32 per round.  The per-edge cap on counted candidates (search_count >
// max_search_iterations, :356-359) is applied with a ballot prefix count, so
// exactly the reference's first max_search counted pairs are taken.
struct EeSearch {
  uint32_t start[28], end[28], beg[28];
  uint32_t q[32 * kRounds];
};
// the counted pairs of up to 32 * kRounds candidates at a time go to
// take(queue of candidate slots, length)
template <class F>
__device__ __forceinline__ void ee_search(const SCArgs& s, const EdgeCtx& c, EeSearch& m, int lane, F&& take) {
  const int4 bc4 = s.ecell[c.ei];
  const I3 base = I3{bc4.x, bc4.y, bc4.z};
  // lane k = (dz+1)*9 + (dy+1)*3 + (dx+1)
  uint32_t cnt = 0, beg = 0;
  if (lane < 27) {
    const uint32_t h = hash3(base.x - 1 + lane % 3, base.y - 1 + (lane / 3) % 3, base.z - 1 + lane / 9, s.table);
    beg = s.ecs[h];
    const uint32_t en = s.ecs[h + 1];
    // buckets are in ascending edge order and a pair belongs to its smaller
    // edge index: skip straight to the first edge > ei (never counted before)
    uint32_t lo = beg, hi = en > beg ? en : beg;
    while (lo < hi) {
      const uint32_t mid = lo + (hi - lo) / 2u;
      if ((uint32_t)s.es_c[mid].w <= c.ei) lo = mid + 1u; else hi = mid;
    }
    beg = lo;
    cnt = en > beg ? en - beg : 0u;
  }
  uint32_t incl = cnt;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  __syncwarp();
  if (lane < 27) {
    m.start[lane] = incl - cnt;
    m.end[lane] = incl;
    m.beg[lane] = beg;
  }
  __syncwarp();
  const uint32_t total = __shfl_sync(0xffffffffu, incl, 26);
  uint32_t counted = 0;
  int k = 0;
  const uint32_t lt_mask = (1u << lane) - 1u;
  for (uint32_t chunk = 0; chunk < total && counted < s.max_search; chunk += 32u * kRounds) {
    uint32_t qn = 0;
    for (uint32_t r = 0; r < kRounds; ++r) {
      const uint32_t t = chunk + r * 32u + lane;
      bool pass = false;
      uint32_t slot = 0;
      if (t < total) {
        while (t >= m.end[k]) ++k;
        slot = m.beg[k] + (t - m.start[k]);
        // one level of loads for the whole filter
        const int4 bc = s.es_c[slot];
        const float4 bmin = s.es_lo[slot], bmax = s.es_hi[slot];
        const uint2 ebv = make_uint2(__float_as_uint(bmin.w), __float_as_uint(bmax.w));
        const uint32_t eb = (uint32_t)bc.w;
        pass = c.ei < eb && !(ebv.x == c.u0 || ebv.x == c.u1 || ebv.y == c.u0 || ebv.y == c.u1) &&
               bc.x == base.x - 1 + k % 3 && bc.y == base.y - 1 + (k / 3) % 3 && bc.z == base.z - 1 + k / 9 &&
               !(c.amin.x > bmax.x || c.amin.y > bmax.y || c.amin.z > bmax.z || c.amax.x < bmin.x ||
                 c.amax.y < bmin.y || c.amax.z < bmin.z);
      }
      const uint32_t b = __ballot_sync(0xffffffffu, pass);
      const uint32_t rank = counted + __popc(b & lt_mask);
      if (pass && rank < s.max_search) m.q[qn + __popc(b & lt_mask)] = slot;
      const uint32_t nb = __popc(b);
      qn += counted + nb <= s.max_search ? nb : (counted < s.max_search ? s.max_search - counted : 0u);
      counted += nb;
    }
    __syncwarp();
    take(m.q, qn);
    __syncwarp();
  }
}

// A warp appends qn pairs to its block's segment of the pair list of
// k_ee_pairs; pairs past the segment's capacity get their contact work here.
// pair(q): the q-th.
template <class F>
__device__ __forceinline__ void ee_append(const SCArgs& s, uint32_t qn, uint32_t lane, F&& pair) {
  const uint32_t seg = blockIdx.x % kEeSeg, segcap = s.ee_cap / kEeSeg;
  uint32_t lbase = segcap;
  if (lane == 0 && qn && segcap) lbase = atomicAdd(s.ee_n + seg, qn);
  lbase = __shfl_sync(0xffffffffu, lbase, 0);
  for (uint32_t q = lane; q < qn; q += 32u) {
    const uint2 pr = pair(q);
    if (lbase < segcap && q < segcap - lbase) {
      s.ee_q[size_t(seg) * segcap + lbase + q] = pr;
    } else {
      if (s.rec_ee) record_ee(s, pr.x, pr.y);
      ee_listed_pair_call(s, pr);
    }
  }
}
__device__ __noinline__ void ee_list_ordered(const SCArgs& s, uint32_t ei, EeSearch& m, int lane) {
  ee_search(s, edge_ctx(s, ei), m, lane, [&](const uint32_t* q, uint32_t qn) {
    ee_append(s, qn, uint32_t(lane), [&](uint32_t i) { return make_uint2(ei, (uint32_t)s.es_c[q[i]].w); });
  });
}

// Counted (edge, edge) pairs for k_ee_pairs.  As in k_sc_solve a warp works a
// cluster of kEeV edges that are neighbours in space: the union of their
// 27-cell neighbourhoods is staged 32 candidates at a time in shared memory,
// those that miss the box around all of the cluster's swept boxes are dropped
// there, and 32 / kEeV candidates are tested against all the edges at once.  Counted
// pairs wait in shared memory until the cluster's search is over; an edge with
// more than max_search of them is searched again in the reference's order
// (ee_list_ordered), as is every edge of a cluster whose pairs outgrow the
// buffer.  The list's order is free.  A warp per edge (candidates over the
// lanes) took 0.45 ms per pass on config 2 (261,120 edges, 20 counted pairs
// each), most of it bucket walks and searches.
// The larger the buffer the fewer crowded edges are searched twice, but the
// less L1 is left to the gathers.  us of this pass with 288 / 416 / 576 / 1,024
// entries, layers of 58,080 edges pressed together to 4, 12, 20, 31 and 55 pairs
// an edge (all of them listed but with 1,024): 59 / 60 / 62 / 79, 70 / 72 / 75 /
// 98, 102 / 87 / 88 / 123, 206 / 140 / 123, 279 / 289 / 198.  A warp per edge
// took 61, 68 and 73; the frame with it, 31 and 55 pairs an edge: 2.93 and 5.3
// ms, 2.43 and 4.3 here.  More than 288 costs a frame of config 2 1 %.
constexpr int kEeClusterWarps = 4;
constexpr uint32_t kEePairBuf = 288;
constexpr uint32_t kEeEdgeBits = 29;  // buffered pairs: edge of the cluster << 29 | candidate edge
template <uint32_t kEeV>
struct EeWarp {
  uint32_t end[kScCells], beg[kScCells];  // (see ScWarp)
  uint8_t box[kScCells];
  float4 lo[32u + 32u / kEeV], hi[32u + 32u / kEeV];  // staged candidates: swept box, endpoints in .w
  uint2 c[32u + 32u / kEeV];           // cell in the box (x, y, z bytes), index
  uint32_t edge[kEeV];
  union {
    uint32_t pq[kEePairBuf];
    EeSearch search;
  };
};
template <uint32_t kEeV>
__global__ void __launch_bounds__(32 * kEeClusterWarps, 8) k_ee_cluster(const __grid_constant__ SCArgs s) {
  __shared__ EeWarp<kEeV> sh[kEeClusterWarps];
  const uint32_t lane = threadIdx.x & 31u;
  EeWarp<kEeV>& m = sh[threadIdx.x >> 5];
  const uint32_t lt_mask = (1u << lane) - 1u;
  const uint32_t at = (blockIdx.x * kEeClusterWarps + (threadIdx.x >> 5)) * kEeV;
  if (at >= s.ne) return;  // whole warp
  const uint32_t v = lane % kEeV, sub = lane / kEeV;
  constexpr uint32_t kSub = 32u / kEeV;
  const bool live = at + v < s.ne;
  uint32_t ei = 0xFFFFFFFFu, u0 = 0, u1 = 0, vmask = 0;
  V3 amin = mk(0.f, 0.f, 0.f), amax = amin;
  I3 cell{0, 0, 0};
  for (uint32_t q = v; q < 32u; q += kEeV) vmask |= 1u << q;
  if (live) {
    ei = s.eorder[at + v];
    const EdgeCtx c = edge_ctx(s, ei);
    u0 = c.u0;
    u1 = c.u1;
    amin = c.amin;
    amax = c.amax;
    const int4 bc = s.ecell[ei];
    cell = I3{bc.x, bc.y, bc.z};
    m.edge[v] = ei;
  }
  uint32_t todo = __ballot_sync(0xffffffffu, live);
  while (todo) {
    bool mine;
    const UnionBox ub = union_box<kEeV>(cell, todo, v, lane, mine);
    todo &= ~__ballot_sync(0xffffffffu, mine);
    const uint32_t first = __reduce_min_sync(0xffffffffu, mine ? ei : 0xFFFFFFFFu);
    // buckets are in ascending edge order and a pair belongs to its smaller
    // edge index: start past the cluster's smallest
    const uint32_t total = union_ranges(ub, s.table, s.ecs, m.end, m.beg, m.box, lane, [&](uint32_t beg, uint32_t en) {
      uint32_t lo = beg;
      while (lo < en) {
        const uint32_t mid = lo + (en - lo) / 2u;
        if ((uint32_t)s.es_c[mid].w <= first) lo = mid + 1u; else en = mid;
      }
      return lo;
    });
    const uint32_t rx = uint32_t(cell.x - ub.ox) - 1u, ry = uint32_t(cell.y - ub.oy) - 1u,
                   rz = uint32_t(cell.z - ub.oz) - 1u;
    // the box around the edges' swept boxes; unbounded with a NaN among them,
    // whose box test rejects nothing
    const bool odd = mine && !(amin.x <= amax.x && amin.y <= amax.y && amin.z <= amax.z);
    const float inf = __any_sync(0xffffffffu, odd) ? -__int_as_float(0x7F800000) : __int_as_float(0x7F800000);
    V3 blo = mine && !odd ? vmin(amin, mk(inf, inf, inf)) : mk(inf, inf, inf);
    V3 bhi = mine && !odd ? vmax(amax, mk(-inf, -inf, -inf)) : mk(-inf, -inf, -inf);
    for (int o = 1; o < int(kEeV); o <<= 1) {
      blo = vmin(blo, mk(__shfl_xor_sync(0xffffffffu, blo.x, o), __shfl_xor_sync(0xffffffffu, blo.y, o),
                         __shfl_xor_sync(0xffffffffu, blo.z, o)));
      bhi = vmax(bhi, mk(__shfl_xor_sync(0xffffffffu, bhi.x, o), __shfl_xor_sync(0xffffffffu, bhi.y, o),
                         __shfl_xor_sync(0xffffffffu, bhi.z, o)));
    }
    uint32_t counted = 0, pn = 0, k = 0, cn = 0;
    bool full = false;
    for (uint32_t pos = 0; pos < total && !full; pos += 32u) {
      const uint32_t t = pos + lane;
      bool keep = false;
      float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
      int4 c = make_int4(0, 0, 0, 0);
      if (t < total) {
        while (t >= m.end[k]) ++k;
        const uint32_t slot = m.beg[k] + t;
        c = s.es_c[slot];
        lo = s.es_lo[slot];
        hi = s.es_hi[slot];
        keep = ub.at(c) == uint32_t(m.box[k]) && !(blo.x > hi.x || blo.y > hi.y || blo.z > hi.z || bhi.x < lo.x ||
                                                   bhi.y < lo.y || bhi.z < lo.z);
      }
      const uint32_t kb = __ballot_sync(0xffffffffu, keep);
      if (keep) {
        const uint32_t q = cn + __popc(kb & lt_mask);
        m.lo[q] = lo;
        m.hi[q] = hi;
        m.c[q] = make_uint2(uint32_t(c.x - ub.ox) | uint32_t(c.y - ub.oy) << 8 | uint32_t(c.z - ub.oz) << 16, uint32_t(c.w));
      }
      cn += __popc(kb);
      __syncwarp();
      // kSub at a time from the end; fewer than that wait for the next round
      const bool last = pos + 32u >= total;
      while (cn >= kSub || (last && cn)) {
        const uint32_t nb = min(cn, kSub);
        cn -= nb;
        const uint32_t ci = cn + sub;
        bool pass = false;
        uint32_t eb = 0;
        if (mine && sub < nb) {
          const float4 clo = m.lo[ci], chi = m.hi[ci];
          if (!(amin.x > chi.x || amin.y > chi.y || amin.z > chi.z || amax.x < clo.x || amax.y < clo.y ||
                amax.z < clo.z)) {
            const uint2 bc = m.c[ci];
            const uint32_t b0 = __float_as_uint(clo.w), b1 = __float_as_uint(chi.w);
            eb = bc.y;
            // (cells apart by at most 1 on each axis: 0, 1 or 2 from the edge's cell - 1)
            pass = ei < eb && !(b0 == u0 || b0 == u1 || b1 == u0 || b1 == u1) && (bc.x & 0xFFu) - rx <= 2u &&
                   ((bc.x >> 8) & 0xFFu) - ry <= 2u && (bc.x >> 16) - rz <= 2u;
          }
        }
        const uint32_t b = __ballot_sync(0xffffffffu, pass);
        if (pass) m.pq[pn + __popc(b & lt_mask)] = v << kEeEdgeBits | eb;
        pn += __popc(b);
        counted += __popc(b & vmask);
        if (pn > kEePairBuf - 32u) {
          full = true;
          break;
        }
      }
      __syncwarp();
    }
    __syncwarp();
    const bool again = mine && (full || counted > s.max_search);
    const uint32_t over = __ballot_sync(0xffffffffu, again && sub == 0u);  // bit v
    if (!full) {
      uint32_t kept = pn;
      if (over) {  // drop the pairs of the edges that are searched again
        kept = 0;
        for (uint32_t q0 = 0; q0 < pn; q0 += 32u) {
          const uint32_t q = q0 + lane, e = q < pn ? m.pq[q] : 0u;
          const bool keep = q < pn && !((over >> (e >> kEeEdgeBits)) & 1u);
          const uint32_t b = __ballot_sync(0xffffffffu, keep);
          if (keep) m.pq[kept + __popc(b & lt_mask)] = e;
          kept += __popc(b);
          __syncwarp();
        }
      }
      ee_append(s, kept, lane, [&](uint32_t q) {
        const uint32_t e = m.pq[q];
        return make_uint2(m.edge[e >> kEeEdgeBits], e & ((1u << kEeEdgeBits) - 1u));
      });
      __syncwarp();  // the buffer is the ordered search's too
    }
    for (uint32_t o = over; o; o &= o - 1u)
      ee_list_ordered(s, __shfl_sync(0xffffffffu, ei, __ffs(o) - 1), m.search, int(lane));
    __syncwarp();
  }
}

// The search with the contact work in the edge's warp: a warp per edge, no
// pair list.
__global__ void __launch_bounds__(256, 4) k_ee(const __grid_constant__ SCArgs s) {
  __shared__ EeSearch sh[8];
  __shared__ uint32_t sh_th[8][2][kTwoHopCache];
  __shared__ float sh_thr[8][2][kTwoHopCache];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t ei = blockIdx.x * 8u + warp;
  if (ei >= s.ne) return;  // whole warp
  const EdgeCtx c = edge_ctx(s, ei);
  const TwoHop th0 = stage_two_hop(s.th_off, s.th_idx, s.th_rest, c.u0, sh_th[warp][0], sh_thr[warp][0], lane);
  const TwoHop th1 = stage_two_hop(s.th_off, s.th_idx, s.th_rest, c.u1, sh_th[warp][1], sh_thr[warp][1], lane);
  ee_search(s, c, sh[warp], lane, [&](const uint32_t* queue, uint32_t qn) {
    for (uint32_t q = lane; q < qn; q += 32u) {
      const uint32_t slot = queue[q];
      const uint32_t eb = (uint32_t)s.es_c[slot].w;
      const uint2 ebv = s.es_v[slot];
      const float4 qj = s.p4[ebv.x], qvj = s.p4[ebv.y], xj = s.x4[ebv.x], xvj = s.x4[ebv.y];
      if (s.rec_ee) record_ee(s, ei, eb);
      ee_pair(s, c, th0, th1, eb, ebv.x, ebv.y, qj, qvj, xj, xvj, true);
    }
  });
}

// Grouped variant of k_ee, one lane per edge.  A warp takes 32 consecutive
// slots of the hash-sorted edge order, which are mostly edges of one
// midpoint cell, so they share the reference's 27-cell candidate set.  For
// each distinct cell among its edges the warp builds the cell-matched
// candidates (es_* records) in shared memory, in the reference's visiting
// order (dz outer, dx inner, bucket order), up to kEeChunk at a time; every
// lane of that cell then walks them for its own edge with the reference's
// tests (e_a < e_b, no shared vertex, swept boxes) and per-edge count cap
// (search_count > max_search_iterations ends the edge's search,
// shaders/self_collision_ee_direct.wgsl:330-360).  Counted pairs go to a
// per-warp queue whose contact work (ee_pair) runs 32 pairs at a time.
// The set of counted pairs and the work on each are those of k_ee.
constexpr uint32_t kEeChunk = 128;
constexpr uint32_t kEeWarps = 4;
__global__ void __launch_bounds__(128) k_ee_grouped(SCArgs s) {
  __shared__ int4 ch_c[kEeWarps][kEeChunk];
  __shared__ uint2 ch_v[kEeWarps][kEeChunk];
  __shared__ float4 ch_lo[kEeWarps][kEeChunk], ch_hi[kEeWarps][kEeChunk];
  __shared__ uint32_t q_a[kEeWarps][64], q_b[kEeWarps][64];
  __shared__ uint32_t sh_start[kEeWarps][28], sh_end[kEeWarps][28], sh_beg[kEeWarps][28];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t slot0 = (blockIdx.x * kEeWarps + uint32_t(warp)) * 32u;
  if (slot0 >= s.ne) return;  // whole warp
  const uint32_t my = slot0 + uint32_t(lane);
  const bool valid = my < s.ne;
  // this lane's edge: what the filter needs
  uint32_t ei = 0, u0 = 0, u1 = 0;
  V3 amin = mk(0.f, 0.f, 0.f), amax = amin;
  int4 bc = make_int4(0, 0, 0, 0);
  if (valid) {
    ei = (uint32_t)s.es_c[my].w;
    const EdgeCtx c = edge_ctx(s, ei);
    u0 = c.u0;
    u1 = c.u1;
    amin = c.amin;
    amax = c.amax;
    bc = s.ecell[ei];
  }
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint32_t qn = 0;
  // contact work on the first 32 queued pairs, one per lane
  auto drain32 = [&](uint32_t m) {
    if (uint32_t(lane) < m) {
      const uint32_t a = q_a[warp][lane], b = q_b[warp][lane];
      const EdgeCtx c = edge_ctx(s, a);
      TwoHop th0, th1;
      th0.idx = s.th_idx + s.th_off[c.u0];
      th0.rest = s.th_rest + s.th_off[c.u0];
      th0.n = s.th_off[c.u0 + 1] - s.th_off[c.u0];
      th1.idx = s.th_idx + s.th_off[c.u1];
      th1.rest = s.th_rest + s.th_off[c.u1];
      th1.n = s.th_off[c.u1 + 1] - s.th_off[c.u1];
      const uint2 ebv = s.edges[b];
      if (s.rec_ee) record_ee(s, a, b);
      ee_pair(s, c, th0, th1, b, ebv.x, ebv.y, s.p4[ebv.x], s.p4[ebv.y], s.x4[ebv.x], s.x4[ebv.y], true);
    }
    __syncwarp();
  };
  uint32_t todo = __ballot_sync(0xffffffffu, valid);
  while (todo) {
    const int leader = __ffs(todo) - 1;
    const int32_t cx = __shfl_sync(0xffffffffu, bc.x, leader);
    const int32_t cy = __shfl_sync(0xffffffffu, bc.y, leader);
    const int32_t cz = __shfl_sync(0xffffffffu, bc.z, leader);
    const bool mine = valid && bc.x == cx && bc.y == cy && bc.z == cz;
    todo &= ~__ballot_sync(0xffffffffu, mine);
    // bucket ranges of the cell's 27 neighbours, lane k = (dz+1)*9 + (dy+1)*3 + (dx+1)
    uint32_t cnt = 0, beg = 0;
    if (lane < 27) {
      const uint32_t h = hash3(cx - 1 + lane % 3, cy - 1 + (lane / 3) % 3, cz - 1 + lane / 9, s.table);
      beg = s.ecs[h];
      cnt = s.ecs[h + 1] - beg;
    }
    uint32_t incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane < 27) {
      sh_start[warp][lane] = incl - cnt;
      sh_end[warp][lane] = incl;
      sh_beg[warp][lane] = beg;
    }
    __syncwarp();
    const uint32_t total = __shfl_sync(0xffffffffu, incl, 26);
    uint32_t counted = 0;
    bool active = mine;
    int k = 0;
    for (uint32_t t0 = 0; t0 < total && __any_sync(0xffffffffu, active);) {
      // the next cell-matched candidates, in order, into the chunk
      uint32_t nch = 0;
      while (t0 < total && nch + 32u <= kEeChunk) {
        const uint32_t t = t0 + uint32_t(lane);
        bool keep = false;
        uint32_t slot = 0;
        int4 c4 = make_int4(0, 0, 0, 0);
        if (t < total) {
          while (t >= sh_end[warp][k]) ++k;
          slot = sh_beg[warp][k] + (t - sh_start[warp][k]);
          c4 = s.es_c[slot];
          keep = c4.x == cx - 1 + k % 3 && c4.y == cy - 1 + (k / 3) % 3 && c4.z == cz - 1 + k / 9;
        }
        const uint32_t b = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const uint32_t o = nch + __popc(b & lt_mask);
          ch_c[warp][o] = c4;
          ch_v[warp][o] = s.es_v[slot];
          ch_lo[warp][o] = s.es_lo[slot];
          ch_hi[warp][o] = s.es_hi[slot];
        }
        nch += __popc(b);
        t0 += 32u;
      }
      __syncwarp();
      // every lane of the cell walks the chunk for its own edge
      for (uint32_t j = 0; j < nch; ++j) {
        bool pass = false;
        uint32_t eb = 0;
        if (active) {
          const int4 c4 = ch_c[warp][j];
          const uint2 v = ch_v[warp][j];
          eb = (uint32_t)c4.w;
          const float4 lo = ch_lo[warp][j], hi = ch_hi[warp][j];
          pass = ei < eb && !(v.x == u0 || v.x == u1 || v.y == u0 || v.y == u1) &&
                 !(amin.x > hi.x || amin.y > hi.y || amin.z > hi.z || amax.x < lo.x || amax.y < lo.y ||
                   amax.z < lo.z);
          if (pass && ++counted > s.max_search) {
            pass = false;
            active = false;
          }
        }
        const uint32_t b = __ballot_sync(0xffffffffu, pass);
        if (pass) {
          const uint32_t o = qn + __popc(b & lt_mask);
          q_a[warp][o] = ei;
          q_b[warp][o] = eb;
        }
        qn += __popc(b);
        __syncwarp();
        if (qn >= 32u) {
          drain32(32u);
          qn -= 32u;
          if (uint32_t(lane) < qn) {
            q_a[warp][lane] = q_a[warp][32 + lane];
            q_b[warp][lane] = q_b[warp][32 + lane];
          }
          __syncwarp();
        }
      }
      __syncwarp();
    }
  }
  if (qn) drain32(qn);
}

// ---------------- edge colliders: shaders/edge_collision.wgsl:82-276
// Collider edge (mesh.rs:1503-1565): endpoints, the largest thickness and the
// mean friction of its triangles, their summed then normalised normals, and
// bit 0 set when every triangle is single-sided.
struct ColEdge {
  float4 p0t;  // p0, thickness
  float4 p1f;  // p1, friction
  float4 nfl;  // normal, flags bits
};
struct EdgeColArgs {
  uint32_t ne, nce;            // cloth edges, collider edges
  const uint2* edges;
  const float4* x4;
  const float4* p4;
  const ColEdge* ce;
  const uint32_t* cs;          // collider-edge grid: cell starts [table + 1]
  const uint32_t* srt;         // and edge indices
  float cell;
  uint32_t table;
  float mscale, moff;          // contact distance = thickness sum * mscale + moff
  int32_t* acc;
};
// closest points of segments p0-p1 and q0-q1 (edge_collision.wgsl:96-149)
__device__ __forceinline__ float seg_closest(V3 p0, V3 p1, V3 q0, V3 q1, float& s, float& t) {
  const V3 d1 = p1 - p0, d2 = q1 - q0, r = p0 - q0;
  const float a = dot(d1, d1), e = dot(d2, d2), f = dot(d2, r);
  s = 0.0f;
  t = 0.0f;
  if (a <= 1e-12f && e <= 1e-12f) return length(p0 - q0);
  if (a <= 1e-12f) {
    t = clampf(f / e, 0.0f, 1.0f);
  } else {
    const float c = dot(d1, r);
    if (e <= 1e-12f) {
      s = clampf(-c / a, 0.0f, 1.0f);
    } else {
      const float b = dot(d1, d2);
      const float denom = a * e - b * b;
      s = denom > a * e * 1e-7f ? clampf((b * f - c * e) / denom, 0.0f, 1.0f) : 0.0f;
      t = (b * s + f) / e;
      if (t < 0.0f) {
        t = 0.0f;
        s = clampf(-c / a, 0.0f, 1.0f);
      } else if (t > 1.0f) {
        t = 1.0f;
        s = clampf((b - c) / a, 0.0f, 1.0f);
      }
    }
  }
  return length((p0 + d1 * s) - (q0 + d2 * t));
}
// One thread per cloth edge: collider edges of the 27 cells around its
// midpoint; a contact pushes both endpoints out (collider edges do not move)
// through the pin channel of the self-collision accumulator.
__global__ void __launch_bounds__(256) k_edge_collision(EdgeColArgs a) {
  const uint32_t ei = blockIdx.x * blockDim.x + threadIdx.x;
  if (ei >= a.ne || a.nce == 0u) return;
  const uint2 e = a.edges[ei];
  const uint32_t u0 = e.x, u1 = e.y;
  const float w0 = a.x4[u0].w, w1 = a.x4[u1].w;
  if (w0 + w1 <= kEps) return;
  const float4 q0v = a.p4[u0], q1v = a.p4[u1];
  const V3 p0 = mk(q0v), p1 = mk(q1v);
  const V3 pmid = (p0 + p1) * 0.5f;
  const float cth = fmaxf(q0v.w, q1v.w);
  const I3 cc = cell_of(pmid, a.cell);
  const V3 lo = vmin(p0, p1), hi = vmax(p0, p1);
  for (int dz = -1; dz <= 1; ++dz)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dx = -1; dx <= 1; ++dx) {
        const uint32_t h = hash3(cc.x + dx, cc.y + dy, cc.z + dz, a.table);
        const uint32_t st = a.cs[h], en = a.cs[h + 1];
        for (uint32_t k = st; k < en; ++k) {
          const ColEdge ce = a.ce[a.srt[k]];
          const V3 c0 = mk(ce.p0t), c1 = mk(ce.p1f);
          const float tgt = (cth + ce.p0t.w) * a.mscale + a.moff;
          const V3 clo = vmin(c0, c1), chi = vmax(c0, c1);
          if (hi.x + tgt < clo.x || lo.x - tgt > chi.x || hi.y + tgt < clo.y || lo.y - tgt > chi.y ||
              hi.z + tgt < clo.z || lo.z - tgt > chi.z)
            continue;
          float s, t;
          const float dist = seg_closest(p0, p1, c0, c1, s, t);
          if (!(dist < tgt)) continue;
          const V3 diff = (p0 + (p1 - p0) * s) - (c0 + (c1 - c0) * t);
          const V3 en_ = mk(ce.nfl);
          const bool single = (__float_as_uint(ce.nfl.w) & 1u) != 0u;
          const bool has_n = dot(en_, en_) > 0.25f;
          V3 nrm = mk(0.0f, 0.0f, 1.0f);
          float pen = tgt - dist;
          if (single && has_n) {
            const float sp = dot(diff, en_);
            if (sp >= 0.0f) {
              nrm = dist > kEps ? diff / dist : en_;
              pen = tgt - dist;
            } else {
              nrm = en_;
              pen = fminf(tgt - sp, tgt * 2.0f);
            }
          } else if (dist > kEps) {
            nrm = diff / dist;
          } else {
            const V3 cr = cross(p1 - p0, c1 - c0);
            const float cl = length(cr);
            if (cl > kEps) nrm = cr / cl;
          }
          const V3 push = nrm * pen;
          const float ca = 1.0f - s, cb = s;
          const float den = ca * ca * w0 + cb * cb * w1;
          if (den > kEps) {
            const float f0 = fminf((ca * w0) / den, 2.0f), f1 = fminf((cb * w1) / den, 2.0f);
            if (w0 > 0.0f) add_pin(a.acc, u0, push * f0);
            if (w1 > 0.0f) add_pin(a.acc, u1, push * f1);
          }
        }
      }
}

// ---------------- sc_apply: shaders/self_collision_apply.wgsl:57-177
// kUpdate: followed by the substep's velocity update (update_vertex_m).
template <bool kUpdate>
__global__ void k_apply(uint32_t n, float4* __restrict__ x4, float4* __restrict__ p4,
                        const float* __restrict__ local_len, int32_t* __restrict__ acc, float relief, int enable_relief,
                        float max_disp_ratio, float4* __restrict__ v4, float dt_sub) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int4* a4 = reinterpret_cast<int4*>(acc + (size_t)i * A_N);
  const int4 r0 = a4[0], r1 = a4[1], r2 = a4[2], r3 = a4[3];
  const bool pinned = x4[i].w <= 0.0f;
  V3 fd = mk(0.f, 0.f, 0.f);
  const uint32_t cnt = (uint32_t)r0.w;
  if (cnt > 0u && !pinned) {
    const V3 tdp = mk((float)r0.x, (float)r0.y, (float)r0.z) * (1.0f / 1000000.0f);
    V3 ed = tdp / fmaxf(1.0f, sqrtf((float)cnt));
    if (enable_relief) ed = ed * relief;
    const float pl = length(ed);
    const float ratio = max_disp_ratio > 0.0f ? max_disp_ratio : 0.50f;
    const float ms = fminf(local_len[i] * ratio, 0.10f);
    if (pl > ms && pl > kEps) ed = (ed / pl) * ms;
    fd = fd + ed;
  }
  const uint32_t pc = (uint32_t)r1.w;
  V3 avg = mk(0.f, 0.f, 0.f);
  if (pc > 0u && !pinned) avg = (mk((float)r1.x, (float)r1.y, (float)r1.z) * (1.0f / 1000000.0f)) / (float)pc;
  const uint32_t eec = (uint32_t)r3.w;
  if (!pinned) {
    const V3 cp = mk((float)r2.x, (float)r2.y, (float)r2.z) * (1.0f / 1000000.0f);
    const V3 cn = mk((float)r2.w, (float)r3.x, (float)r3.y) * (1.0f / 1000000.0f);
    V3 env = cp + cn;
    if (eec >= 4u) env = env * fmaxf(0.5f, sqrtf(3.0f / (float)eec));
    const V3 z = mk(0.f, 0.f, 0.f);
    fd = fd + (vmax(vmax(env, z), vmax(avg, z)) + vmin(vmin(env, z), vmin(avg, z)));
  }
  const int4 zero = make_int4(0, 0, 0, 0);
  a4[0] = zero; a4[1] = zero; a4[2] = zero; a4[3] = zero;
  if (length(fd) > kEps) {
    float4 p = p4[i];
    p.x += fd.x; p.y += fd.y; p.z += fd.z;
    p4[i] = p;
  }
  if (kUpdate) update_vertex<false>(i, x4, p4, v4, dt_sub);
}

}  // namespace tcloth
