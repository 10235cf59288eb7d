// Resident solver: the constraint phase of one cloth on one thread-block
// cluster, its vertices and constraints on chip.
//
// A cloth of up to about 20,000 vertices gives a colour step a few hundred to
// a few thousand constraints, far less work than the barrier over the whole
// chip that separates two steps (about 5.5 us in k_solver_persistent) or than
// a launch per step (2.1 us with programmatic launches); a frame has 300 to
// 3,000 steps.  Here a cluster of K CTAs owns the cloth: the vertices are cut
// into K slices in Morton order, each CTA keeps (p, inverse mass) of its slice
// and the records and lambdas of the constraints whose first vertex it owns in
// shared memory, the other vertex is reached through distributed shared
// memory, and colour steps are separated by the cluster's hardware barrier
// (__syncthreads for one CTA).  The per-element arithmetic and the order of the
// steps are those of the other paths, so the results are the same bits.
//
// Bound by the latency of one constraint's chain (load, square root, divide,
// divide, store) plus the barrier: 0.5 us a step on one CTA, 1.05 us on 16.
// Records in global memory, prefetched a step ahead, were slower (265
// vertices: 0.29 against 0.20 ms a frame; 8,065 vertices: 1.34 against 0.89).
// ms a frame, persistent solver -> here: 265 vertices, 10 substeps x 2
// iterations 1.75 -> 0.19; 8,065 vertices, 10 x 5 4.18 -> 0.89; sewn garment
// of 18,432 vertices with self-collision, 10 x 4 4.67 -> 2.36 (2.67 with a
// launch per colour).
#pragma once
#include "solver_kernels.cuh"
#include "tcgen05.cuh"

namespace tcloth {

constexpr uint32_t kResThreads = 512;
constexpr uint32_t kResMaxCtas = 16;

struct ResidentArgs {
  uint32_t ctas;            // K
  uint32_t chunk;           // vertices per slice
  uint32_t ccap;            // constraint records per CTA (the largest slice's)
  const uint32_t* order;    // vertex of slice position rank * chunk + slot
  const uint32_t* sid;      // vertex -> rank << 16 | slot
  // constraint steps: the distance colours, then the bending colours.  The
  // records are ordered by (rank, step); tab[rank * (nsteps + 1) + step] are
  // their offsets
  uint32_t nsteps, ndsteps;
  const uint32_t* tab;
  const uint2* ids;         // (kind << 16 | slot, rank << 16 | slot) of the projected pair
  const float4* par;        // rest, compliance when stretched, when compressed, -
  const uint2* gate_ids;    // kind 3: the sewn pair that gates the constraint, and its gap
  const float* gate_gap;
  const uint32_t* pin_tab;  // K + 1 offsets into pin_idx (indices into pin_v / pin_t)
  const uint32_t* pin_idx;
  const uint32_t* sew_tab;  // per sewing colour K + 1 offsets into sew_idx
  const uint32_t* sew_idx;
};

// Parameters in staged order: out[k] from distance constraint perm[k], or
// with the top bit set from a bending constraint (one compliance).
__global__ void k_resident_gather(uint32_t cnt, const uint32_t* __restrict__ perm, const float4* __restrict__ dist,
                                  const float4* __restrict__ bend, float4* __restrict__ out) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= cnt) return;
  const uint32_t q = perm[k];
  if (q >> 31) {
    const float4 c = bend[q & 0x7FFFFFFFu];
    out[k] = make_float4(c.x, c.y, c.y, 0.f);
  } else {
    out[k] = dist[q];
  }
}

__device__ __forceinline__ float4 ld_cluster(uint32_t addr, uint32_t rank) {
  float4 v;
  asm volatile(
      "{\n .reg .u32 a;\n mapa.shared::cluster.u32 a, %4, %5;\n"
      " ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [a];\n}"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "r"(addr), "r"(rank)
      : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t rank, float4 v) {
  asm volatile(
      "{\n .reg .u32 a;\n mapa.shared::cluster.u32 a, %0, %1;\n"
      " st.shared::cluster.v4.f32 [a], {%2, %3, %4, %5};\n}" ::"r"(addr),
      "r"(rank), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
      : "memory");
}
__device__ __forceinline__ void res_sync(bool one) {
  if (one) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// A slice position of the cluster, its own CTA's directly.
struct ResSlice {
  float4* s;
  uint32_t rank;
  __device__ __forceinline__ float4 ld(uint32_t id) const {
    const uint32_t r = id >> 16;
    float4* q = s + (id & 0xFFFFu);
    return r == rank ? *q : ld_cluster(smem_addr(q), r);
  }
  __device__ __forceinline__ void st(uint32_t id, float4 v) const {
    const uint32_t r = id >> 16;
    float4* q = s + (id & 0xFFFFu);
    if (r == rank) *q = v;
    else st_cluster(smem_addr(q), r, v);
  }
};

// Vertex policy of the per-vertex passes on the owner's slice: p on chip with
// the inverse mass in .w (the thickness of p4.w stays in global memory), x and
// v on chip too when kFull.
template <bool kFull>
struct ResOwn {
  static constexpr bool kCg = false;
  float4 *sp, *sx, *sv;
  float4 *gx, *gp, *gv;
  uint32_t slot;
  __device__ __forceinline__ float4 ldx(uint32_t i) const { return kFull ? sx[slot] : gx[i]; }
  __device__ __forceinline__ float4 ldp(uint32_t i) const {
    const float4 p = sp[slot];
    return make_float4(p.x, p.y, p.z, gp[i].w);
  }
  __device__ __forceinline__ float4 ldv(uint32_t i) const { return kFull ? sv[slot] : gv[i]; }
  __device__ __forceinline__ void stx(uint32_t i, float4 v) const {
    if (kFull) sx[slot] = v;
    else gx[i] = v;
  }
  __device__ __forceinline__ void stp(uint32_t, float4 v) const {
    sp[slot] = make_float4(v.x, v.y, v.z, sp[slot].w);
  }
  __device__ __forceinline__ void stv(uint32_t i, float4 v) const {
    if (kFull) sv[slot] = v;
    else gv[i] = v;
  }
};
// Pins: only the inverse mass of x is read.
struct ResPin {
  float4* sp;
  const uint32_t* sid;
  __device__ __forceinline__ float4 ldx(uint32_t i) const { return sp[sid[i] & 0xFFFFu]; }
  __device__ __forceinline__ float4 ldp(uint32_t i) const { return sp[sid[i] & 0xFFFFu]; }
  __device__ __forceinline__ void stp(uint32_t i, float4 v) const { sp[sid[i] & 0xFFFFu] = v; }
};
// Sewing: pairs anywhere in the cluster, thickness from global memory.
struct ResSew {
  ResSlice s;
  const uint32_t* sid;
  const float4* gp;
  __device__ __forceinline__ float4 ldx(uint32_t i) const { return s.ld(sid[i]); }
  __device__ __forceinline__ float4 ldp(uint32_t i) const {
    const float4 p = s.ld(sid[i]);
    return make_float4(p.x, p.y, p.z, gp[i].w);
  }
  __device__ __forceinline__ void stp(uint32_t i, float4 v) const {
    const uint32_t id = sid[i];
    s.st(id, make_float4(v.x, v.y, v.z, s.ld(id).w));
  }
};

// A compliance as alpha~ = compliance / dt^2, computed once per launch; the
// flag says that the constraint is off on that side (>= 1e9).
constexpr uint32_t kResOffT = 1u << 18, kResOffC = 1u << 19;

// One constraint of the CTA: distance_core and bending_core on the on-chip
// records (kind 0 stretch, 1 shear, 2 bending, 3 gated bending).  rec =
// (rest, alpha~ stretched, alpha~ compressed, lambda).
template <bool kFull>
__device__ __forceinline__ void res_project(uint32_t k, uint32_t g0, const uint2 e, float4* __restrict__ rec,
                                            bool first, const ResSlice& sp, const ResSlice& sx, const SolverArgs& a,
                                            const ResidentArgs& t) {
  const float4 q0 = sp.s[e.x & 0xFFFFu], q1 = sp.ld(e.y);
  const float4 c = rec[k];
  const float w0 = q0.w, w1 = q1.w;
  const float ws = w0 + w1;
  const V3 p0 = mk(q0), p1 = mk(q1);
  const V3 delta = p0 - p1;
  const float dist = length(delta);
  const float l = first ? 0.f : c.w;
  if (first) rec[k].w = 0.f;
  if (ws <= kEps || dist <= kEps) return;
  const float cv = dist - c.x;
  if (e.x & (cv >= 0.0f ? kResOffT : kResOffC)) return;
  const uint32_t kind = (e.x >> 16) & 3u;
  if (kind == 3u) {
    if (dist >= c.x) return;
    const uint2 g = t.gate_ids[g0 + k];
    if (length(mk(sp.ld(g.x)) - mk(sp.ld(g.y))) > t.gate_gap[g0 + k]) return;
  }
  const V3 dir = delta / dist;
  const float alpha = cv >= 0.0f ? c.y : c.z;
  float dl;
  if (kind >= 2u ? a.bdamp : a.ddamp) {
    const float dt = fmaxf(a.sp.dt, 1e-8f);
    const float damp = kind >= 2u ? a.sp.bd : (kind ? a.sp.sd : (cv >= 0.0f ? a.sp.td : a.sp.cd));
    const float tau = damp * 1e-5f;
    const float gamma = fminf(tau / dt, 1e4f);
    V3 xa, xb;
    if (kFull) {
      xa = mk(sx.s[e.x & 0xFFFFu]);
      xb = mk(sx.ld(e.y));
    } else {
      xa = mk(__ldcg(a.x4 + t.order[sp.rank * t.chunk + (e.x & 0xFFFFu)]));
      xb = mk(__ldcg(a.x4 + t.order[(e.y >> 16) * t.chunk + (e.y & 0xFFFFu)]));
    }
    const V3 rel = (p0 - xa) - (p1 - xb);
    const float vp = dot(dir, rel);
    dl = (-cv - alpha * l - gamma * vp) / ((1.0f + gamma) * ws + alpha);
  } else {
    dl = (-cv - alpha * l) / (1.0f * ws + alpha);
  }
  rec[k].w = l + dl;
  const V3 n0 = p0 + dir * (w0 * dl), n1 = p1 + dir * (-w1 * dl);
  sp.s[e.x & 0xFFFFu] = make_float4(n0.x, n0.y, n0.z, w0);
  sp.st(e.y, make_float4(n1.x, n1.y, n1.z, w1));
}

template <bool kFull, bool kBone>
__global__ void __launch_bounds__(kResThreads, 1) k_solver_resident(SolverArgs a, ResidentArgs t) {
  extern __shared__ float4 res_smem[];
  const bool one = t.ctas == 1u;
  const uint32_t K = t.ctas, rank = blockIdx.x;
  float4* sp = res_smem;
  float4* sx = sp + t.chunk;
  float4* sv = sx + (kFull ? t.chunk : 0u);
  float4* rec = sv + (kFull ? t.chunk : 0u);
  uint2* ids = reinterpret_cast<uint2*>(rec + t.ccap);
  uint32_t* steps = reinterpret_cast<uint32_t*>(ids + t.ccap);
  const uint32_t base = min(rank * t.chunk, a.n), nown = min(t.chunk, a.n - base);
  const uint32_t* tab = t.tab + rank * (t.nsteps + 1u);
  const uint32_t c0 = tab[0], ncon = tab[t.nsteps] - c0;
  const float dts = a.sp.dt;
  for (uint32_t s = threadIdx.x; s <= t.nsteps; s += kResThreads) steps[s] = tab[s] - c0;
  for (uint32_t s = threadIdx.x; s < nown; s += kResThreads) {
    const uint32_t v = t.order[base + s];
    const float4 x = a.x4[v], p = a.p4[v];
    sp[s] = make_float4(p.x, p.y, p.z, x.w);
    if (kFull) {
      sx[s] = x;
      sv[s] = a.v4[v];
    }
  }
  const float dt = fmaxf(dts, 1e-8f);
  for (uint32_t k = threadIdx.x; k < ncon; k += kResThreads) {
    const float4 c = t.par[c0 + k];
    uint2 e = t.ids[c0 + k];
    if (c.y >= 1e9f) e.x |= kResOffT;
    if (c.z >= 1e9f) e.x |= kResOffC;
    ids[k] = e;
    rec[k] = make_float4(c.x, c.y / (dt * dt), c.z / (dt * dt), 0.f);
  }
  const ResSlice slice{sp, rank}, slice_x{sx, rank};
  const ResPin pinm{sp, t.sid};
  const uint32_t pin_lo = a.npins ? t.pin_tab[rank] : 0u, pin_hi = a.npins ? t.pin_tab[rank + 1u] : 0u;
  auto pins = [&] {
    for (uint32_t k = pin_lo + threadIdx.x; k < pin_hi; k += kResThreads)
      pin_one_m(t.pin_idx[k], a.pin_v, a.pin_t, pinm, dts);
  };
  auto sewing = [&] {
    for (uint32_t c = 0; c < a.nsc; ++c) {
      const uint32_t* r = t.sew_tab + c * (K + 1u);
      if (r[0] == r[K]) continue;
      for (uint32_t k = r[rank] + threadIdx.x; k < r[rank + 1u]; k += kResThreads)
        project_sewing_m<true>(t.sew_idx[k], a.sew_ids, a.sew_rest, ResSew{slice, t.sid, a.p4}, a.slam, dts, a.sw);
      res_sync(one);
    }
  };
  auto own = [&](auto&& f) {
    for (uint32_t s = threadIdx.x; s < nown; s += kResThreads)
      f(t.order[base + s], ResOwn<kFull>{sp, sx, sv, a.x4, a.p4, a.v4, s});
  };
  __syncthreads();
  for (uint32_t sub = 0; sub < a.nsub; ++sub) {
    for (uint32_t c = 0; c < a.nsc; ++c) {
      const uint32_t* r = t.sew_tab + c * (K + 1u);
      for (uint32_t k = r[rank] + threadIdx.x; k < r[rank + 1u]; k += kResThreads) {
        const uint32_t i = t.sew_idx[k];
        a.slam[i] = 0.f;
        float2 q = __ldcg(a.sew_rest + i);
        q.x = fmaxf(q.y, q.x - a.sew_speed * dt);
        a.sew_rest[i] = q;
      }
    }
    own([&](uint32_t v, const ResOwn<kFull>& m) { predict_vertex_m(v, m, a.sp); });
    for (uint32_t it = 0; it < a.iters; ++it) {
      if (a.npins) {
        if (it == 0) __syncthreads();  // the slice's own predicted positions
        pins();
      }
      if (it == 0 || a.npins) res_sync(one);
      uint32_t lo = 0;
      for (uint32_t s = 0; s < t.nsteps; ++s) {
        if (s == t.ndsteps && a.nsc) sewing();
        const uint32_t hi = steps[s + 1u];
        for (uint32_t k = lo + threadIdx.x; k < hi; k += kResThreads)
          res_project<kFull>(k, c0, ids[k], rec, it == 0u, slice, slice_x, a, t);
        lo = hi;
        res_sync(one);
      }
      if (t.nsteps == t.ndsteps && a.nsc) sewing();
      if (a.hascol && a.coupled) {
        own([&](uint32_t v, const ResOwn<kFull>& m) { collide_vertex_m<kBone>(v, m, a.ca, dts); });
        if (it + 1u < a.iters && !a.npins) res_sync(one);
        else __syncthreads();
      }
    }
    if (a.iters_only) {  // collision, pins and update are launches of their own
      __syncthreads();
      continue;
    }
    // the rest of the substep touches only the CTA's own slice
    if (a.hascol && !a.coupled) own([&](uint32_t v, const ResOwn<kFull>& m) { collide_vertex_m<kBone>(v, m, a.ca, dts); });
    if (a.npins) {
      __syncthreads();
      pins();
      __syncthreads();
    }
    if (a.with_update) {
      if (a.nsc) {  // final sewing
        res_sync(one);
        sewing();
      }
      own([&](uint32_t v, const ResOwn<kFull>& m) { update_vertex_m(v, m, dts); });
    }
  }
  for (uint32_t s = threadIdx.x; s < nown; s += kResThreads) {
    const uint32_t v = t.order[base + s];
    const float4 p = sp[s];
    a.p4[v] = make_float4(p.x, p.y, p.z, a.p4[v].w);
    if (kFull) {
      a.x4[v] = sx[s];
      a.v4[v] = sv[s];
    }
  }
}

}  // namespace tcloth
