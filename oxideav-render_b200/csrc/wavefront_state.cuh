// Path state of the wavefront schedule in structure-of-arrays form: loads,
// stores and queue appends.
#pragma once

#include "dev_integrator.cuh"

namespace ptd {

enum : uint32_t { PF_MEDIUM = 1u, PF_COVERED = 2u, PF_HERO_SHIFT = 2u };

PT_DEV void wf_store(const WaveBuffers &w, uint32_t slot, const PathState &ps, uint32_t request) {
  w.o[slot] = make_float4(ps.o.x, ps.o.y, ps.o.z, __uint_as_float(ps.k));
  w.d[slot] = make_float4(ps.d.x, ps.d.y, ps.d.z, ps.prev_pdf);
  uint32_t flags = (ps.has_medium ? PF_MEDIUM : 0u) | (ps.covered ? PF_COVERED : 0u) |
                   ((uint32_t)(ps.hero + 1) << PF_HERO_SHIFT);
  w.beta[slot] = make_float4(ps.beta.x, ps.beta.y, ps.beta.z, __uint_as_float(flags));
  w.rad[slot] = make_float4(ps.radiance.x, ps.radiance.y, ps.radiance.z, ps.covered ? 1.0f : 0.0f);
  w.prev[slot] = make_float4(ps.prev_pos.x, ps.prev_pos.y, ps.prev_pos.z, 0.0f);
  w.sigma[slot] = make_float4(ps.sigma.x, ps.sigma.y, ps.sigma.z, 0.0f);
  w.seed[slot] = make_uint4(ps.smp.pixel_seed, ps.smp.index, ps.smp.path_seed, request);
}

// wf_store without the sampler seeds and request, which never change after
// ray generation (shade writes back only what a vertex can change).
PT_DEV void wf_store_vertex(const WaveBuffers &w, uint32_t slot, const PathState &ps) {
  w.o[slot] = make_float4(ps.o.x, ps.o.y, ps.o.z, __uint_as_float(ps.k));
  w.d[slot] = make_float4(ps.d.x, ps.d.y, ps.d.z, ps.prev_pdf);
  uint32_t flags = (ps.has_medium ? PF_MEDIUM : 0u) | (ps.covered ? PF_COVERED : 0u) |
                   ((uint32_t)(ps.hero + 1) << PF_HERO_SHIFT);
  w.beta[slot] = make_float4(ps.beta.x, ps.beta.y, ps.beta.z, __uint_as_float(flags));
  w.rad[slot] = make_float4(ps.radiance.x, ps.radiance.y, ps.radiance.z, ps.covered ? 1.0f : 0.0f);
  w.prev[slot] = make_float4(ps.prev_pos.x, ps.prev_pos.y, ps.prev_pos.z, 0.0f);
  if (ps.has_medium) w.sigma[slot] = make_float4(ps.sigma.x, ps.sigma.y, ps.sigma.z, 0.0f);
}

PT_DEV uint32_t wf_load(const WaveBuffers &w, uint32_t slot, PathState &ps) {
  float4 o = w.o[slot], d = w.d[slot], b = w.beta[slot], r = w.rad[slot], p = w.prev[slot];
  uint4 sd = w.seed[slot];
  // The medium coefficients are read (and written) only inside a medium.
  const float4 s = (__float_as_uint(b.w) & PF_MEDIUM) ? w.sigma[slot] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  ps.o = {o.x, o.y, o.z};
  ps.k = __float_as_uint(o.w);
  ps.d = {d.x, d.y, d.z};
  ps.prev_pdf = d.w;
  uint32_t flags = __float_as_uint(b.w);
  ps.beta = {b.x, b.y, b.z};
  ps.has_medium = (flags & PF_MEDIUM) ? 1u : 0u;
  ps.covered = (flags & PF_COVERED) ? 1u : 0u;
  ps.hero = (int32_t)(flags >> PF_HERO_SHIFT) - 1;
  ps.radiance = {r.x, r.y, r.z};
  ps.prev_pos = {p.x, p.y, p.z};
  ps.sigma = {s.x, s.y, s.z};
  ps.smp.pixel_seed = sd.x;
  ps.smp.index = sd.y;
  ps.smp.path_seed = sd.z;
  return sd.w;
}

// Warp-aggregated append: one atomic per warp for the lanes with `pred`.
PT_DEV void wf_append(uint32_t *queue, uint32_t *count, bool pred, uint32_t value) {
  uint32_t active = __activemask();
  uint32_t mask = __ballot_sync(active, pred);
  if (mask == 0) return;
  uint32_t lane = threadIdx.x & 31u;
  uint32_t leader = __ffs(mask) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(count, (uint32_t)__popc(mask));
  base = __shfl_sync(active, base, leader);
  if (pred) queue[base + __popc(mask & ((1u << lane) - 1u))] = value;
}

// Warp-aggregated maximum: one atomic per warp.
PT_DEV void wf_max(uint32_t *dst, uint32_t v) {
  const uint32_t active = __activemask();
  const uint32_t m = __reduce_max_sync(active, v);
  if ((threadIdx.x & 31u) == (uint32_t)(__ffs(active) - 1) && m) atomicMax(dst, m);
}

struct DeferredSink {
  const WaveBuffers *w;
  uint32_t slot, count;
  PT_DEV void emit(const ShadowRay &sr) {
    if (count >= w->shadow_slots) return;  // host sizes shadow_slots >= lights + 1
    size_t i = (size_t)count * w->capacity + slot;
    w->sh_o[i] = make_float4(sr.o.x, sr.o.y, sr.o.z, sr.tmax);
    w->sh_d[i] = make_float4(sr.d.x, sr.d.y, sr.d.z, __uint_as_float(sr.ray_id));
    w->sh_c[i] = make_float4(sr.contrib.x, sr.contrib.y, sr.contrib.z, __uint_as_float(sr.skip));
    ++count;
  }
};

}  // namespace ptd
