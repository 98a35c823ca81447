// Path state of the wavefront schedule in structure-of-arrays form: loads,
// stores and queue appends.
#pragma once

#include "dev_integrator.cuh"

namespace ptd {

enum : uint32_t { PF_MEDIUM = 1u, PF_COVERED = 2u, PF_HERO_SHIFT = 2u };

PT_DEV uint32_t wf_flags(const PathState &ps) {
  return (ps.has_medium ? PF_MEDIUM : 0u) | (ps.covered ? PF_COVERED : 0u) |
         ((uint32_t)(ps.hero + 1) << PF_HERO_SHIFT);
}

// A path at the camera: the previous vertex and the medium coefficients are
// only read once a vertex has written them.
PT_DEV void wf_store_camera(const WaveBuffers &w, uint32_t slot, const PathState &ps, uint32_t request) {
  w.o[slot] = make_float4(ps.o.x, ps.o.y, ps.o.z, 0.0f);
  w.d[slot] = make_float4(ps.d.x, ps.d.y, ps.d.z, ps.prev_pdf);
  w.beta[slot] = make_float4(ps.beta.x, ps.beta.y, ps.beta.z, __uint_as_float(wf_flags(ps)));
  w.rad[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  w.seed[slot] = make_uint4(ps.smp.pixel_seed, ps.smp.index, ps.smp.path_seed, request);
}

// What shading vertex `iter` needs of a path. The ray's origin and the
// previous vertex are not read there (the hit's position comes from its
// barycentrics, the emission's light pdf from k_wf_nee); `radiance` starts
// at zero and holds what the vertex adds.
PT_DEV uint32_t wf_load_vertex(const WaveBuffers &w, uint32_t slot, uint32_t iter, PathState &ps) {
  const float4 d = w.d[slot], b = w.beta[slot];
  const uint4 sd = w.seed[slot];
  const uint32_t flags = __float_as_uint(b.w);
  // The medium coefficients are read (and written) only inside a medium.
  const float4 s = (flags & PF_MEDIUM) ? w.sigma[slot] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  ps.o = vzero();
  ps.k = iter;
  ps.d = {d.x, d.y, d.z};
  ps.prev_pdf = d.w;
  ps.beta = {b.x, b.y, b.z};
  ps.has_medium = (flags & PF_MEDIUM) ? 1u : 0u;
  ps.covered = (flags & PF_COVERED) ? 1u : 0u;
  ps.hero = (int32_t)(flags >> PF_HERO_SHIFT) - 1;
  ps.radiance = vzero();
  ps.prev_pos = vzero();
  ps.sigma = {s.x, s.y, s.z};
  ps.smp.pixel_seed = sd.x;
  ps.smp.index = sd.y;
  ps.smp.path_seed = sd.z;
  return sd.w;
}

// Writes back a shaded vertex: the radiance it added, if any (a vertex adds
// at most once, and to a sum that is never -0, so adding to zero first
// changes no bit), and the path's next ray unless it ended here.
PT_DEV void wf_store_vertex(const WaveBuffers &w, uint32_t slot, uint32_t iter, const PathState &ps, bool alive) {
  const V3 r = ps.radiance;
  if (iter == 0) {
    w.rad[slot] = make_float4(r.x, r.y, r.z, ps.covered ? 1.0f : 0.0f);
  } else if (!(r.x == 0.0f && r.y == 0.0f && r.z == 0.0f)) {
    const float4 was = w.rad[slot];
    w.rad[slot] = make_float4(was.x + r.x, was.y + r.y, was.z + r.z, was.w);
  }
  if (!alive) return;
  w.o[slot] = make_float4(ps.o.x, ps.o.y, ps.o.z, 0.0f);
  w.d[slot] = make_float4(ps.d.x, ps.d.y, ps.d.z, ps.prev_pdf);
  w.beta[slot] = make_float4(ps.beta.x, ps.beta.y, ps.beta.z, __uint_as_float(wf_flags(ps)));
  w.prev[slot] = make_float4(ps.prev_pos.x, ps.prev_pos.y, ps.prev_pos.z, 0.0f);
  if (ps.has_medium) w.sigma[slot] = make_float4(ps.sigma.x, ps.sigma.y, ps.sigma.z, 0.0f);
}

// Appends the threads' slots to two queues (the paths that go on, the paths
// with shadow rays) and raises `most` to their largest shadow-ray count, by
// one atomic each per block (block-collective). Against one per warp, the
// shading of the sphere grid took 2 % less and the queues keep a block's
// paths together, which traces the shadow rays 1 % faster.
template <int kThreads>
struct BlockAppend {
  static constexpr int kWarps = kThreads / 32;
  uint32_t count[2][kWarps], base[2], most[kWarps];
  PT_DEV void run(uint32_t slot, bool alive, uint32_t shadow_rays, uint32_t *q_next, uint32_t *n_next,
                  uint32_t *q_shadow, uint32_t *n_shadow, uint32_t *most_rays) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t m0 = __ballot_sync(0xffffffffu, alive), m1 = __ballot_sync(0xffffffffu, shadow_rays > 0);
    const uint32_t mx = __reduce_max_sync(0xffffffffu, shadow_rays);
    if (lane == 0) {
      count[0][warp] = __popc(m0);
      count[1][warp] = __popc(m1);
      most[warp] = mx;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      uint32_t total = 0;
#pragma unroll
      for (int k = 0; k < kWarps; ++k) {
        const uint32_t c = count[threadIdx.x][k];
        count[threadIdx.x][k] = total;
        total += c;
      }
      base[threadIdx.x] = total ? atomicAdd(threadIdx.x ? n_shadow : n_next, total) : 0u;
    } else if (threadIdx.x == 32) {
      uint32_t v = 0;
#pragma unroll
      for (int k = 0; k < kWarps; ++k) v = max(v, most[k]);
      if (v) atomicMax(most_rays, v);
    }
    __syncthreads();
    const uint32_t before = (1u << lane) - 1u;
    if (alive) q_next[base[0] + count[0][warp] + __popc(m0 & before)] = slot;
    if (shadow_rays > 0) q_shadow[base[1] + count[1][warp] + __popc(m1 & before)] = slot;
  }
};

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
