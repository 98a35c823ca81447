// The wavefront's shading kernel. Each occupancy is a translation unit of its
// own (shade3.cu, shade4.cu): the kernel takes a minute to compile.
#pragma once

#include "kernels.h"
#include "wavefront_state.cuh"

namespace ptd {

// kBlocks 128-thread blocks per SM. Three (168 registers) measured faster
// than the unconstrained 234-register build despite a few spills, and than
// four on scenes with light shading (C1); four (128 registers, more
// spills) is faster where shading is heavy (C2's f64 area-light sampling).
// The tuner picks per scene class.
template <int kBlocks>
__global__ void __launch_bounds__(128, kBlocks) k_wf_shade(WaveBuffers w, uint32_t iter) {
  const DevRequest *reqs = w.desc->reqs;
  const uint32_t n = w.counters[iter * kWfCounterStride + 0];
  const uint32_t *q = w.sort_materials ? w.q_sorted : w.q[iter & 1u];
  uint32_t *q_next = w.q[(iter + 1) & 1u];
  uint32_t *n_next = w.counters + (iter + 1) * kWfCounterStride + 0;
  uint32_t *n_shadow = w.counters + iter * kWfCounterStride + 1;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    uint32_t slot = q[i];
    PathState ps;
    uint32_t request = wf_load(w, slot, ps);
    const DevRequest &rq = reqs[request];
    uint32_t hg = w.hit_g[slot];
    bool found = (hg & HIT_FOUND) != 0;
    Hit h;
    if (found) {
      float4 tb = w.hit_tb[slot];
      h.t = tb.x;
      h.b0 = tb.y;
      h.b1 = tb.z;
      h.b2 = tb.w;
      h.g = hg & HIT_G_MASK;
      h.front = (hg & HIT_FRONT) != 0;
    }
    DeferredSink sink{&w, slot, 0};
    NeeInput pre;
    pre.area.go = false;
    pre.pl_emit = 0.0f;
    if (found && (rq.env || rq.scene->em_count > 0)) {
      const size_t cap = w.capacity;
      const float4 n2 = w.nee[2 * cap + slot];
      pre.area.go = n2.y != 0.0f;
      pre.area.skip = __float_as_uint(n2.x);
      pre.pl_emit = n2.z;
      if (pre.area.go) {
        const float4 n0 = w.nee[slot], n1 = w.nee[cap + slot];
        pre.area.l = {n0.x, n0.y, n0.z};
        pre.area.pl = n0.w;
        pre.area.le = {n1.x, n1.y, n1.z};
        pre.area.tmax = n1.w;
      }
    }
    bool alive = shade<DeferredSink, true>(rq, ps, found, h, sink, &pre);
    wf_store_vertex(w, slot, ps);
    w.sh_n[slot] = sink.count;
    wf_append(q_next, n_next, alive, slot);
    wf_append(w.q_shadow, n_shadow, sink.count > 0, slot);
    wf_max(n_shadow + 3, sink.count);
  }
}

}  // namespace ptd
