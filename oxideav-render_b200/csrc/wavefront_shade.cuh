// The wavefront's shading kernel. Each occupancy is a translation unit of its
// own (shade3.cu, shade4.cu): the kernel takes a minute to compile.
#pragma once

#include "kernels.h"
#include "wavefront_state.cuh"

namespace ptd {

// Emission, material, light samples and the next direction of every queued
// vertex. kPlain: the entries of plain materials and misses, [0, cut) of the
// material-sorted queue; otherwise the layered ones, [cut, n), or the whole
// queue when it is not sorted. kThreads * kBlocks threads share an SM.
//
// Some 1,500 instructions (plain) to 4,000 run once per vertex, straight
// down, from 12 to 16 warps: bound by instruction fetch and by the latency
// of scattered loads. A block's warps therefore start each vertex together
// and fetch the same code (the barrier of the loop's condition), and the
// plain materials' smaller code and state have a kernel of their own. Stage
// times with neither (and all of a path's state read and written) / the
// barrier / both: sphere grid 31.0 / 27.4 / 20.2 ms a frame, stress scene
// 46.9 / 27.3 / 25.1, material extensions 4.20 / 2.94 / 2.62. Prefetching the
// next vertex's state made all of them slower (1 to 10 %, without the
// barrier).
template <int kThreads, int kBlocks, bool kPlain>
__global__ void __launch_bounds__(kThreads, kBlocks) k_wf_shade(WaveBuffers w, uint32_t iter) {
  __shared__ BlockAppend<kThreads> append;
  const DevRequest *reqs = w.desc->reqs;
  uint32_t n = w.counters[iter * kWfCounterStride + 0], begin = 0;
  if (w.sort_materials) {
    const uint32_t cut = w.counters[iter * kWfCounterStride + 5];
    if (kPlain)
      n = cut;
    else
      begin = cut;
  }
  const uint32_t *q = w.sort_materials ? w.q_sorted : w.q[iter & 1u];
  uint32_t *q_next = w.q[(iter + 1) & 1u];
  uint32_t *n_next = w.counters + (iter + 1) * kWfCounterStride + 0;
  uint32_t *n_shadow = w.counters + iter * kWfCounterStride + 1;
  for (uint32_t i = begin + blockIdx.x * blockDim.x + threadIdx.x; __syncthreads_or(i < n);
       i += gridDim.x * blockDim.x) {
    uint32_t slot = 0, shadow_rays = 0;
    bool alive = false;
    if (i < n) {
      slot = q[i];
      PathState ps;
      const DevRequest &rq = reqs[wf_load_vertex(w, slot, iter, ps)];
      const uint32_t hg = w.hit_g[slot];
      const bool found = (hg & HIT_FOUND) != 0;
      Hit h;
      if (found) {
        const float4 tb = w.hit_tb[slot];
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
      alive = shade<DeferredSink, true, kPlain>(rq, ps, found, h, sink, &pre);
      wf_store_vertex(w, slot, iter, ps, alive);
      w.sh_n[slot] = shadow_rays = sink.count;
    }
    append.run(slot, alive, shadow_rays, q_next, n_next, w.q_shadow, n_shadow, n_shadow + 3);
  }
}

}  // namespace ptd
