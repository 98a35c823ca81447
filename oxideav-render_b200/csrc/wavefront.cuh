// Wavefront schedule of the path loop: the per-vertex steps of
// dev_integrator.cuh run as separate kernels over compacted queues of path
// slots, with the path state held in structure-of-arrays form.
//
//   k_wf_raygen   camera rays for every slot of the wave (active queue 0);
//   k_wf_extend   closest hit of each queued path (wavefront_trace.cuh:
//                 traversal only, small register footprint, high occupancy);
//   k_wf_nee      per queued vertex, the area-light sample of next-event
//                 estimation and the emission MIS pdf (the f64
//                 spherical-triangle and environment sampling), kept out of
//                 the shade kernel's instruction footprint;
//   k_wf_shade    emission, material, BSDF, NEE shadow-ray generation, BSDF
//                 sampling, roulette (wavefront_shade.cuh); survivors are
//                 appended to the next active queue and paths with shadow
//                 rays to the shadow queue (one atomic per block and queue);
//   k_wf_shadow   one lane per queued shadow ray (ray k of every path
//                 before ray k + 1): whether it reaches its light;
//   k_wf_shadow_add  each path's visible contributions, added to its
//                 radiance in generation order.
// The contributions of a vertex therefore reach the radiance sum in the
// reference's order (emission, punctual lights, area sample, next vertex):
// the per-sample radiance is bit-identical to the megakernel's.
// Queue lengths live in device memory (one counter block per bounce), so a
// wave runs max_bounces + 1 iterations without a host round trip; kernels
// of an exhausted iteration exit at once.
#pragma once

#include "dev_integrator.cuh"
#include "wavefront_state.cuh"

namespace ptd {

// Camera rays for every slot of the wave (grid-stride over the wave's
// slots, read from the wave descriptor).
__global__ void __launch_bounds__(256) k_wf_raygen(WaveBuffers w) {
  const WaveDesc wd = *w.desc;
  if (blockIdx.x == 0 && threadIdx.x == 0) w.counters[0] = wd.total;
  for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < wd.total; slot += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = wd.nseg;
    while (hi - lo > 1) {
      uint32_t mid = (lo + hi) >> 1;
      if (wd.segs[mid].slot_begin <= slot)
        lo = mid;
      else
        hi = mid;
    }
    const WaveSegment &seg = wd.segs[lo];
    const DevRequest &rq = wd.reqs[seg.request];
    uint32_t local = slot - seg.slot_begin;
    uint32_t sidx = local / seg.pixel_count, i = local - sidx * seg.pixel_count;
    uint32_t p = seg.pixel_begin + i;
    uint32_t y = p / rq.width, x = p - y * rq.width;
    PathState ps;
    init_path(rq, x, y, seg.sample_begin + sidx, ps);
    wf_store_camera(w, slot, ps, seg.request);
    w.q[0][slot] = slot;
  }
}

// In-order f64 accumulation of the wave's per-slot results into each
// request's accumulator (a pixel's samples in index order, as the
// reference's per-pixel loop adds them).
__global__ void __launch_bounds__(256) k_wf_accumulate(WaveBuffers w) {
  const WaveDesc wd = *w.desc;
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t sg = 0; sg < wd.nseg; ++sg) {
    const WaveSegment seg = wd.segs[sg];
    double4 *accum = reinterpret_cast<double4 *>(wd.reqs[seg.request].accum) + seg.pixel_begin;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < seg.pixel_count; i += stride) {
      double4 a = accum[i];
      const float4 *src = w.rad + seg.slot_begin + i;
      for (uint32_t k = 0; k < seg.spp; ++k) {
        float4 v = src[(size_t)k * seg.pixel_count];
        if (v.w > 0.0f) {
          // Non-finite radiance counts as a covered black sample (src/pathtrace.rs:2324-2328).
          if (!(isfinite(v.x) && isfinite(v.y) && isfinite(v.z))) v = make_float4(0.0f, 0.0f, 0.0f, v.w);
          a.x += (double)v.x;
          a.y += (double)v.y;
          a.z += (double)v.z;
          a.w += 1.0;
        }
      }
      accum[i] = a;
    }
  }
}

// ---- material sort: the active queue bucketed by (scene, material) before
// shade, stable within each warp's group of equal keys. Bucket 0 holds the
// paths whose ray missed.
// Tiles of kSortTile queue entries per block: a shared-memory histogram per
// tile, then one global atomic per non-empty bucket (the hot buckets - the
// material most paths hit - would serialise per-warp global atomics).
constexpr uint32_t kSortPerThread = 8, kSortTile = 256 * kSortPerThread;

__global__ void __launch_bounds__(256) k_wf_sort_count(WaveBuffers w, uint32_t iter) {
  __shared__ uint32_t hist[kSortBuckets];
  const uint32_t n = w.counters[iter * kWfCounterStride + 0];
  uint32_t *count = w.sort_counts + (size_t)iter * 2 * kSortBuckets;
  const uint32_t t = threadIdx.x;
  for (uint32_t base = blockIdx.x * kSortTile; base < n; base += gridDim.x * kSortTile) {
    hist[t] = 0;
    __syncthreads();
#pragma unroll
    for (uint32_t e = 0; e < kSortPerThread; ++e) {
      const uint32_t i = base + e * 256 + t;
      if (i < n) atomicAdd(&hist[w.sort_keys[i]], 1u);
    }
    __syncthreads();
    if (hist[t]) atomicAdd(count + t, hist[t]);
    __syncthreads();
  }
}

// One block of kSortBuckets threads: bucket sizes -> start cursors.
__global__ void __launch_bounds__(kSortBuckets) k_wf_sort_scan(WaveBuffers w, uint32_t iter) {
  __shared__ uint32_t s[kSortBuckets];
  uint32_t *count = w.sort_counts + (size_t)iter * 2 * kSortBuckets;
  const uint32_t t = threadIdx.x;
  const uint32_t own = count[t];
  s[t] = own;
  __syncthreads();
  for (uint32_t off = 1; off < kSortBuckets; off <<= 1) {
    uint32_t v = t >= off ? s[t - off] : 0u;
    __syncthreads();
    s[t] += v;
    __syncthreads();
  }
  count[kSortBuckets + t] = s[t] - own;
  if (t == kLayeredBucket) w.counters[iter * kWfCounterStride + 5] = s[t] - own;
}

__global__ void __launch_bounds__(256) k_wf_sort_scatter(WaveBuffers w, uint32_t iter) {
  __shared__ uint32_t hist[kSortBuckets], start[kSortBuckets];
  const uint32_t n = w.counters[iter * kWfCounterStride + 0];
  const uint32_t *q = w.q[iter & 1u];
  uint32_t *cursor = w.sort_counts + (size_t)iter * 2 * kSortBuckets + kSortBuckets;
  const uint32_t t = threadIdx.x;
  for (uint32_t base = blockIdx.x * kSortTile; base < n; base += gridDim.x * kSortTile) {
    hist[t] = 0;
    __syncthreads();
    uint32_t key[kSortPerThread], rank[kSortPerThread];
#pragma unroll
    for (uint32_t e = 0; e < kSortPerThread; ++e) {
      const uint32_t i = base + e * 256 + t;
      key[e] = i < n ? w.sort_keys[i] : 0u;
      rank[e] = i < n ? atomicAdd(&hist[key[e]], 1u) : 0u;
    }
    __syncthreads();
    if (hist[t]) start[t] = atomicAdd(cursor + t, hist[t]);
    __syncthreads();
#pragma unroll
    for (uint32_t e = 0; e < kSortPerThread; ++e) {
      const uint32_t i = base + e * 256 + t;
      if (i < n) w.q_sorted[start[key[e]] + rank[e]] = q[i];
    }
    __syncthreads();
  }
}

// The area-light sample and emission MIS pdf of every queued vertex that
// hit something, in the order shade will read them (its queue). Values are
// those shade would compute inline (the same functions on the same inputs).
// 1,024 threads per SM (64 registers, a few spills): the sampling is latency
// bound (CDF searches, dependent f64 steps), so occupancy beats the
// spill-free 106-register form (Cornell box 2.06 ms a frame at 512 threads,
// 1.81 at 768 of 80 registers). The barrier keeps a block's warps on the same
// code, as in k_wf_shade: blocks of 256 without it 1.74, with it 1.66, of 512
// 1.62 (stress scene 12.5 / 12.3 / 11.8).
constexpr int kNeeThreads = 512, kNeeBlocks = 2;
__global__ void __launch_bounds__(kNeeThreads, kNeeBlocks) k_wf_nee(WaveBuffers w, uint32_t iter) {
  if (!(w.desc->flags & WAVE_AREA_LIGHTS)) return;  // nothing to sample in this wave
  const DevRequest *reqs = w.desc->reqs;
  const uint32_t n = w.counters[iter * kWfCounterStride + 0];
  const uint32_t *q = w.sort_materials ? w.q_sorted : w.q[iter & 1u];
  const size_t cap = w.capacity;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; __syncthreads_or(i < n); i += gridDim.x * blockDim.x) {
    if (i >= n) continue;
    const uint32_t slot = q[i];
    const uint32_t hg = w.hit_g[slot];
    if (!(hg & HIT_FOUND)) continue;
    const uint4 sd = w.seed[slot];
    const DevRequest &rq = reqs[sd.w];
    const DevScene &s = *rq.scene;
    if (!rq.env && s.em_count == 0) continue;  // shade reads nothing for this request
    const uint32_t k = iter;  // every queued path is at this vertex
    const uint32_t g = hg & HIT_G_MASK;
    const float4 tb = w.hit_tb[slot];
    const V3 pos = interp3(s.pos, g, tb.y, tb.z, tb.w);
    float pl_emit = 0.0f;
    if (k > 0) {
      const float4 pv = w.prev[slot];
      pl_emit = emission_light_pdf(rq, s, g, {pv.x, pv.y, pv.z}, pos);
    }
    AreaSample as;
    as.go = false;
    if (k < rq.max_bounces && area_nee(rq, s)) {
      Sampler smp;
      smp.pixel_seed = sd.x;
      smp.index = sd.y;
      smp.path_seed = sd.z;
      float pl_u[4];
      smp.pattern(2 + 2 * k, pl_u);
      as = sample_area_light(rq, s, pos, pl_u);
    }
    if (as.go) {
      w.nee[slot] = make_float4(as.l.x, as.l.y, as.l.z, as.pl);
      w.nee[cap + slot] = make_float4(as.le.x, as.le.y, as.le.z, as.tmax);
    }
    w.nee[2 * cap + slot] = make_float4(__uint_as_float(as.skip), as.go ? 1.0f : 0.0f, pl_emit, 0.0f);
  }
}

// Each queued path's visible shadow-ray contributions, added to its
// radiance in generation order (the order the reference adds them).
__global__ void __launch_bounds__(256) k_wf_shadow_add(WaveBuffers w, uint32_t iter) {
  const uint32_t n = w.counters[iter * kWfCounterStride + 1];
  for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
    const uint32_t slot = w.q_shadow[q];
    const uint32_t cnt = w.sh_n[slot];
    const float4 r = w.rad[slot];
    V3 rad = {r.x, r.y, r.z};
    for (uint32_t k = 0; k < cnt; ++k) {
      const size_t e = (size_t)k * w.capacity + slot;
      if (w.sh_vis[e]) {
        const float4 c = w.sh_c[e];
        rad = vadd(rad, {c.x, c.y, c.z});
      }
    }
    w.rad[slot] = make_float4(rad.x, rad.y, rad.z, r.w);
  }
}

}  // namespace ptd
