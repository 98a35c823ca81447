// The wavefront schedule's traversal kernels: closest hits of the queued
// paths (extend) and any-hit tests of their shadow rays (shadow), over the
// path state and queues of wavefront.cuh.
#pragma once

#include "dev_integrator.cuh"
#include "dev_traverse.cuh"

namespace ptd {

// A warp writes out its finished rays and takes new ones once this many of
// its lanes stand idle: it costs a few hundred instructions and a chain of
// loads, which the whole warp waits for however few lanes take part. Extend
// on the sphere grid / stress scene / 500k-triangle soup, ms a frame, at 10,
// 14, 18 lanes: 27.4 / 33.5 / 50.9, 26.4 / 33.3 / 51.6, 25.9 / 32.7 / 53.3;
// shadow rays, which are shorter: 24.1 / 22.6 / 34.5, 23.5 / 22.5 / 34.4,
// 22.9 / 22.4 / 34.8. With every finished ray replaced at once 39.4 / 51.5 /
// 72.1 and 35.6 / 27.2 / 53.4.
constexpr int kRefillExtend = 14, kRefillShadow = 18;
// Steps of one kind between votes (a vote and its control flow are a tenth
// of a step): extend 28.1 / 35.5 / 53.5 with one node visit a vote, 26.9 /
// 34.0 / 52.5 with two, 27.0 / 33.7 / 52.9 with three; with two triangle
// tests as well as two visits 26.4 / 33.3 / 51.6.
constexpr int kStepsPerVote = 2;

// The shared words of a traversal block: the stacks and counts by row (only
// touched through shared_load / shared_store / TravStack::count), then each
// warp's run of queue entries.
template <int kThreads>
struct TraceShared {
  uint32_t rows[ROW_COUNT][kThreads];
  WarpRun runs[kThreads / 32];
  PT_DEV uint32_t words() const { return (uint32_t)__cvta_generic_to_shared(&rows[0][0]); }
  PT_DEV uint32_t word(int row) const { return words() + 4u * ((uint32_t)row * kThreads + threadIdx.x); }
  PT_DEV void reset() {
    shared_store(word(ROW_NODES), 0);
    shared_store(word(ROW_TRIS), 0);
    shared_store(word(ROW_RAYS), 0);
    if (threadIdx.x % 32 == 0) runs[threadIdx.x / 32] = WarpRun{0, 0, 0};
    __syncwarp();
  }
  PT_DEV uint32_t counted(int row) const { return (uint32_t)shared_load(word(row)); }
  PT_DEV WarpRun *run() { return runs + threadIdx.x / 32; }
  // No entry is left for this warp (valid after take_entry).
  PT_DEV bool drained() { return run()->exhausted && run()->next >= run()->end; }
};

// AcceptFilter for a queued ray of path `slot`; the sampler's seeds are only
// read for the stochastic-transparency coin.
PT_DEV bool accept_candidate(const WaveBuffers &w, uint32_t slot, uint32_t ray, bool primary, uint32_t g,
                             uint32_t rflags, float b0, float b1, float b2, bool front) {
  if (primary && !front && !(rflags & REC_DOUBLE_SIDED)) return false;
  if (rflags & REC_OPAQUE) return true;
  const uint4 sd = w.seed[slot];
  const DevScene &s = *w.desc->reqs[sd.w].scene;
  Sampler smp;
  smp.pixel_seed = sd.x;
  smp.index = sd.y;
  smp.path_seed = sd.z;
  const AcceptFilter slow{&s, &smp, ray, primary, 0xffffffffu};
  return slow(g, rflags, 0.0f, b0, b1, b2, front);
}

// The material-sort key of a ray that hit (a miss has key 0), stored by queue position, so the
// count / scatter passes read keys and slots contiguously.
PT_DEV uint32_t sort_key(const DevScene *s, uint32_t g) {
  const uint2 info = __ldg(s->tri_info + g);
  const uint32_t h = info.x + (uint32_t)((uintptr_t)s >> 8) * 0x9E3779B1u;
  return (info.y & TRI_PLAIN) ? 1u + h % (kLayeredBucket - 1u) : kLayeredBucket + h % (kSortBuckets - kLayeredBucket);
}

// Closest hit of every queued path: persistent lanes, one ray each, refilled
// from the queue as rays finish (dev_traverse.cuh), w.claim_chunk entries a
// lane at a time. kThreads per block, 1,024 threads per SM.
// kOnly4: every request of the wave walks the four-child layout for
// extension rays (WaveBuffers::all_wide).
template <int kThreads, bool kOnly4>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads) k_wf_extend(WaveBuffers w, uint32_t iter,
                                                                       DevCounters *ctr) {
  __shared__ TraceShared<kThreads> sh;
  const uint32_t words = sh.words();
  sh.reset();
  // A queue entry's path is at vertex `iter`: entries of iteration k were
  // appended by the shading of vertex k - 1.
  const bool primary = iter == 0;
  TravStack<kThreads> stk;
  TravCore<kThreads, kOnly4> tr;
  tr.idle();
  stk.sp = words + 4u * threadIdx.x;
  constexpr uint32_t kNoEntry = 0xffffffffu;
  uint32_t qpos = kNoEntry;  // the queue entry this lane holds
  uint32_t found = 0;        // its closest hit so far, as WaveBuffers::hit_g (0: none)
  // The warp turns to the queue when at most this many lanes have work; once
  // it has no entries left, only when none has.
  int refill_at = 32 - kRefillExtend;
  for (;;) {
    const uint32_t nodes = __ballot_sync(0xffffffffu, tr.wants_node());
    const uint32_t leaves = __ballot_sync(0xffffffffu, tr.wants_tri());
    if (__popc(nodes | leaves) <= refill_at) {
      bool busy = tr.wants_node() || tr.wants_tri();
      if (!busy && tr.leaf_waits()) {  // behind an empty leaf
        tr.settle(stk, words);
        busy = true;
      }
      const uint32_t *q = w.q[iter & 1u];
      if (!busy && qpos != kNoEntry) {  // write the finished ray out
        const uint32_t slot = q[qpos];
        w.hit_g[slot] = found;
        if (w.sort_materials)
          w.sort_keys[qpos] = found ? sort_key(w.desc->reqs[w.seed[slot].w].scene, found & HIT_G_MASK) : 0u;
        qpos = kNoEntry;
      }
      const uint32_t n = w.counters[iter * kWfCounterStride + 0];
      uint32_t idx;
      if (take_entry(sh.run(), w.counters + iter * kWfCounterStride + 2, !busy, n, w.claim_chunk, idx)) {
        qpos = idx;
        const uint32_t slot = q[idx];
        const float4 o = w.o[slot], d = w.d[slot];
        const DevRequest &rq = w.desc->reqs[w.seed[slot].w];
        tr.start(*rq.scene, {o.x, o.y, o.z}, {d.x, d.y, d.z}, inf(), (rq.wide_nodes & WIDE_EXTENSION) != 0, stk,
                 words);
        found = 0;
        stk.count(words, ROW_RAYS);
      }
      if (!__any_sync(0xffffffffu, qpos != kNoEntry)) break;
      if (sh.drained()) refill_at = 0;
      continue;
    }
    if (__popc(nodes) > __popc(leaves)) {
#pragma unroll
      for (int k = 0; k < kStepsPerVote; ++k)
        if (tr.wants_node()) tr.node_step(stk, words, ctr);
    } else {
#pragma unroll 1
      for (int k = 0; k < kStepsPerVote && tr.wants_tri(); ++k)
        tr.tri_step(stk, words, [&](uint32_t g, uint32_t flags, float t, float b0, float b1, float b2, bool front) {
          if (found && !(t < tr.t_far || (t == tr.t_far && g < (found & HIT_G_MASK)))) return;
          const uint32_t slot = w.q[iter & 1u][qpos];
          if (!accept_candidate(w, slot, iter << 16, primary, g, flags, b0, b1, b2, front)) return;
          tr.t_far = t;
          found = (g & HIT_G_MASK) | HIT_FOUND | (front ? HIT_FRONT : 0u);
          w.hit_tb[slot] = make_float4(t, b0, b1, b2);
        });
    }
  }
  ThreadStats ts{sh.counted(ROW_RAYS), 0, sh.counted(ROW_NODES), sh.counted(ROW_TRIS),
                 0, 0, 0};
  flush_stats(ctr, ts);
}

// Shadow rays of the queued paths, one lane per ray: entry i of the
// flattened queue is ray k = i / n of queued path i % n (n paths, k below
// the wave's largest per-path count), so neighbouring lanes trace the same
// light's rays from neighbouring queue positions. A lane records whether
// its ray reached the light (sh_vis); k_wf_shadow_add then adds each path's
// visible contributions in generation order. Entries past a path's own
// count carry no ray. n times the largest count fits 32 bits: the arena
// holds 48 bytes per (ray, slot).
// kOnly4: every request of the wave walks the four-child layout for shadow
// rays.
template <int kThreads, bool kOnly4>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads) k_wf_shadow(WaveBuffers w, uint32_t iter,
                                                                       DevCounters *ctr) {
  __shared__ TraceShared<kThreads> sh;
  const uint32_t words = sh.words();
  sh.reset();
  TravStack<kThreads> stk;
  TravCore<kThreads, kOnly4> tr;
  tr.idle();
  stk.sp = words + 4u * threadIdx.x;
  constexpr uint32_t kNoEntry = 0xffffffffu;
  uint32_t entry = kNoEntry;  // the flattened queue entry this lane holds
  bool occluded = false;
  int refill_at = 32 - kRefillShadow;  // as in k_wf_extend
  for (;;) {
    const uint32_t nodes = __ballot_sync(0xffffffffu, tr.wants_node());
    const uint32_t leaves = __ballot_sync(0xffffffffu, tr.wants_tri());
    if (__popc(nodes | leaves) <= refill_at) {
      bool busy = tr.wants_node() || tr.wants_tri();
      if (!busy && tr.leaf_waits()) {  // behind an empty leaf
        tr.settle(stk, words);
        busy = true;
      }
      const uint32_t n = w.counters[iter * kWfCounterStride + 1];
      const uint32_t kmax = min(w.counters[iter * kWfCounterStride + 4], w.shadow_slots);
      if (!busy && entry != kNoEntry) {
        const uint32_t k = entry / n;
        w.sh_vis[(size_t)k * w.capacity + w.q_shadow[entry - k * n]] = occluded ? 0 : 1;
        entry = kNoEntry;
      }
      uint32_t idx;
      if (take_entry(sh.run(), w.counters + iter * kWfCounterStride + 3, !busy, n * kmax, w.claim_chunk, idx)) {
        const uint32_t k = idx / n;
        const uint32_t slot = w.q_shadow[idx - k * n];
        if (k < w.sh_n[slot]) {
          const DevRequest &rq = w.desc->reqs[w.seed[slot].w];
          const size_t e = (size_t)k * w.capacity + slot;
          const float4 so = w.sh_o[e], sdd = w.sh_d[e];
          tr.start(*rq.scene, {so.x, so.y, so.z}, {sdd.x, sdd.y, sdd.z}, so.w, (rq.wide_nodes & WIDE_SHADOW) != 0,
                   stk, words);
          entry = idx;
          occluded = false;
          stk.count(words, ROW_RAYS);
        }
      }
      // Lanes that drew entries without a ray draw again; the warp ends
      // once no lane holds a ray and the queue has no more.
      if (sh.drained()) {
        if (!__any_sync(0xffffffffu, entry != kNoEntry)) break;
        refill_at = 0;
      }
      continue;
    }
    if (__popc(nodes) > __popc(leaves)) {
#pragma unroll
      for (int k = 0; k < kStepsPerVote; ++k)
        if (tr.wants_node()) tr.node_step(stk, words, ctr);
    } else {
#pragma unroll 1
      for (int k = 0; k < kStepsPerVote && tr.wants_tri(); ++k) {
        bool stop = false;
        tr.tri_step(stk, words, [&](uint32_t g, uint32_t flags, float t, float b0, float b1, float b2, bool front) {
          if (!(t <= tr.t_far)) return;
          const uint32_t n = w.counters[iter * kWfCounterStride + 1], ray = entry / n;
          const uint32_t slot = w.q_shadow[entry - ray * n];
          const size_t e = (size_t)ray * w.capacity + slot;
          if (g == __float_as_uint(w.sh_c[e].w)) return;  // the light's own triangle
          stop = accept_candidate(w, slot, __float_as_uint(w.sh_d[e].w), false, g, flags, b0, b1, b2, front);
        });
        if (stop) {
          occluded = true;
          tr.idle();
        }
      }
    }
  }
  ThreadStats ts{0, sh.counted(ROW_RAYS), 0, 0, sh.counted(ROW_NODES),
                 sh.counted(ROW_TRIS), 0};
  flush_stats(ctr, ts);
}

}  // namespace ptd
