// Persistent-thread traversal for the wavefront's extend and shadow kernels.
//
// Each lane owns one ray at a time; a warp takes new rays from the queue
// when enough of its lanes stand idle (Aila & Laine, "Understanding the
// Efficiency of Ray Traversal on GPUs", HPG 2009: persistent threads with
// dynamic fetch). A ray has up to two pieces of work at hand: a node to
// visit and triangles of one parked leaf to test (their speculative
// traversal with postponed leaves). Each step the warp votes which kind of
// work to do, one node visit or one triangle test per lane that has it, so
// whichever more lanes wait for goes first and no phase is held up by its
// slowest lane.
//
// The traversal stack keeps its first entries in shared memory (one column
// per thread, conflict-free) and the deeper ones in local memory. Rays walk
// either node layout of the scene: two-child 64-byte nodes or the same tree
// as quantised four-child 64-byte nodes (fewer, wider steps).
//
// These loops are bound by instruction issue and by the registers that a
// resident ray takes (1,024 rays an SM leave 64 each), so what a ray can
// look up again when it needs it, at a hit or at its end, is not held.
//
// Results equal closest_hit / occluded of dev_scene.cuh: the closest hit is
// the accepted candidate with the smallest t (ties: lowest global id), a
// definition that does not depend on traversal order, and the any-hit
// answer is a yes/no.
#pragma once

#include "dev_scene.cuh"

namespace ptd {

// Stack entries a thread keeps in shared memory. A node visit whose pushes
// stay within them takes the short, branch-free way; L1 loses what they take.
// Extend + shadow stage at 8 / 12 / 16 / 20 / 24 entries: 500k-triangle soup
// 100.8 / 94.0 / 86.5 / 83.9 / 83.3 ms a frame, stress scene 62.0 / 56.6 /
// 55.7 / 56.0 / 56.1 ms, sphere grid 50.6 / 49.5 / 49.3 / 49.7 / 49.6 ms.
constexpr int kShortStack = 16;
constexpr int kTravDone = (int)0x80000000;  // "no next node": neither a node index nor a leaf reference
// Rows of a block's shared words, one word per thread each: the stack, then
// the thread's node visits, triangle tests and rays.
enum TravRows : int { ROW_NODES = kShortStack, ROW_TRIS, ROW_RAYS, ROW_COUNT };

PT_DEV int shared_load(uint32_t a) {
  int v;
  asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
PT_DEV void shared_store(uint32_t a, int v) { asm volatile("st.shared.s32 [%0], %1;" ::"r"(a), "r"(v)); }

// A thread's stack: `sp` is the shared byte address of the next free row of
// its column (rows past kShortStack live in `spill`); kThreads is a power of
// two, so the address gives the column too.
template <int kThreads>
struct TravStack {
  static constexpr uint32_t kRow = 4u * kThreads;
  uint32_t sp;
  int spill[kTravStackSize - kShortStack];
  // The block's shared words start at address `words` (a constant).
  static PT_DEV uint32_t limit(uint32_t words) { return words + kShortStack * kRow; }
  // An empty stack holds kTravDone, so popping needs no test.
  PT_DEV void reset(uint32_t words) {
    sp = words + 4u * threadIdx.x;
    shared_store(sp, kTravDone);
    sp += kRow;
  }
  PT_DEV bool room_for_three(uint32_t words) const { return sp < limit(words) - 2u * kRow; }
  PT_DEV void push_shared(bool yes, int v) {
    if (yes) {
      shared_store(sp, v);
      sp += kRow;
    }
  }
  PT_DEV int pop_shared() {
    sp -= kRow;
    return shared_load(sp);
  }
  PT_DEV void push(uint32_t words, int v, DevCounters *ctr) {
    const uint32_t lim = limit(words);
    if (sp < lim) {
      shared_store(sp, v);
    } else {
      const uint32_t i = (sp - lim) / kRow;
      if (i >= (uint32_t)(kTravStackSize - kShortStack)) {
        atomicOr(&ctr->error_flags, (unsigned)ERR_STACK_OVERFLOW);
        return;
      }
      spill[i] = v;
    }
    sp += kRow;
  }
  PT_DEV int pop(uint32_t words) {
    const uint32_t lim = limit(words);
    sp -= kRow;
    return sp < lim ? shared_load(sp) : spill[(sp - lim) / kRow];
  }
  // One more of what `row` counts for this thread.
  PT_DEV void count(uint32_t words, int row) const {
    const uint32_t a = words + ((sp - words) & (kRow - 1u)) + (uint32_t)row * kRow;
    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(a));
  }
};

// Traversal state of one ray. `cur` is the next node (>= 0), a leaf that
// waits for the parked one (< 0) or kTravDone; `leaf` the parked leaf's
// records still to test (first | count << kLeafCountShift). A leaf waits in
// `cur` only while `leaf` holds records, but for the empty leaves of unused
// child slots (settle).
constexpr uint32_t kOneRecord = 1u << kLeafCountShift;
template <int kThreads, bool kOnly4>
struct TravCore {
  V3 o, inv;
  float sx, sy, sz;
  uint32_t axes;  // kx | ky << 2 | kz << 4
  const Bvh4Node *nodes4;
  const BvhNode *nodes2;
  const float4 *tris;
  int cur;
  uint32_t leaf;
  float t_far;
  bool wide;

  PT_DEV void start(const DevScene &s, V3 org, V3 dir, float tmax, bool wide_nodes, TravStack<kThreads> &stk,
                    uint32_t words) {
    const Ray r = make_ray(org, dir);
    o = r.o;
    inv = r.inv;
    sx = r.sx;
    sy = r.sy;
    sz = r.sz;
    axes = (uint32_t)(r.kx | r.ky << 2 | r.kz << 4);
    nodes4 = s.nodes4;
    nodes2 = s.nodes;
    tris = s.tris;
    cur = s.node_count ? 0 : kTravDone;
    leaf = 0;
    t_far = tmax;
    wide = wide_nodes && s.nodes4;
    stk.reset(words);
  }
  PT_DEV void idle() {
    cur = kTravDone;
    leaf = 0;
  }
  PT_DEV bool wants_node() const { return cur >= 0; }
  PT_DEV bool wants_tri() const { return leaf >= kOneRecord; }
  // A leaf in `cur` (not a node, not kTravDone).
  PT_DEV bool leaf_waits() const { return (uint32_t)cur > 0x80000000u; }
  // Parks the leaf in `cur` when no other is parked.
  PT_DEV void settle(TravStack<kThreads> &stk, uint32_t words) {
    if (leaf < kOneRecord && leaf_waits()) {
      leaf = (uint32_t)~cur;
      cur = stk.pop(words);
    }
  }

  // Visits node `cur`: the nearest hit child is next, the others go on the
  // stack farthest first.
  PT_DEV void node_step(TravStack<kThreads> &stk, uint32_t words, DevCounters *ctr) {
    stk.count(words, ROW_NODES);
    if (kOnly4 || wide) {
      const Bvh4Node *nd = nodes4 + cur;
      const NodeVisit4 nv(nd, o, inv, t_far);
      const int4 &ch = nv.child;
      const uint32_t none = NodeVisit4::kNone, first = nv.first, second = nv.second, third = nv.third, last = nv.last;
      if (stk.room_for_three(words)) {
        // Everything below stays in shared memory: no branches but the last.
        if (third != none) {
          stk.push_shared(last != none, child_of(ch, last));
          stk.push_shared(true, child_of(ch, third));
        }
        stk.push_shared(second != none, child_of(ch, second));
        cur = child_of(ch, first);
        if (first == none) cur = stk.pop_shared();
        if (leaf < kOneRecord && leaf_waits()) {
          leaf = (uint32_t)~cur;
          cur = stk.pop_shared();
        }
        return;
      }
      if (last != none) stk.push(words, child_of(ch, last), ctr);
      if (third != none) stk.push(words, child_of(ch, third), ctr);
      if (second != none) stk.push(words, child_of(ch, second), ctr);
      cur = first != none ? child_of(ch, first) : stk.pop(words);
    } else {
      Ray r;
      r.o = o;
      r.inv = inv;
      bool h0, h1;
      float e0, e1;
      int4 dd;
      node_boxes(nodes2 + cur, r, 0.0f, t_far, h0, h1, e0, e1, dd);
      const bool swap = e1 < e0;
      if (h0 && h1) stk.push(words, swap ? dd.x : dd.y, ctr);
      cur = h0 && h1 ? (swap ? dd.y : dd.x) : (h0 ? dd.x : (h1 ? dd.y : stk.pop(words)));
    }
    settle(stk, words);
  }

  // Tests the parked leaf's next triangle. `hit(g, flags, t, b0, b1, b2,
  // front)` is called for one that the ray meets at t >= 0.
  template <class OnHit>
  PT_DEV void tri_step(TravStack<kThreads> &stk, uint32_t words, const OnHit &hit) {
    stk.count(words, ROW_TRIS);
    const float4 *tr = tris + 3u * (leaf & kLeafFirstMask);
    const float4 p0 = ldg4(tr), p1 = ldg4(tr + 1), p2 = ldg4(tr + 2);
    leaf += 1u - kOneRecord;
    Ray r;
    r.o = o;
    r.sx = sx;
    r.sy = sy;
    r.sz = sz;
    r.kx = (int)(axes & 3u);
    r.ky = (int)(axes >> 2 & 3u);
    r.kz = (int)(axes >> 4);
    float t, b0, b1, b2;
    bool front;
    if (intersect_watertight(r, {p0.x, p0.y, p0.z}, {p1.x, p1.y, p1.z}, {p2.x, p2.y, p2.z}, t, b0, b1, b2, front) &&
        t >= 0.0f)
      hit(__float_as_uint(p0.w), __float_as_uint(p1.w), t, b0, b1, b2, front);
    settle(stk, words);
  }
};

// A warp's share of the ray queue: entries [next, end) are claimed and not
// yet handed out. Lives in shared memory, read and written by whole warps.
struct WarpRun {
  uint32_t next, end, exhausted;
};
// Hands each lane with `need` its next entry of the queue's `n` (warp
// collective); true where one was taken. Claims `chunk` entries per lane
// still without one.
PT_DEV bool take_entry(WarpRun *run, uint32_t *counter, bool need, uint32_t n, uint32_t chunk, uint32_t &idx) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t mask = __ballot_sync(0xffffffffu, need);
  const uint32_t rank = __popc(mask & ((1u << lane) - 1u)), want = __popc(mask);
  const uint32_t next = run->next, have = run->end - next;
  uint32_t base = n, got = 0;
  if (want > have && !run->exhausted) {
    got = (want - have) * chunk;
    if (lane == 0) base = atomicAdd(counter, got);
    base = __shfl_sync(0xffffffffu, base, 0);
    got = base < n ? min(got, n - base) : 0u;
  }
  const uint32_t taken = min(want - min(want, have), got);  // of the new entries
  __syncwarp();
  if (lane == 0) {
    if (want > have) {
      run->next = base + taken;
      run->end = base + got;
      if (got < (want - have) * chunk) run->exhausted = 1u;
    } else {
      run->next = next + want;
    }
  }
  __syncwarp();
  if (!need) return false;
  if (rank < have) {
    idx = next + rank;
    return true;
  }
  idx = base + (rank - have);
  return rank - have < taken;
}

}  // namespace ptd
