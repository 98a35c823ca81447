"""Scene uploads: the device binned-SAH build at the sizes where its kernels
change hands (64 triangles is its least, subtrees of at most 32 go to a warp,
tiles of 1,024), with coinciding, flat and NaN triangles, against the host
build; the context's memory pool: its reuse, its limit, and that failing
allocations give its cache back; and contexts in several threads."""
import os
import subprocess
import sys
import threading

import numpy as np
import pytest

from oxideav_render_b200 import abi, api, testscenes as ts
from oxideav_render_b200.scene import PreparedScene, Primitive

pytestmark = pytest.mark.gpu


def cloud(kind, n, seed=1):
    rng = np.random.default_rng(seed + n)
    c = rng.random((n, 1, 3)).astype(np.float32)
    e = (rng.normal(size=(n, 3, 3)) * 0.03).astype(np.float32)
    pos = c + e
    if kind == "same":  # every centroid alike: no split plane, ranges are halved
        pos[:] = pos[0]
    elif kind == "flat":
        pos[..., 1] = 0.5
    elif kind == "piles":  # a few places, many triangles each
        pos = (np.round(c * 2) / 2 + e * 0.01).astype(np.float32)
    elif kind == "nan":
        pos[::7, 1, 2] = np.nan
    s = PreparedScene()
    m = s.add_material(ts.diffuse_material((0.7, 0.6, 0.5), 1.0))
    s.add_primitive(Primitive(np.ascontiguousarray(pos.reshape(-1, 3).astype(np.float32)), material=m))
    s.add_camera([0.5, 0.6, 2.4], [0.5, 0.5, 0.5], 0.6)
    return s


def render(ctx, scene, opts):
    t = api.PathTracer(ctx)
    t.sync(scene, opts)
    t.refine(opts.path_trace.samples_per_pixel)
    out = t.accum(), ctx.bvh_stats(t.scene_id), ctx.bvh_on_device(t.scene_id)
    t.close()
    return out


@pytest.mark.parametrize("n", [64, 65, 97, 1023, 1025, 4097])
@pytest.mark.parametrize("kind", ["random", "same", "flat", "piles", "nan"])
def test_device_build_equals_the_host_build(ctx, kind, n):
    scene, o = cloud(kind, n), ts.pt_opts(33, 2, 4, h=31, ambient=0.5)
    out = {}
    for b in (abi.PT_BVH_BUILD_HOST, abi.PT_BVH_BUILD_DEVICE):
        ctx.set_bvh_builder(b)
        try:
            out[b] = render(ctx, scene, o)
        finally:
            ctx.set_bvh_builder(abi.PT_BVH_BUILD_AUTO)
    (a, sa, _), (b, sb, on_device) = out[abi.PT_BVH_BUILD_HOST], out[abi.PT_BVH_BUILD_DEVICE]
    # NaN triangles leave the scene; what is left may be too few for the device.
    assert (on_device or (kind == "nan" and n < 97)) and np.array_equal(a, b)
    if kind in ("random", "flat"):  # no fallback splits: the same tree
        assert (sa["nodes"], sa["leaves"], sa["max_depth"]) == (sb["nodes"], sb["leaves"], sb["max_depth"])
        assert sa["sah_cost"] == pytest.approx(sb["sah_cost"], rel=1e-9)


def test_uploads_and_releases_reuse_the_pool():
    scene, o = cloud("random", 50000), ts.pt_opts(16, 1, 2, ambient=0.5)
    c = api.Context(0)
    try:
        d = scene.to_desc(o)
        want, ids, one = None, [], 0
        for k in range(40):
            ids.append(c.upload(d))
            if k % 3:
                c.release(ids.pop(0))
            if k % 10 == 5:
                got = render(c, scene, o)[0]
                want = got if want is None else want
                assert np.array_equal(got, want)
            if k == 0:
                one = c.pool_bytes()[1]
        # 14 scenes stay; the 26 released ones made room for others and for
        # what the builds and renders took and returned.
        reserved, used = c.pool_bytes()
        assert len(ids) == 14 and used == 14 * one and reserved <= used + 6 * one + (128 << 20)
    finally:
        c.close()


def test_pool_keeps_at_most_a_gigabyte():
    big = ts.stress_c2(64, 64, 1, grid=384, spheres=50)[0].to_desc(ts.pt_opts(16, 1, 2))
    c = api.Context(0)
    try:
        ids, keep = [], 1 << 30
        while c.pool_bytes()[1] < 2 * keep and len(ids) < 40:
            ids.append(c.upload(big))
        one = c.pool_bytes()[1] // len(ids)
        assert c.pool_bytes()[1] >= 2 * keep and one < keep // 4
        for i in ids:
            c.release(i)
        # What is over the limit goes back in whole blocks of the pool, at the
        # next synchronisation: nothing like the 2 GiB that were in use.
        reserved, used = c.pool_bytes()
        assert used == 0 and one <= reserved <= keep + one
        # The cache serves the next upload.
        c.upload(big)
        assert c.pool_bytes()[0] <= reserved + one
    finally:
        c.close()


@pytest.mark.parametrize("which", ["upload", "refit", "accumulator", "wave arena", "another context"])
def test_a_failing_allocation_gives_the_cache_back(which):
    scene, o = cloud("random", 300000), ts.pt_opts(24, 2, 3, ambient=0.5)
    c, other = api.Context(0), api.Context(0)
    try:
        c.set_schedule(abi.PT_SCHEDULE_WAVEFRONT)
        d = scene.to_desc(o)
        kept = c.upload(d)
        used = c.pool_bytes()[1]
        gone = [c.upload(d) for _ in range(8)]
        for i in gone:
            c.release(i)
        assert c.pool_bytes()[0] >= used + (192 << 20) and c.pool_bytes()[1] == used
        t = api.PathTracer(c)
        if which == "wave arena":
            t.sync_resident(kept, scene, o)
        failing = other if which == "another context" else c
        failing.fail_allocations(1)
        with pytest.raises(api.RenderError) as e:
            if which == "refit":
                c.refit(kept, d)
            elif which == "accumulator":
                t.sync_resident(kept, scene, o)
            elif which == "wave arena":
                t.refine(2)
            else:
                failing.upload(d)
        assert e.value.status == abi.PT_ERR_OOM
        reserved, now = c.pool_bytes()
        assert now == used and reserved <= used + (64 << 20)  # whole blocks of the pool
        # Both contexts go on.
        a, b = render(c, scene, o)[0], render(other, scene, o)[0]
        assert np.array_equal(a, b)
    finally:
        c.close()
        other.close()


def test_two_contexts_in_two_threads():
    scenes = [cloud("random", 20000, 1), cloud("piles", 30000, 2)]
    o = ts.pt_opts(40, 2, 4, ambient=0.5)
    out = [[], []]

    def work(k):
        c = api.Context(0)
        try:
            c.set_schedule(abi.PT_SCHEDULE_WAVEFRONT)  # of itself so small a refine is the megakernel's
            for _ in range(6):
                out[k].append(render(c, scenes[k], o)[0])
        finally:
            c.close()

    th = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [t.start() for t in th]
    [t.join() for t in th]
    for k in range(2):
        c = api.Context(0)
        c.set_schedule(abi.PT_SCHEDULE_WAVEFRONT)
        want = render(c, scenes[k], o)[0]
        c.close()
        assert len(out[k]) == 6 and all(np.array_equal(x, want) for x in out[k])


FIRST_WAVES = """
import sys, threading, time
sys.path.insert(0, {root!r})
import __graft_entry__ as entry
entry.load_package()
import numpy as np
from oxideav_render_b200 import abi, api, testscenes as ts
scene, o = ts.sphere_grid(3, 2, 12, 6), ts.pt_opts(48, 1, 3, ambient=0.5)
N, out, failed = 8, [None] * 8, []
ready = threading.Barrier(N)

def work(k):
    try:
        c = api.Context(0)
        c.set_schedule(abi.PT_SCHEDULE_WAVEFRONT)
        c.set_traversal((256, 128)[k % 2], 1)
        t = api.PathTracer(c)
        t.sync(scene, o)
        ready.wait(60)
        time.sleep(k * {step})
        t.refine(1)
        out[k] = t.accum()
    except Exception as e:
        failed.append(repr(e))

th = [threading.Thread(target=work, args=(k,)) for k in range(N)]
[t.start() for t in th]
[t.join() for t in th]
assert not failed, failed
assert all(np.array_equal(a, out[0]) for a in out)
print("whole")
"""


@pytest.mark.parametrize("step", [0.0, 1e-4, 1e-3])
def test_first_waves_of_several_threads(step):
    """A process's first waves, started by eight contexts a little apart: the
    grid sizes are looked up while the others already launch."""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", FIRST_WAVES.format(root=root, step=step)], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "whole", r.stderr[-2000:]
