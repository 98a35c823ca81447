"""Traversal of the quantised four-child nodes (the wavefront's voted steps,
and the raycast backend's walk in its own tests) against the two-child nodes,
whose boxes are full precision, in the wavefront and in the megakernel: the
accumulators are equal bit for bit for geometry of any size, place and
distance from the camera, for rays along the axes, for deep stacks and for
queues smaller than a warp."""
import copy
import math

import numpy as np
import pytest

from oxideav_render_b200 import abi, api, testscenes as ts
from oxideav_render_b200.scene import PreparedScene, Primitive

pytestmark = pytest.mark.gpu


def placed_soup(tris, scale, offset, distance):
    """A soup of unit extent scaled, moved, and seen from `distance` extents."""
    s = copy.deepcopy(ts.random_soup(tris, seed=5))
    for it in s.items:
        it.positions = (it.positions.astype(np.float64) * scale + offset).astype(np.float32)
    s._bounds = None
    s.cameras = []
    mid = np.array([0.5, 0.5, 0.5]) * scale + offset
    s.add_camera(list(mid + np.array([0.03, 0.02, 0.5 + distance]) * scale), list(mid),
                 2.0 * math.atan(0.6 / (0.5 + distance)))
    return s


def both(ctx, scene, opts):
    """(accumulator, ray counts) with the four-child nodes, then with the
    two-child ones; the megakernel (two-child nodes, one thread a path) must
    agree with them."""
    out = []
    for schedule, width in ((abi.PT_SCHEDULE_WAVEFRONT, 4), (abi.PT_SCHEDULE_WAVEFRONT, 2),
                            (abi.PT_SCHEDULE_MEGAKERNEL, 4)):
        ctx.set_schedule(schedule)
        ctx.set_node_width(width, width)
        try:
            t = api.PathTracer(ctx)
            t.sync(scene, opts)
            t.refine(opts.path_trace.samples_per_pixel)
            out.append((t.accum(), t.ray_counts()))
            t.close()
        finally:
            ctx.set_schedule(abi.PT_SCHEDULE_WAVEFRONT)
            ctx.set_node_width(4, 4)
    assert np.array_equal(out[0][0], out[2][0], equal_nan=True) and out[0][1] == out[2][1]
    return out[:2]


@pytest.mark.parametrize("scale,offset,distance", [(1.0, 0.0, 1.0), (1e-3, 0.0, 600.0), (1e4, -3e4, 0.1),
                                                   (1.0, 300.0, 50.0), (1e-6, 0.0, 1.0), (1e9, 0.0, 3.0)])
@pytest.mark.parametrize("builder", ["auto", "spatial"])
def test_placed_geometry(ctx, scale, offset, distance, builder):
    ctx.set_bvh_builder(abi.PT_BVH_BUILD_HOST_SPATIAL if builder == "spatial" else abi.PT_BVH_BUILD_AUTO)
    try:
        (a, ra), (b, rb) = both(ctx, placed_soup(20000, scale, offset, distance),
                                ts.pt_opts(61, 3, 4, h=47, ambient=0.4))
    finally:
        ctx.set_bvh_builder(abi.PT_BVH_BUILD_AUTO)
    assert np.array_equal(a, b) and ra == rb
    assert a[..., 3].sum() > 0.3 * 61 * 47  # the soup is in view


def test_axis_parallel_rays_and_flat_boxes(ctx):
    # Walls whose triangles lie in axis planes, seen straight on by an
    # orthographic camera: zero direction components, boxes without depth.
    s = PreparedScene()
    m = s.add_material(ts.diffuse_material((0.7, 0.6, 0.5), 1.0))
    rng = np.random.default_rng(3)
    for k in range(40):
        x, y = rng.uniform(-1, 1, 2)
        z, e = float(rng.integers(0, 4)) * 0.25, rng.uniform(0.05, 0.4)
        s.add_primitive(ts.with_material(ts.quad([[x, y, z], [x + e, y, z], [x + e, y + e, z], [x, y + e, z]]), m))
    from oxideav_render_b200.options import CameraSpec, Projection
    o = ts.pt_opts(96, 2, 3, ambient=0.5, scene_camera=None, camera=CameraSpec(0.0, 0.0, 4.0),
                   projection=Projection.Orthographic)
    (a, ra), (b, rb) = both(ctx, s, o)
    assert np.array_equal(a, b) and ra == rb


def test_unbounded_and_missing_corners(ctx):
    # Triangles reaching out to 1e30 and to infinity, and one with a NaN
    # corner, among ordinary ones: their boxes bound nothing on some axes.
    s = copy.deepcopy(ts.random_soup(3000, seed=9))
    m = s.items[0].material
    far = np.array([[-1e30, 0.2, -1e30], [1e30, 0.2, -1e30], [0.0, 0.2, 1e30],
                    [0.1, 0.1, -np.inf], [0.3, 0.1, 0.5], [0.2, np.inf, 0.5],
                    [np.nan, 0.1, 0.2], [0.3, 0.1, 0.5], [0.2, 0.4, 0.5]], np.float32)
    s.add_primitive(Primitive(far, material=m))
    (a, ra), (b, rb) = both(ctx, s, ts.pt_opts(48, 2, 3, ambient=0.3))
    assert np.array_equal(a, b, equal_nan=True) and ra == rb


@pytest.mark.parametrize("threads,chunk", [(256, 1), (256, 4), (128, 2)])
@pytest.mark.parametrize("width,height", [(1, 1), (5, 3), (33, 1), (257, 31)])
def test_small_queues(ctx, width, height, threads, chunk):
    ctx.set_traversal(threads, chunk)
    try:
        (a, ra), (b, rb) = both(ctx, ts.random_soup(500, seed=2), ts.pt_opts(width, 2, 5, h=height, ambient=0.3))
    finally:
        ctx.set_traversal(256, 1)
    assert np.array_equal(a, b) and ra == rb


def test_stacks_deeper_than_shared_memory(ctx):
    # A long thin row of overlapping slabs seen end on: every node's children
    # are all hit, so stacks outgrow their shared-memory rows.
    s = PreparedScene()
    m = s.add_material(ts.diffuse_material((0.8, 0.8, 0.8), 1.0))
    n = 3000
    z = -np.geomspace(1.0, 4000.0, n)
    tri = np.array([[-1.0, -1.0, 0.0], [1.0, -1.0, 0.0], [0.0, 1.5, 0.0]])
    pos = (tri[None] * (1.0 + 0.001 * np.arange(n)[:, None, None]) + np.stack([0 * z, 0 * z, z], 1)[:, None]).astype(
        np.float32)
    mask = ts.Texture(np.array([[[255, 255, 255, 0]]], np.uint8))
    cut = ts.diffuse_material((0.8, 0.8, 0.8), 1.0)
    cut.alpha_mode, cut.alpha_cutoff = abi.PT_ALPHA_MASK, 0.5
    cut.base_color = (0.8, 0.8, 0.8, 0.1)  # cut out everywhere: a ray meets every slab
    s.textures.append(mask)
    mc = s.add_material(cut)
    s.add_primitive(Primitive(np.ascontiguousarray(pos[:-1].reshape(-1, 3)), material=mc))
    s.add_primitive(Primitive(np.ascontiguousarray(pos[-1:].reshape(-1, 3)), material=m))
    s.add_camera([0.0, 0.1, 3.0], [0.0, 0.1, 0.0], 0.2)
    (a, ra), (b, rb) = both(ctx, s, ts.pt_opts(24, 2, 3, ambient=0.3))
    assert np.array_equal(a, b) and ra == rb
