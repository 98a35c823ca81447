"""Small refines: a context whose schedule nobody chose runs them on the
megakernel where that is the faster one, by paths, bounces, shadow rays a vertex
and the tree's cost; the accumulator and the ray counts are those of the
wavefront on both sides of each limit, alone and in a batch, and over several
calls. Which schedule ran is asked, not assumed."""
import numpy as np
import pytest

from oxideav_render_b200 import abi, api, testscenes as ts
from oxideav_render_b200.scene import point_light

pytestmark = pytest.mark.gpu
W, M = abi.PT_SCHEDULE_WAVEFRONT, abi.PT_SCHEDULE_MEGAKERNEL


def render(fixed, scene, opts, calls, env=None):
    c = api.Context(0)
    try:
        if fixed:
            c.set_schedule(abi.PT_SCHEDULE_WAVEFRONT)
        t = api.PathTracer(c)
        if env is not None:
            t.set_environment(api.EnvironmentMap(env))
        t.sync(scene, opts)
        rays, schedules = [], []
        for n in calls:
            t.refine(n)
            rays.append(t.ray_counts())
            schedules.append(api.batch_schedule(c))
        return t.accum(), rays, t.samples(), schedules, c.bvh_stats(t.scene_id)["sah_cost"]
    finally:
        c.close()


def choice(paths, bounces, lights, area, cost):
    """The rule: most shadow rays a vertex by tree cost and bounces, then paths."""
    dear, long = (cost >= 64) + (cost >= 128), (bounces >= 2) + (bounces >= 8)
    rays = lights + area
    if rays > ((1, 2, 4), (0, 1, 2), (-1, -1, 1))[dear][long]:
        return W
    kpaths = 24 if area else 64 if dear == 0 and long == 2 and rays <= 2 else 48
    return M if paths <= kpaths << 10 else W


def lights(scene, n):
    scene.scene_lights = []
    for k in range(n):
        scene.add_light(point_light((1, 1, 1), 1.0 / n), [0.5 + 0.3 * k, 1.6, 1.0 - 0.2 * k], [0, -1, 0])
    return scene


@pytest.mark.parametrize("lit", [True, False])
@pytest.mark.parametrize("bounces", [1, 5, 8])
@pytest.mark.parametrize("width,height", [(1, 1), (127, 97), (192, 128), (193, 128), (256, 192), (257, 192), (256, 256),
                                          (257, 256)])
def test_small_refines_equal_the_wavefront(lit, bounces, width, height):
    scene = lights(ts.cornell_c0()[0], 0) if lit else lights(ts.sphere_grid(3, 2, 12, 6), 1)
    o = ts.pt_opts(width, 1, bounces, h=height, ambient=0.3)
    calls = (1, 1, 2)
    a, ra, na, sa, cost = render(False, scene, o, calls)
    b, rb, nb, sb, _ = render(True, scene, o, calls)
    assert np.array_equal(a, b) and ra == rb and na == nb == 4 and cost < 64
    assert sa == [choice(n * width * height, bounces, int(not lit), lit, cost) for n in calls] and sb == [W, W, W]


# Trees of SAH cost 13 (sphere grid), 77 and 374 (soups: their boxes overlap).
@pytest.mark.parametrize("kind", ["spheres", 10000, 100000])
@pytest.mark.parametrize("area", [False, True])
@pytest.mark.parametrize("bounces", [0, 1, 2, 7, 8])
def test_long_walks_and_many_lights_stay_on_the_wavefront(kind, area, bounces):
    scene = ts.sphere_grid(3, 2, 12, 6) if kind == "spheres" else ts.random_soup(kind, seed=9)
    for m in scene.materials:
        m.emissive_factor = (2.0, 2.0, 2.0) if area and m is scene.materials[-1] else (0.0, 0.0, 0.0)
    for n in (0, 1, 2, 3, 4, 5):
        o = ts.pt_opts(41, 1, bounces, h=23, ambient=0.3)
        a, ra, _, sa, cost = render(False, lights(scene, n), o, (1,))
        b, rb, _, _, _ = render(True, scene, o, (1,))
        assert np.array_equal(a, b) and ra == rb
        assert (cost >= 64) + (cost >= 128) == {"spheres": 0, 10000: 1, 100000: 2}[kind]
        assert sa == [choice(41 * 23, bounces, n, area, cost)], (n, cost)


def test_small_batch_equals_the_wavefront():
    scenes = [ts.cornell_c0()[0], lights(ts.material_extensions(), 1), lights(ts.random_soup(800, seed=4), 1)]
    out = []
    for fixed in (False, True):
        c = api.Context(0)
        try:
            if fixed:
                c.set_schedule(abi.PT_SCHEDULE_WAVEFRONT)
            tr = []
            for k, s in enumerate(scenes):
                t = api.PathTracer(c)
                t.sync(s, ts.pt_opts(31 + k, 2, 4, h=17, seed=k, ambient=0.2))
                tr.append(t)
            api.refine_many(c, tr, [2, 1, 3])
            assert api.batch_schedule(c) == (W if fixed else M)
            out.append([t.accum() for t in tr])
        finally:
            c.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)
