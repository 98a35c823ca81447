"""Small refines: a context whose schedule nobody chose runs them on the
megakernel up to a size that depends on area lights; the accumulator and the
ray counts are those of the wavefront on both sides of each limit, alone and
in a batch, and over several calls. Which schedule ran is asked, not assumed."""
import numpy as np
import pytest

from oxideav_render_b200 import abi, api, testscenes as ts

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
        return t.accum(), rays, t.samples(), schedules
    finally:
        c.close()


@pytest.mark.parametrize("lit", [True, False])
@pytest.mark.parametrize("width,height", [(1, 1), (127, 97), (192, 128), (193, 128), (384, 256), (385, 256)])
def test_small_refines_equal_the_wavefront(lit, width, height):
    scene = ts.cornell_c0()[0] if lit else ts.sphere_grid(3, 2, 12, 6)
    o = ts.pt_opts(width, 1, 5, h=height, ambient=0.3)
    calls = (1, 1, 2)
    a, ra, na, sa = render(False, scene, o, calls)
    b, rb, nb, sb = render(True, scene, o, calls)
    assert np.array_equal(a, b) and ra == rb and na == nb == 4
    limit = (24 if lit else 96) << 10
    assert sa == [M if n * width * height <= limit else W for n in calls] and sb == [W, W, W]


def test_small_batch_equals_the_wavefront():
    scenes = [ts.cornell_c0()[0], ts.material_extensions(), ts.random_soup(800, seed=4)]
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
