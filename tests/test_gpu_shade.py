"""Wavefront shading: plain and layered materials through their own kernels,
sorted and unsorted queues, both occupancies, and what a vertex writes back
of its path, against the megakernel's one shade function: accumulators equal
bit for bit. Texture wrapping against the oracle at large and negative
coordinates: equal bit for bit."""
import numpy as np
import pytest

from oxideav_render_b200 import abi, api, testscenes as ts
from oxideav_render_b200.options import LightStrategy
from oxideav_render_b200.scene import (Camera, Clearcoat, Material, MaterialExt, PreparedScene, Sampler, Sheen, Specular,
                                       Texture, TextureRef, Transmission, Volume, lambert)

pytestmark = pytest.mark.gpu


def accum(ctx, scene, opts, env=None, schedule=abi.PT_SCHEDULE_WAVEFRONT, calls=(None,)):
    ctx.set_schedule(schedule)
    try:
        t = api.PathTracer(ctx)
        if env is not None:
            t.set_environment(api.EnvironmentMap(env))
        t.sync(scene, opts)
        for n in calls:
            t.refine(opts.path_trace.samples_per_pixel if n is None else n)
        a, rays = t.accum(), t.ray_counts()
        t.close()
        return a, rays
    finally:
        ctx.set_schedule(abi.PT_SCHEDULE_WAVEFRONT)


def kinds():
    m = {"plain": Material(base_color=(0.8, 0.5, 0.3, 1), metallic=0.4, roughness=0.4),
         "specular": Material(base_color=(0.4, 0.5, 0.9, 1), metallic=0.0, roughness=0.3,
                              ext=MaterialExt(specular=Specular(factor=0.6, color_factor=(1.0, 0.7, 0.4)), ior=1.8)),
         "clearcoat": Material(base_color=(0.2, 0.6, 0.3, 1), metallic=0.0, roughness=0.6,
                               ext=MaterialExt(clearcoat=Clearcoat(factor=1.0, roughness=0.1))),
         "sheen": Material(base_color=(0.5, 0.2, 0.5, 1), metallic=0.0, roughness=0.8,
                           ext=MaterialExt(sheen=Sheen(color_factor=(0.9, 0.8, 0.9), roughness=0.4))),
         "thin": Material(base_color=(1, 1, 1, 1), metallic=0.0, roughness=0.1,
                          ext=MaterialExt(transmission=Transmission(1.0))),
         "body": Material(base_color=(0.9, 1, 0.9, 1), metallic=0.0, roughness=0.05,
                          ext=MaterialExt(transmission=Transmission(1.0),
                                          volume=Volume(thickness=1.0, attenuation_distance=0.7,
                                                        attenuation_color=(0.4, 0.9, 0.5)), ior=1.4))}
    return m


def room(names):
    """A lit box with one sphere of each material kind (plain walls)."""
    s, o = ts.cornell_c0()
    for k, name in enumerate(names):
        mat = s.add_material(kinds()[name])
        x = -0.35 + 0.7 * k / max(len(names) - 1, 1)
        w = np.diag([0.11, 0.11, 0.11, 1.0])
        w[:3, 3] = [x, -0.3 + 0.12 * (k % 3), 0.2]
        s.add_primitive(ts.with_material(ts.uv_sphere(1.0, 24, 12), mat), w)
    s.add_light(ts.point_light((1, 0.9, 0.8), 0.4), [0.2, 0.3, 0.4], [0, -1, 0])
    return s


@pytest.mark.parametrize("names", [("plain", "specular"), ("thin", "body"),
                                   ("plain", "specular", "clearcoat", "sheen", "thin", "body")])
@pytest.mark.parametrize("strategy", [LightStrategy.Mis, LightStrategy.BsdfOnly])
def test_material_classes(ctx, names, strategy):
    s = room(names)
    o = ts.pt_opts(45, 6, 7, h=37, strategy=strategy, ambient=0.2)
    env = ts.env_noise(32, 16, np.random.default_rng(1))
    for e in (None, env):
        want = accum(ctx, s, o, e, abi.PT_SCHEDULE_MEGAKERNEL, calls=(4, 2))
        assert np.isfinite(want[0]).all()
        for sort in (True, False):
            for blocks in (3, 4):
                ctx.set_material_sort(sort)
                ctx.set_shade_blocks(blocks)
                try:
                    got = accum(ctx, s, o, e, calls=(4, 2))
                finally:
                    ctx.set_material_sort(True)
                    ctx.set_shade_blocks(3)
                assert np.array_equal(got[0], want[0]) and got[1] == want[1], (sort, blocks, e is not None)


def test_mixed_batch_of_plain_and_layered_scenes(ctx):
    # Requests of a plain scene and of layered ones share waves: the sorted
    # queue of a wave holds both classes, of several scenes.
    scenes = [room(("plain",)), room(("clearcoat", "thin")), ts.sphere_grid(3, 3, 16, 8)]
    opts = [ts.pt_opts(33, 5, 5, h=29, seed=k, ambient=0.3) for k in range(3)]
    want = [accum(ctx, s, o, schedule=abi.PT_SCHEDULE_MEGAKERNEL)[0] for s, o in zip(scenes, opts)]
    ts_ = []
    for s, o in zip(scenes, opts):
        t = api.PathTracer(ctx)
        t.sync(s, o)
        ts_.append(t)
    api.refine_many(ctx, ts_, [5, 5, 5])
    for t, w in zip(ts_, want):
        assert np.array_equal(t.accum(), w)
        t.close()


@pytest.mark.parametrize("size", [(1, 1), (2, 3), (5, 64), (1000, 7)])
@pytest.mark.parametrize("wrap", [abi.PT_WRAP_REPEAT, abi.PT_WRAP_MIRROR, abi.PT_WRAP_CLAMP])
@pytest.mark.parametrize("filt", [abi.PT_FILTER_NEAREST, abi.PT_FILTER_LINEAR])
def test_texture_wrap_equals_the_oracle(oracle, ctx, size, wrap, filt):
    w, h = size
    px = np.random.default_rng(w * 31 + h).integers(0, 256, (h, w, 4)).astype(np.uint8)
    px[..., 3] = 255
    s = PreparedScene()
    tex = s.add_texture(Texture(px, Sampler(filt, abi.PT_MIN_LINEAR if filt == abi.PT_FILTER_LINEAR
                                            else abi.PT_MIN_NEAREST, wrap, wrap)))
    m = s.add_material(Material(base_color_texture=TextureRef(tex), ext=MaterialExt(unlit=True)))
    # Bands of rising coordinates, both signs, up to and past the clamp at
    # 1e6 repeats.
    for k, (u0, u1) in enumerate([(-2.0, 3.0), (-517.3, -509.1), (9.9e4, 1.0e5), (-1.2e6, -0.9e6), (0.9e6, 1.3e6),
                                  (3.9999995, 4.0000005)]):
        q = ts.quad([[-1, k - 3, 0], [1, k - 3, 0], [1, k - 2, 0], [-1, k - 2, 0]])
        q.uvs = [np.array([[u0, u1], [u1, u1], [u1, u0], [u0, u0]], np.float32)]
        s.add_primitive(ts.with_material(q, m))
    s.add_camera([0.0, 0.0, 4.5], [0.0, 0.0, 0.0], 1.2)
    o = ts.pt_opts(64, 2, 1, ambient=0.0)
    got, _ = accum(ctx, s, o)
    desc = s.to_desc(o)
    sc = oracle.OracleScene(desc)
    t = oracle.OracleTracer(sc, Camera.resolve(s, o, 64, 64), o, None)
    t.refine(2)
    assert np.array_equal(got, np.asarray(t.accum).reshape(got.shape))
    assert got[..., 3].sum() > 0.3 * 2 * 64 * 64
