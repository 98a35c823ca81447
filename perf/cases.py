"""Performance cases of the renderer: what a program that uses it has it do,
through the package's public entry points (`PathTracer`, `refine_many`,
`PathTraceCudaRenderer`, `RaycastCudaRenderer`, `RenderServer`).

The scenes are the package's own procedural ones (`testscenes`): the Cornell
box, the material-extension showcase, grids of spheres, the stress scene
(heightfield, spheres, emitters, environment) and random triangle soups. A
case's seed is the sample seed of its images (and of a soup that moves), so
another seed gives other paths and other pixels.

Images do not depend on the acceleration structure, on scheduling or on what
else is being rendered: they are compared bit for bit.
"""
import copy
import importlib
import math
import random

import numpy as np

_pkg = importlib.import_module("oxideav-render_b200")
ts = _pkg.testscenes
api = _pkg.api
abi = _pkg.abi
options = _pkg.options
RenderServer = _pkg.serve.RenderServer

MAX_SERVED_WAIT_MS = 120_000


def listed():
    return [
        # A viewer whose camera just moved: one sample a pixel, an image back.
        # The smallest call, all launch latency.
        {"name": "preview_cornell_128_1spp", "kind": "preview", "scene": "cornell", "width": 128, "height": 128,
         "spp": 1, "bounces": 8},
        # A small closed room lit by an area emitter, long paths, tiny tree.
        {"name": "refine_cornell_256_64spp", "kind": "refine", "scene": "cornell", "width": 256, "height": 256,
         "spp": 64, "bounces": 8},
        # Every material extension, textures; a ragged image and sample count.
        {"name": "refine_khr_641x367_33spp", "kind": "refine", "scene": "khr", "width": 641, "height": 367,
         "spp": 33, "bounces": 8},
        # The sphere-grid frame of the benchmark: 200k triangles, a textured
        # floor, two punctual lights.
        {"name": "refine_spheres_512_256spp", "kind": "refine", "scene": "spheres", "width": 512, "height": 512,
         "spp": 256, "bounces": 8},
        # The benchmark's stress scene: 4.1M triangles, four material kinds,
        # emitters and an environment map, a full-HD frame.
        {"name": "refine_stress_1080p_16spp", "kind": "refine", "scene": "stress", "width": 1920, "height": 1080,
         "spp": 16, "bounces": 8},
        # Incoherent geometry: the largest soup of the benchmark's mix.
        {"name": "refine_soup500k_1024x768_16spp", "kind": "refine", "scene": "soup", "tris": 500_000, "width": 1024,
         "height": 768, "spp": 16, "bounces": 8},
        # One render call as the command-line user makes it: flatten the
        # scene, upload, build the tree, trace, read the bytes back.
        {"name": "oneshot_spheres_512_16spp", "kind": "oneshot", "scene": "spheres", "width": 512, "height": 512,
         "spp": 16, "bounces": 8},
        # Many requests of uneven size in shared waves over resident scenes.
        {"name": "batch_16_requests", "kind": "batch", "requests": 16, "mix": 5, "samples": 24_000_000},
        # The same kind of mix through the server, every image back to the host.
        {"name": "served_24_requests", "kind": "served", "requests": 24, "mix": 9, "samples": 12_000_000},
        # Two consecutive frames of an animation: refit, trace, read back.
        {"name": "animate_soup50k_320x240_4spp", "kind": "animate", "scene": "soup", "tris": 50_000, "width": 320,
         "height": 240, "spp": 4, "bounces": 4},
        # The Whitted raycast backend, supersampled, one call.
        {"name": "raycast_phong_spheres_512_aa2", "kind": "raycast", "scene": "spheres", "width": 512, "height": 512,
         "aa": 2, "shading": "Phong", "depth": 4},
        # The same backend shading with the glTF BRDF, shadows and mirrors.
        {"name": "raycast_pbr_spheres_800x600", "kind": "raycast", "scene": "spheres", "width": 800, "height": 600,
         "aa": 1, "shading": "Pbr", "depth": 4},
    ]


#: Samples of a drawn refine over each scene: no dearer than the dearest listed case.
_MOST_SAMPLES = {"cornell": 30e6, "khr": 20e6, "spheres": 67e6, "grid": 40e6, "stress": 33e6, "soup": 12e6}


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _image(rng, pixels):
    """A width and height of about `pixels` pixels, odd ones among them."""
    w = max(8, int(math.sqrt(pixels * rng.uniform(0.6, 1.9))))
    return w, max(8, int(pixels / w))


def draw(rng):
    kind = rng.choice(["preview", "refine", "refine", "refine", "oneshot", "batch", "served", "animate", "raycast"])
    if kind in ("batch", "served"):
        most = 24e6 if kind == "batch" else 12e6
        return {"kind": kind, "requests": rng.randint(3, 24), "mix": rng.randrange(1 << 20),
                "samples": int(_log(rng, 4e5, most))}
    scene = rng.choice(["cornell", "khr", "spheres", "grid", "stress", "soup"])
    case = {"kind": kind, "scene": scene}
    if kind == "animate":
        scene = case["scene"] = "soup"
    if scene == "soup":
        case["tris"] = int(_log(rng, 10_000, 100_000 if kind == "animate" else 500_000))
    if scene == "grid":
        case["cols"], case["rows"], case["segments"] = rng.randint(1, 9), rng.randint(1, 9), rng.randint(8, 96)
    if scene == "stress":
        case["grid"], case["spheres"] = rng.randint(64, 1024), rng.randint(10, 500)
    if kind == "raycast":
        case["aa"] = rng.choice([1, 1, 2, 3])
        case["width"], case["height"] = _image(rng, _log(rng, 64 * 64, 1.0e6 / case["aa"] ** 2))
        case["shading"], case["depth"] = rng.choice(["Phong", "Pbr"]), rng.randint(1, 6)
        return case
    most = _MOST_SAMPLES[scene]
    if kind == "preview":
        samples = _log(rng, 4096, 1e6)
        case["spp"] = rng.randint(1, 2)
    elif kind == "refine":
        samples = _log(rng, 2e5, most)
        case["spp"] = int(_log(rng, 4, min(256, samples / 4096)))
    else:
        samples = _log(rng, 5e4, most / 12)
        case["spp"] = int(_log(rng, 1, 16))
    case["width"], case["height"] = _image(rng, min(samples / case["spp"], 2.1e6))
    case["bounces"] = rng.choice([2, 4, 8])
    return case


# ---------------------------------------------------------------- scenes

_scenes = {}


def _scene(case):
    """(scene, options, environment pixels or None) of a case, built once."""
    name = case["scene"]
    key = (name,) + tuple(case.get(k) for k in ("tris", "cols", "rows", "segments", "grid", "spheres"))
    if key not in _scenes:
        if len(_scenes) > 16:
            _scenes.clear()
        env = None
        if name == "cornell":
            s, o = ts.cornell_c0()
        elif name == "khr":
            s, o = ts.material_extensions(), ts.pt_opts(64, 1, 8, ambient=0.2)
        elif name == "spheres":
            s, o = ts.sphere_grid_c1()
        elif name == "grid":
            s = ts.sphere_grid(case["cols"], case["rows"], case["segments"], max(case["segments"] // 2, 2))
            o = ts.pt_opts(64, 1, 8, ambient=0.3)
        elif name == "stress":
            s, o, env = ts.stress_c2(grid=case.get("grid", 1024), spheres=case.get("spheres", 500))
        else:
            s, o = ts.random_soup(case["tris"], seed=7), ts.pt_opts(64, 1, 8, ambient=0.1)
        _scenes[key] = (s, o, env)
    return _scenes[key]


def _triangles(scene):
    return sum(it.triangle_count for it in scene.items)


def _opts(o, case, seed):
    return o.replace(width=case["width"], height=case["height"],
                     path_trace=options.PathTraceOptions(samples_per_pixel=case["spp"], max_bounces=case["bounces"],
                                                         seed=seed & 0xFFFFFFFF))


def _drifted(base, seed):
    """`base` (a soup) with every triangle moved a little: the same draw items."""
    rng = np.random.default_rng(seed)
    s = copy.copy(base)
    s.items = []
    for it in base.items:
        new = copy.copy(it)
        pos = it.positions.reshape(-1, 3, 3)
        step = rng.normal(size=(pos.shape[0], 1, 3)).astype(np.float32) * np.float32(0.02)
        new.positions = np.ascontiguousarray((pos + step).reshape(it.positions.shape))
        s.items.append(new)
    s._bounds = None
    return s


# A program that renders many requests keeps its scenes: a few small and
# middling ones, uploaded or registered once.
_MIX_SCENES = [{"scene": "cornell"}, {"scene": "spheres"}, {"scene": "khr"},
               {"scene": "stress", "grid": 512, "spheres": 100}, {"scene": "soup", "tris": 20_000},
               {"scene": "soup", "tris": 120_000}]
_resident = {}


def _resident_scenes():
    """The mix's scenes on the default context, with the tree meant for
    scenes that stay resident."""
    if "ids" not in _resident:
        ctx = api.default_context()
        ctx.set_bvh_builder(abi.PT_BVH_BUILD_HOST_SPATIAL)
        try:
            descs = [_scene(c)[0].to_desc(_scene(c)[1]) for c in _MIX_SCENES]
            _resident["descs"] = descs
            _resident["ids"] = [ctx.upload(d) for d in descs]
        finally:
            ctx.set_bvh_builder(abi.PT_BVH_BUILD_AUTO)
    return _resident["ids"]


def _server():
    if "server" not in _resident:
        srv = RenderServer(api.default_context())
        keys = []
        for c in _MIX_SCENES:
            s, o, env = _scene(c)
            keys.append(srv.register(s, o, api.EnvironmentMap(env) if env is not None else None))
        _resident["server"] = (srv, keys)
    return _resident["server"]


def _requests(case):
    """The requests of a batch or served case: (scene index, width, height,
    spp, bounces), about case["samples"] samples in all, sizes uneven."""
    rng = random.Random(case["mix"])
    sizes = [(128, 128), (256, 256), (512, 512), (317, 211), (640, 480)]
    reqs = []
    for _ in range(case["requests"]):
        reqs.append([rng.randrange(len(_MIX_SCENES)), *rng.choice(sizes), rng.choice([1, 4, 16, 64]),
                     rng.choice([2, 4, 8])])
    total = sum(r[1] * r[2] * r[3] for r in reqs)
    for r in reqs:  # scale the sample counts to the total asked for
        r[3] = max(1, min(256, round(r[3] * case["samples"] / total)))
    return reqs


# ---------------------------------------------------------------- the protocol


def prepare(case, seed):
    ctx = api.default_context()
    kind = case["kind"]
    if kind in ("batch", "served"):
        reqs = _requests(case)
        opts = [_opts(_scene(_MIX_SCENES[k])[1], {"width": w, "height": h, "spp": spp, "bounces": b}, seed * 64 + i)
                for i, (k, w, h, spp, b) in enumerate(reqs)]
        if kind == "served":
            srv, keys = _server()
            for k, o in zip(keys, [_scene(c)[1] for c in _MIX_SCENES]):  # a warm server holds its scenes
                t = srv.submit(k, o.replace(width=16, height=16,
                                            path_trace=options.PathTraceOptions(samples_per_pixel=1)))
                srv.wait(t)
                srv.release(t)
            return {"kind": kind, "server": srv, "requests": [(keys[r[0]], o) for r, o in zip(reqs, opts)]}
        ids = _resident_scenes()
        tracers = []
        for r, o in zip(reqs, opts):
            scene, _, env = _scene(_MIX_SCENES[r[0]])
            t = api.PathTracer(ctx)
            if env is not None:
                t.set_environment(api.EnvironmentMap(env))
            t.sync_resident(ids[r[0]], scene, o)
            tracers.append(t)
        return {"kind": kind, "ctx": ctx, "tracers": tracers, "spp": [r[3] for r in reqs]}
    scene, o, env = _scene(case)
    if kind == "raycast":
        # The directional light (Phong) and the ambient term (Pbr) follow the seed.
        turn = random.Random(seed)
        light = options.LightSpec(azimuth_deg=turn.uniform(-80.0, 80.0), elevation_deg=turn.uniform(25.0, 70.0))
        o = o.replace(width=case["width"], height=case["height"], aa=case["aa"], light=light, ambient=turn.uniform(0.1, 0.3),
                      shading=options.ShadingMode[case["shading"]], max_ray_depth=case["depth"], shadows=True,
                      exposure=turn.uniform(0.8, 1.2))
        return {"kind": kind, "renderer": api.RaycastCudaRenderer(ctx), "scene": scene, "opts": o}
    o = _opts(o, case, seed)
    if kind == "oneshot":
        r = api.PathTraceCudaRenderer(ctx)
        if env is not None:
            r.tracer_mut().set_environment(api.EnvironmentMap(env))
        return {"kind": kind, "renderer": r, "scene": scene, "opts": o}
    if kind == "animate":
        r = api.PathTraceCudaRenderer(ctx)
        return {"kind": kind, "renderer": r, "frames": [_drifted(scene, seed * 2 + k) for k in range(2)], "opts": o}
    t = api.PathTracer(ctx)
    if env is not None:
        t.set_environment(api.EnvironmentMap(env))
    t.sync(scene, o)
    return {"kind": kind, "tracer": t, "scene": scene, "opts": o}


def run(state):
    kind = state["kind"]
    if kind == "preview":
        # The camera moved: the accumulation restarts, one refine, an image.
        t, o = state["tracer"], state["opts"]
        t.sync(state["scene"], o)
        t.reset()
        t.refine(o.path_trace.samples_per_pixel)
        return {"image": t.image(), "hdr": t.hdr()}
    if kind == "refine":
        t = state["tracer"]
        t.reset()
        t.refine(state["opts"].path_trace.samples_per_pixel)
        return t.hdr()
    if kind == "oneshot":
        return state["renderer"].render(state["scene"], state["opts"])
    if kind == "animate":
        return [state["renderer"].render_frame(s, state["opts"]) for s in state["frames"]]
    if kind == "raycast":
        return state["renderer"].render_hdr(state["scene"], state["opts"])
    if kind == "batch":
        for t in state["tracers"]:
            t.reset()
        api.refine_many(state["ctx"], state["tracers"], state["spp"])
        return [t.hdr() for t in state["tracers"]]
    srv = state["server"]
    tickets = [srv.submit(k, o) for k, o in state["requests"]]
    images = []
    for t in tickets:
        images.append(srv.wait(t, MAX_SERVED_WAIT_MS)[0])
        srv.release(t)
    return images


def _ray_flops(tris):
    # A walk down a balanced four-wide tree (four slab tests of 24 operations
    # a level) and two watertight triangle tests.
    return 96.0 * (math.log(max(tris, 4), 4) + 1) + 2 * 70.0


def _one(tris, pixels, samples, bounces):
    """Bytes and operations of one image: each triangle's corner positions and
    normals read once, the f64 accumulator read and written, the image written;
    per sample a path of about min(bounces + 1, 3.5) vertices, each with an
    extension ray, a shadow ray and 600 operations of shading."""
    vertices = samples * min(bounces + 1, 3.5)
    return 72.0 * tris + 80.0 * pixels, vertices * (2 * _ray_flops(tris) + 600.0)


def work(case):
    if case["kind"] in ("batch", "served"):
        b = f = 0.0
        seen = set()
        for k, w, h, spp, bounces in _requests(case):
            tris = _triangles(_scene(_MIX_SCENES[k])[0])
            one = _one(0 if k in seen else tris, w * h, 0, 0)[0], _one(tris, w * h, w * h * spp, bounces)[1]
            b, f = b + one[0], f + one[1]
            seen.add(k)
        return {"bytes": b, "flops": f}
    tris = _triangles(_scene(case)[0])
    px = case["width"] * case["height"]
    if case["kind"] == "raycast":
        # One camera ray and one shadow ray a sample at the least.
        return {"bytes": 72.0 * tris + 16.0 * px, "flops": px * case["aa"] ** 2 * (2 * _ray_flops(tris) + 200.0)}
    frames = 2 if case["kind"] == "animate" else 1
    b, f = _one(tris, px, px * case["spp"], case["bounces"])
    return {"bytes": frames * b, "flops": frames * f}


def tolerance(case):
    # Hits are defined by the geometry alone (the accepted candidate of
    # smallest distance, ties to the lowest id), every sample is a function of
    # (seed, pixel, index), and a pixel's samples are added in index order in
    # f64: the same bits whatever the tree, the schedule and the company.
    return "exact"


# ---------------------------------------------------------------- 64 bits


def exact(case, seed):
    """The Whitted image of the Cornell box in f64 (its materials are matt and
    opaque, so a pixel is Lambert plus ambient, a hard shadow and emission).

    None for the rest. A Monte Carlo path has no 64-bit value to compare with:
    its random choices (lobe, light, roulette) are thresholds on f32 numbers,
    and a path that takes the other branch is another, equally valid, sample;
    such images are compared bit for bit instead. The other raycast scenes
    would take minutes without an acceleration structure."""
    if case["kind"] != "raycast" or case["scene"] != "cornell" or case["shading"] != "Phong":
        return None
    state = prepare(case, seed)
    scene, o = state["scene"], state["opts"]
    aa, w, h = case["aa"], case["width"], case["height"]
    if w * h * aa * aa > 1_000_000:
        return None
    cam = _pkg.Camera.resolve(scene, o, w * aa, h * aa)
    tri, base, emit = [], [], []
    for it in scene.items:
        mat = scene.materials[it.material]
        tri.append(np.asarray(it.positions, np.float64).reshape(-1, 3, 3))
        base += [mat.base_color] * it.triangle_count
        emit += [mat.emissive_factor] * it.triangle_count
    tri, base, emit = np.concatenate(tri), np.asarray(base, np.float64), np.asarray(emit, np.float64)
    ng = np.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
    ng /= np.linalg.norm(ng, axis=1, keepdims=True)

    def nearest(org, d):
        """Distance to and index of the closest triangle of each ray."""
        t_best, g_best = np.full(len(org), np.inf), np.full(len(org), -1)
        for g, (a, b, c) in enumerate(tri):
            e1, e2 = b - a, c - a
            q = np.cross(d, e2)
            det = q @ e1
            with np.errstate(divide="ignore", invalid="ignore"):
                s = org - a
                u = np.einsum("ij,ij->i", s, q) / det
                r = np.cross(s, e1)
                v = np.einsum("ij,ij->i", d, r) / det
                t = (r @ e2) / det
                hit = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-9) & (t < t_best)
            t_best[hit], g_best[hit] = t[hit], g
        return t_best, g_best

    c = cam.to_c()
    side, up, fwd, eye = (np.array(list(v), np.float64) for v in (c.side, c.up, c.forward, c.eye))
    ys, xs = np.mgrid[0:h * aa, 0:w * aa]
    nx, ny = (xs.ravel() + 0.5) / (w * aa) * 2 - 1, 1 - (ys.ravel() + 0.5) / (h * aa) * 2
    d = side * (nx * c.half_w)[:, None] + up * (ny * c.half_h)[:, None] + fwd
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    t, g = nearest(np.broadcast_to(eye, d.shape), d)
    hit = g >= 0
    az, el = math.radians(o.light.azimuth_deg), math.radians(o.light.elevation_deg)
    light = np.array([math.cos(el) * math.sin(az), math.sin(el), math.cos(el) * math.cos(az)])
    out = np.zeros((len(d), 4))
    gh, dh = g[hit], d[hit]
    n = ng[gh] * -np.sign(np.einsum("ij,ij->i", dh, ng[gh]))[:, None]
    p = eye + dh * t[hit][:, None]
    dark = nearest(p + n * 1e-7, np.broadcast_to(light, p.shape))[1] >= 0
    f = np.clip(0.2 + 0.8 * np.maximum(n @ light, 0) * o.light.intensity, 0, 1)
    f = np.where(dark, 0.2, f)
    out[hit, :3] = base[gh, :3] * f[:, None] + emit[gh]
    out[hit, 3] = base[gh, 3]
    bg = np.array(o.background.rgba, np.float64) / 255.0
    bg[:3] = np.where(bg[:3] <= 0.04045, bg[:3] / 12.92, ((bg[:3] + 0.055) / 1.055) ** 2.4)
    out[~hit] = bg
    out = out.reshape(h, aa, w, aa, 4).transpose(0, 2, 1, 3, 4).reshape(h, w, aa * aa, 4)
    alpha = out[..., 3].sum(axis=2)
    lit = (out[..., :3] * out[..., 3:]).sum(axis=2)
    with np.errstate(divide="ignore", invalid="ignore"):
        rgb = np.where(alpha[..., None] > 0, lit / alpha[..., None], out[..., :3].mean(axis=2))
    return np.concatenate([rgb, (alpha / (aa * aa))[..., None]], axis=2)
