"""Performance cases of the path tracer: what programs built on it have it do.

A case is a dict of plain values; "kind" says which use it stands for:

frame  an interactive viewer: a resident scene, one sample per pixel per call (`render_iter`)
       with the tone-mapped picture written to a device buffer the program displays, as the
       reference's `pathtrace(pbo, frame, iter)` is called once per displayed frame.
still  an offline picture on a resident scene: `reset`, `render` of all its samples, and the
       FP32 sum read back into page-locked host memory.
cold   a one-off job from host buffers: `Renderer` on a host scene (upload, BVH build, light
       tables, textures), `render`, read-back, `close`.
rays   a program that traces its own rays (picking, visibility, baking): `trace_rays` or, for
       batches of at most 65,536 rays that must not allocate, `trace_rays_static`, on host
       buffers.
jobs   a render farm's batch: many jobs of uneven size, sample count and depth over several
       resident scenes in one job engine.

Scenes are the library's procedural ones: the 36-triangle Cornell box and the random instanced
scenes (10k to 1M triangles, textured, with an HDRI) the repository's benchmark and tests use.
The seed picks the scene's own seed, the camera pose on the orbit the serving workload uses,
and the first iteration (the random streams).
"""
import functools
import math
import random

import numpy as np
import torch

import luxion_b200 as lx
from luxion_b200 import _ffi
from luxion_b200.workloads import CAMERA_LOOK, CAMERA_POS, scene_params

LAYOUTS = {"auto": _ffi.BVH_AUTO, "two": _ffi.BVH_TWO_LEVEL, "single": _ffi.BVH_SINGLE_LEVEL}
TEXSTORE = {"float": 0, "unorm8": 1, "half": 2}  # LUX_TEXSTORE_*
NEE = {"none": {}, "dmis": {"direct_light_sampling": 1}, "emis": {"env_importance_sampling": 1},
       "both": {"direct_light_sampling": 1, "env_importance_sampling": 1}}


def _case(name, kind, **kw):
    """A case with the options a program leaves alone at their defaults."""
    c = {"kind": kind, "tris": 0, "width": 0, "height": 0, "spp": 1, "depth": 8, "nee": "none", "layout": "auto",
         "texstore": "float", "compensated": False, "sorted": False, "rays": 0, "mode": 0, "static": False, "jobs": 0}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls: launches and latency decide
        _case("frame_cornell_256", "frame", width=256, height=256, nee="dmis", depth=8),
        _case("still_thumb_50k", "still", tris=50_000, width=161, height=91, spp=2, nee="emis", depth=8),
        _case("rays_static_4k_any", "rays", tris=200_000, rays=4096, mode=2, static=True),
        # ordinary ones
        _case("rays_300k_closest", "rays", tris=200_000, rays=300_001, mode=0),
        _case("still_dmis_odd", "still", tris=200_000, width=961, height=541, spp=8, nee="dmis", depth=8),
        _case("still_plain_two_level", "still", tris=200_000, width=640, height=480, spp=16, depth=6, layout="two"),
        _case("still_sorted", "still", tris=200_000, width=800, height=600, spp=4, nee="both", depth=8, sorted=True),
        _case("still_precise_half", "still", tris=1_000_000, width=512, height=512, spp=32, nee="both", depth=12,
              texstore="half", compensated=True),
        _case("jobs_24_mixed", "jobs", tris=200_000, jobs=24, nee="both", depth=12),
        # a full-size frame, a one-off job of a full-size scene, and the largest still
        _case("frame_1080p_1m", "frame", tris=1_000_000, width=1920, height=1080, nee="both", depth=12),
        _case("cold_1m_360p", "cold", tris=1_000_000, width=640, height=360, spp=4, nee="both", depth=12),
        _case("still_1080p_1m_16spp", "still", tris=1_000_000, width=1920, height=1080, spp=16, nee="both", depth=12),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["frame", "still", "still", "still", "cold", "rays", "jobs"])
    tris = _log(rng, 10_000, 1_000_000)
    depth = rng.randint(3, 12)
    nee = rng.choice(["none", "dmis", "emis", "both", "both"])
    layout = rng.choice(["auto", "auto", "two"])
    if kind == "rays":
        static = rng.random() < 0.3
        return _case(None, "rays", tris=tris, rays=_log(rng, 200, 65_536 if static else 2_000_000), mode=rng.randint(0, 2),
                     static=static, layout=layout)
    if kind == "jobs":
        return _case(None, "jobs", tris=_log(rng, 10_000, 400_000), jobs=rng.randint(2, 32), nee=nee, depth=depth)
    width = _log(rng, 96, 1920)
    height = max(54, min(1080, int(width * rng.uniform(0.5, 1.0))))
    if kind == "frame":
        if rng.random() < 0.3:
            tris = 0  # the Cornell box has no environment map
            nee = rng.choice(["none", "dmis"])
        return _case(None, "frame", tris=tris, width=width, height=height, nee=nee, depth=depth, layout=layout)
    if kind == "cold":
        return _case(None, "cold", tris=tris, width=min(width, 960), height=min(height, 540), spp=_log(rng, 1, 8), nee=nee,
                     depth=depth, layout=layout)
    spp = _log(rng, 1, 64)
    while width * height * spp > 1920 * 1080 * 16:
        spp = max(1, spp // 2)
    sort = rng.random() < 0.15
    if sort:
        spp = max(1, min(spp, 4_000_000 // (width * height)))
    return _case(None, "still", tris=tris, width=width, height=height, spp=spp, nee=nee, depth=depth, layout=layout,
                 texstore=rng.choice(["float", "float", "unorm8", "half"]), compensated=rng.random() < 0.3, sorted=sort)


@functools.lru_cache(maxsize=6)
def _host_scene(tris, scene_seed, half):
    """A host scene as a program has it loaded. Its generation is not part of any pass; a scene
    is kept, as several states of one program would share it."""
    if tris == 0:
        return lx.cornell36(256, 256)
    p = scene_params(tris, scene_seed, half)
    p.update(texture_size=512, tex_half=int(half))
    if tris < 500_000:
        p.update(env_width=1024, env_height=512)
    return lx.random_scene(**p)


def _camera(case, rng, width, height):
    if case["tris"] == 0:
        return lx.make_camera(width, height, (rng.uniform(-0.4, 0.4), rng.uniform(0.8, 1.2), 3.4), (0.0, 1.0, 0.0), 40.0)
    a = rng.uniform(0.0, 2.0 * math.pi)
    r = math.hypot(CAMERA_POS[0], CAMERA_POS[2])
    return lx.make_camera(width, height, (r * math.sin(a), CAMERA_POS[1], r * math.cos(a)), CAMERA_LOOK, 45.0)


def _options(case):
    return lx.default_options(trace_depth=case["depth"], bvh_layout=LAYOUTS[case["layout"]],
                              texture_storage=TEXSTORE[case["texstore"]], precision=int(case["compensated"]),
                              ray_sorting=int(case["sorted"]), **NEE[case["nee"]])


def _pinned(height, width):
    return torch.empty((height, width, 3), dtype=torch.float32, pin_memory=True).numpy()


def _rays(case, seed):
    """Rays of a baking or visibility pass: from points around the scene into it, a third of
    them from close above the ground in every direction; mode 1 has a finite reach."""
    g = np.random.default_rng(seed)
    n = case["rays"]
    o = g.uniform((-12, 0.2, -12), (12, 8, 12), (n, 3))
    o[: n // 3, 1] = g.uniform(0.0, 1.0, n // 3)
    d = g.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3], r[:, 4:7] = o, d
    r[:, 3] = g.uniform(2.0, 40.0, n) if case["mode"] == 1 else 1e16
    r[:, 7] = np.arange(n, dtype=np.int32).view(np.float32)
    return r


def prepare(case, seed):
    rng = random.Random(seed)
    st = {"case": case, "iter": 1 + rng.randrange(100_000)}
    half = case["texstore"] == "half"
    opt = _options(case)
    kind = case["kind"]
    if kind == "jobs":
        scenes = [_host_scene(max(10_000, case["tris"] // d), seed % 2 + d, half) for d in (1, 2, 4)]
        st["engine"] = lx.Engine(scenes, opt)
        mix = random.Random(case["jobs"])  # the batch's shape is the case's, its pictures are the seed's
        jobs = []
        for k in range(case["jobs"]):
            w, h = mix.choice([(128, 128), (256, 256), (321, 181), (512, 512), (640, 360)])
            jobs.append(dict(scene=mix.randrange(3), spp=mix.choice([1, 4, 7, 16]), first_iter=1 + rng.randrange(1000),
                             trace_depth=mix.randint(max(2, case["depth"] - 6), case["depth"]),
                             camera=_camera(case, rng, w, h)))
        st["jobs"] = jobs
        return st
    host = _host_scene(case["tris"], seed % 3, half)
    if kind == "rays":
        st["renderer"] = lx.Renderer(lx.ResidentScene(host, opt), opt, camera=_camera(case, rng, 64, 64))
        st["rays"] = _rays(case, seed)
        return st
    w, h = case["width"], case["height"]
    cam = _camera(case, rng, w, h)
    if kind == "cold":
        st.update(host=host, options=opt, camera=cam, out=_pinned(h, w))
        return st
    st["renderer"] = lx.Renderer(lx.ResidentScene(host, opt), opt, camera=cam)
    if kind == "frame":
        st["pbo"] = torch.zeros((h, w, 4), dtype=torch.uint8, device="cuda")
        st["sum"] = torch.zeros((h, w, 3), dtype=torch.float32, device="cuda")
    else:
        st["out"] = _pinned(h, w)
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "frame":
        # the next frame of a running viewer: the picture keeps accumulating
        r = st["renderer"]
        r.render_iter(st["iter"], st["pbo"].data_ptr())
        r.copy_image_device(st["sum"].data_ptr())
        st["iter"] += 1
        return {"pbo": st["pbo"], "sum": st["sum"]}
    if kind == "still":
        r = st["renderer"]
        r.reset()
        r.render(st["iter"], case["spp"])
        return r.image_sum_into(st["out"])
    if kind == "cold":
        st["host"].desc.camera = st["camera"]
        r = lx.Renderer(st["host"], st["options"])
        r.render(st["iter"], case["spp"])
        r.image_sum_into(st["out"])
        r.close()
        return st["out"]
    if kind == "rays":
        f = st["renderer"].trace_rays_static if case["static"] else st["renderer"].trace_rays
        return f(st["rays"], case["mode"], st["iter"])
    e = st["engine"]
    ids = [e.submit(**j) for j in st["jobs"]]
    e.run()
    out = [e.image(i) for i in ids]
    for i in ids:
        e.release(i)
    return out


def work(case):
    """Inputs once, outputs once, and the arithmetic of the rays: a sample takes about 1.9
    bounces on the scenes here (Russian roulette from the third on), each with a radiance ray
    and, under NEE, a shadow ray for the hits (about 0.65); a ray makes about 14 node visits of 8
    box tests (13 operations each) and 4 triangle tests (50); a bounce shades with about 800
    operations."""
    scene = case["tris"] * (36 + 12 + 24) + (0 if case["tris"] == 0 else 16 * 512 * 512 * 4 + 1024 * 512 * 16)
    ray = 14 * 8 * 13 + 4 * 50
    if case["kind"] == "rays":
        return {"bytes": case["rays"] * 52 + scene, "flops": case["rays"] * ray}
    if case["kind"] == "jobs":
        samples, pixels = case["jobs"] * 130_000 * 7, case["jobs"] * 130_000
    else:
        pixels = case["width"] * case["height"]
        samples = pixels * case["spp"]
    bounces = min(1.9, case["depth"])
    rays = samples * bounces * (1.0 if case["nee"] == "none" else 1.65)
    return {"bytes": scene + pixels * (28 if case["kind"] == "frame" else 12), "flops": rays * ray + samples * bounces * 800}


def exact(case, seed):
    """A rendered picture has no 64-bit value that plain array code could give in seconds, and
    hit records are identities and bit patterns, which have to stay equal as they are."""
    return None
