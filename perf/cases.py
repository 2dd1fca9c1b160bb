"""Timed cases of the hybrid pass and the calls around it, through the Python
host API (vulkanhybridraytracer_gb300.hybrid / diffrender).

A case is a dict of plain values; its "kind" says which part of a program's
life it stands for:

* ``frame``      the pass of one frame (hy_hybrid_forward), optionally followed
                 by the post resolve, over a G-buffer the raster pass left in
                 device memory;
* ``host``       the same from pinned host buffers (hy_hybrid_forward_host);
* ``batch``      many views of several scenes in one call (hy_batch_forward);
* ``pathtrace``  a frame of the path-traced mode;
* ``fit``        one step of fitting materials and lights to an image: render,
                 loss gradient, adjoint;
* ``build``      the acceleration structure of a newly loaded scene and the
                 first ray queries on it;
* ``refit``      a frame whose objects moved: structure update and G-buffer;
* ``trace``      ray queries (picking, probes, baking).

``listed`` are the sizes measured by name, ``draw`` gives others of the same
ranges.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300 import diffrender, scenes
from vulkanhybridraytracer_gb300.hybrid import GBUF_FP32_FORMATS, HybridContext, pass_config
from vulkanhybridraytracer_gb300.scene import Camera, Light, Material

# the reference's attachment formats (position, normal, albedo, motion, material, emissive)
PACKED_FORMATS = (L.HY_FMT_RGBA16F, L.HY_FMT_RGBA16F, L.HY_FMT_RGBA8, L.HY_FMT_RG16F, L.HY_FMT_RGBA8, L.HY_FMT_RGBA8)


# ---- the cases ---------------------------------------------------------------------
def listed():
    return [
        # the smallest frame a program renders (a preview, a thumbnail, a test scene):
        # 5k triangles, one ray per light; latency and launches
        dict(name="frame-256", kind="frame", scene="small", width=256, height=256, lights=2, spp=1, bounces=1,
             rng=0, reset=False, packed=False, f32=False, ggx=False, instanced=False, out="8", post=False, sync=False),
        # the reference application's own frame after the camera moved: its window size,
        # its attachment formats, three lights, glass and mirrors, history reprojected
        # and clamped, then the gamma resolve that is presented
        dict(name="frame-1700x900-moving", kind="frame", scene="glass", width=1700, height=900, lights=3, spp=1,
             bounces=8, rng=0, reset=True, packed=True, f32=False, ggx=False, instanced=False, out="8", post=True,
             sync=False),
        # the benchmark's frame: 1080p, 1.5M triangles, 4 area lights x 16 samples,
        # GGX-sampled reflection, steady accumulation
        dict(name="frame-1080p", kind="frame", scene="hd", width=1920, height=1080, spheres=48, subdiv=5, terrain=512,
             lights=4, spp=16, bounces=1, rng=1, reset=False, packed=False, f32=False, ggx=True, instanced=False,
             out="f8", post=False, sync=False),
        # the largest frame: 4K, 8.8M triangles in one structure, 64 lights x 1 sample
        dict(name="frame-4k-64lights", kind="frame", scene="large", width=3840, height=2160, instances=4096,
             terrain=512, lights=64, spp=1, bounces=2, rng=1, reset=False, packed=False, f32=False, ggx=False,
             instanced=False, out="f8", post=False, sync=False),
        # a scene of many placed objects kept as meshes and instances (two-level structure),
        # an odd window size, float history, the caller reading the pass's counters
        dict(name="frame-1277x719-instanced", kind="frame", scene="large", width=1277, height=719, instances=1024,
             terrain=256, lights=12, spp=4, bounces=2, rng=1, reset=False, packed=False, f32=True, ggx=False,
             instanced=True, out="f", post=False, sync=True),
        # a renderer whose G-buffer comes from host memory and whose image goes back there
        dict(name="host-960x540", kind="host", scene="hd", width=960, height=540, spheres=16, subdiv=4, terrain=256,
             lights=3, spp=4, bounces=1, rng=1, packed=False, ggx=False),
        # offline rendering of many views: mixed sizes, samples and lights over several scenes
        dict(name="batch-12-views", kind="batch", views=12, scenes=3, tris_lo=60_000, tris_hi=400_000),
        # the path-traced mode, progressive accumulation into the window's image
        dict(name="pathtrace-1280x720", kind="pathtrace", scene="hd", width=1280, height=720, spheres=24, subdiv=5,
             terrain=256, lights=4, spp=4, bounces=8, rng=1),
        # one optimisation step of the differentiable form: 64 materials, 8 lights, 82k triangles
        dict(name="fit-512", kind="fit", width=512, height=512, spp=16, bounces=1),
        # loading a scene: the default (SAH) build of 1.5M triangles, then its first queries
        dict(name="build-1505k", kind="build", spheres=48, subdiv=5, terrain=512, lbvh=False, instanced=False,
             rays=262_144),
        # a frame in which every object moved: refit of 1.5M triangles and the G-buffer at 1080p
        dict(name="refit-1080p", kind="refit", spheres=48, subdiv=5, terrain=512, instanced=False, width=1920,
             height=1080),
        # incoherent closest-hit queries (probes, baking)
        dict(name="trace-262k", kind="trace", spheres=8, subdiv=4, terrain=128, any_hit=False, rays=262_147),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_hd(rng):
    return dict(spheres=_log(rng, 4, 48), subdiv=rng.choice([3, 4, 5]), terrain=_log(rng, 64, 512))


def _spp_for(rng, pixels, lights, budget):
    """Samples per light, odd ones among them, within a budget of pixel-light samples."""
    most = max(1, min(64, int(budget / (pixels * lights))))
    return rng.choice([s for s in (1, 2, 3, 4, 5, 8, 13, 16, 32, 64) if s <= most])


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "frame", "host", "batch", "pathtrace", "fit", "build", "refit",
                       "trace", "trace"])
    if kind in ("frame", "host"):
        w = _log(rng, 200, 2560)
        h = max(64, int(w * rng.uniform(0.5, 0.8)))
        names = ["small", "glass", "textured", "hd", "hd", "large"] if kind == "frame" else ["hd"]
        c = dict(kind=kind, scene=rng.choice(names), width=w, height=h,
                 rng=rng.choice([0, 1, 1]), bounces=rng.choice([1, 2, 4, 8]),
                 packed=rng.random() < 0.4, ggx=rng.random() < 0.4)
        if c["scene"] == "hd":
            c.update(_draw_hd(rng), lights=rng.randint(1, 4))
        elif c["scene"] == "large":
            c.update(instances=_log(rng, 64, 1024), terrain=_log(rng, 64, 256), lights=_log(rng, 2, 32))
        else:
            c.update(lights=rng.randint(2, 4))
        c["spp"] = _spp_for(rng, w * h, c["lights"], 1.0e8)
        if kind == "frame":
            c.update(reset=rng.random() < 0.3, f32=rng.random() < 0.3,
                     instanced=rng.random() < (0.6 if c["scene"] == "large" else 0.15),
                     out=rng.choice(["f", "8", "f8"]), post=rng.random() < 0.3, sync=rng.random() < 0.3)
        return c
    if kind == "batch":
        return dict(kind=kind, views=rng.randint(3, 12), scenes=rng.randint(1, 3), tris_lo=50_000,
                    tris_hi=_log(rng, 60_000, 500_000))
    if kind == "pathtrace":
        w = _log(rng, 200, 1280)
        return dict(kind=kind, scene=rng.choice(["glass", "textured", "hd"]), width=w,
                    height=max(64, int(w * rng.uniform(0.5, 0.8))), **_draw_hd(rng), lights=rng.randint(2, 4),
                    spp=rng.choice([1, 2, 3, 4]), bounces=rng.choice([2, 4, 8]), rng=rng.choice([0, 1]))
    if kind == "fit":
        w = _log(rng, 128, 640)
        return dict(kind=kind, width=w, height=max(64, int(w * rng.uniform(0.6, 1.0))), spp=rng.choice([1, 4, 8, 16]),
                    bounces=rng.choice([1, 2, 4]))
    if kind == "build":
        return dict(kind=kind, **_draw_hd(rng), lbvh=rng.random() < 0.25, instanced=rng.random() < 0.25,
                    rays=_log(rng, 1_000, 100_000))
    if kind == "refit":
        w = _log(rng, 200, 1920)
        return dict(kind=kind, **_draw_hd(rng), instanced=rng.random() < 0.3, width=w,
                    height=max(64, int(w * rng.uniform(0.5, 0.8))))
    return dict(kind="trace", **_draw_hd(rng), any_hit=rng.random() < 0.4, rays=_log(rng, 1_000, 4_000_000))


# ---- scenes --------------------------------------------------------------------------
def _workload(case, seed):
    """The case's scene (a scenes.Workload) from the seed, its camera moved a little by it."""
    kind, sc = case["kind"], case.get("scene", "hd")
    w, h = int(case.get("width", 512)), int(case.get("height", 512))
    rng = np.random.default_rng(seed)
    if kind == "fit":
        wl = scenes.diff(seed, w, h)
    elif sc == "hd":
        wl = scenes.hd(seed, w, h, n_spheres=case["spheres"], sphere_subdiv=case["subdiv"], terrain_n=case["terrain"])
    elif sc == "large":
        wl = scenes.large(seed, w, h, n_instances=case["instances"], terrain_n=case["terrain"],
                          n_lights=case["lights"])
    elif sc == "textured":
        wl = scenes.small_textured(w, h)
    elif sc == "glass":
        wl = scenes.small_glass(w, h)
        wl.scene.materials[0] = Material(0, tuple(rng.random(3)) + (1.0,), 0.0, 0.6, 1.0)  # a dull floor
    else:
        wl = scenes.small(seed, w, h)
    s = wl.scene
    n = int(case.get("lights", len(s.lights)))
    while len(s.lights) < n:
        s.lights.append(Light(0, (1, 1, 1), (float(rng.uniform(-5, 5)), float(rng.uniform(4, 8)),
                                             float(rng.uniform(-5, 5))), float(rng.uniform(10, 30)), 500.0, 0.2))
    s.lights = s.lights[:n] if sc not in ("small", "glass", "textured") or n >= len(s.lights) else s.lights
    p = s.camera.position
    s.camera = Camera(tuple(float(a + d) for a, d in zip(p, rng.uniform(-0.5, 0.5, 3))), s.camera.target, s.camera.fov)
    return wl


def _context(stream, scene, instanced=False, lbvh=False):
    ctx = HybridContext(0, stream=stream.cuda_stream)
    ctx.set_scene(scene)
    if lbvh:
        ctx.set_build_mode(L.HY_BUILD_LBVH)
    ctx.build_bvh(instanced=instanced)
    return ctx


def _pack(planes):
    """The six float planes in the reference's attachment formats."""
    q = lambda p: (p.clamp(0, 1) * 255).round().to(torch.uint8)  # noqa: E731
    return [planes[0].half(), planes[1].half(), q(planes[2]), planes[3].half(), q(planes[4]), q(planes[5])]


def _rays(case, seed, device):
    """Incoherent rays in the volume over the terrain: (n, 8) origin, tmin, direction, tmax."""
    g = torch.Generator(device=device).manual_seed(int(seed))
    n = case["rays"]
    r = torch.empty((n, 8), dtype=torch.float32, device=device)
    lo = torch.tensor([-45.0, 0.5, -45.0], device=device)
    hi = torch.tensor([45.0, 14.0, 45.0], device=device)
    r[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), generator=g, device=device)
    d = torch.randn((n, 3), generator=g, device=device)
    r[:, 4:7] = d / d.norm(dim=1, keepdim=True)
    r[:, 3] = 1e-3
    r[:, 7] = 1000.0
    return r


def _moved(xf, seed, k):
    """The transforms of frame k: every object but the first (the ground) moved and scaled a little."""
    rng = np.random.default_rng([int(seed), k])
    out = xf.copy()
    n = len(xf)
    out[1:, 12:15] += rng.uniform(-0.5, 0.5, (n - 1, 3)).astype(np.float32)
    out[1:, [0, 1, 2, 4, 5, 6, 8, 9, 10]] *= rng.uniform(0.9, 1.1, (n - 1, 1)).astype(np.float32)
    return out


# ---- prepare / run ----------------------------------------------------------------------
def prepare(case, seed):
    dev = torch.device("cuda", 0)
    stream = torch.cuda.Stream(device=dev)
    with torch.cuda.stream(stream):
        st = dict(kind=case["kind"], case=case, stream=stream, frame=0)
        globals()["_prepare_" + ("frame" if case["kind"] == "host" else case["kind"])](case, int(seed), st, dev)
    torch.cuda.synchronize(dev)
    return st


def _prepare_frame(case, seed, st, dev):
    wl = _workload(case, seed)
    w, h = wl.width, wl.height
    ctx = _context(st["stream"], wl.scene, instanced=bool(case.get("instanced")))
    cam = wl.camera(0.0)
    planes = ctx.gbuffer(cam, w, h)
    formats = GBUF_FP32_FORMATS
    fmt = L.HY_ACCUM_F32 if case.get("f32") else L.HY_ACCUM_U8
    flags = L.HY_FLAG_GGX_REFLECTION if case["ggx"] else 0
    # the history a running program has: a first frame's, then a running mean goes on
    hist = ctx.new_history(w, h, fmt)
    ctx.forward(planes, cam, pass_config(1, 1, case["rng"], 0, flags), hist, fmt,
                out_8=torch.empty((h, w, 4), dtype=torch.uint8, device=dev))
    if case.get("reset"):
        # the camera moved: a smooth screen-space motion field in plane 3
        y, x = torch.meshgrid(torch.linspace(-1, 1, h, device=dev), torch.linspace(-1, 1, w, device=dev),
                              indexing="ij")
        planes[3] = torch.stack([0.5 + 0.004 * x + 0.002, 0.5 + 0.004 * y], -1).contiguous()
    if case["packed"]:
        planes, formats = _pack(planes), PACKED_FORMATS
    st.update(ctx=ctx, wl=wl, cam=cam, planes=planes, formats=formats, fmt=fmt, hist=hist, flags=flags, w=w, h=h)
    if case["kind"] == "host":
        torch.cuda.synchronize(dev)
        st["planes"] = [p.cpu().pin_memory() for p in planes]
        st["out_8"] = torch.empty((h, w, 4), dtype=torch.uint8, pin_memory=True)
        return
    st["out_f"] = torch.empty((h, w, 4), dtype=torch.float32, device=dev) if "f" in case["out"] else None
    st["out_8"] = torch.empty((h, w, 4), dtype=torch.uint8, device=dev) if "8" in case["out"] else None
    st["shown"] = torch.empty((h, w, 4), dtype=torch.uint8, device=dev) if case["post"] else None


def _camera(st):
    """The frame's RTCameraData: the frame counter seeds the RNG."""
    st["frame"] += 1
    cam = st["cam"].copy()
    cam[32:36] = float(st["frame"])
    return cam


def _run_frame(st):
    c, cam = st["case"], _camera(st)
    flags = st["flags"] | (0 if c["sync"] else L.HY_FLAG_NO_STATUS_SYNC)
    cfg = pass_config(c["spp"], c["bounces"], c["rng"], 0 if c["reset"] else st["frame"], flags)
    rays = st["ctx"].forward(st["planes"], cam, cfg, st["hist"], st["fmt"], out_f=st["out_f"], out_8=st["out_8"],
                             formats=st["formats"], stats=c["sync"])
    out = dict(history=st["hist"], color=st["out_f"], image=st["out_8"])
    if c["post"]:
        out["shown"] = st["ctx"].post(st["out_8"] if st["out_8"] is not None else st["out_f"], st["shown"])
    if c["sync"]:
        out["rays"] = [rays["shadow_rays"], rays["reflection_rays"], rays["hit_shadow_rays"]]
    return out


def _run_host(st):
    c, cam = st["case"], _camera(st)
    cfg = pass_config(c["spp"], c["bounces"], c["rng"], st["frame"], st["flags"])
    st["ctx"].forward_host(st["planes"], cam, cfg, st["hist"], st["fmt"], out_8=st["out_8"], formats=st["formats"],
                           stats=False)
    return dict(history=st["hist"], image=st["out_8"])


def _batch_plan(case, seed):
    """The views: sizes, samples and lights of the mixed batch's ranges (each view within a
    budget of samples), which are the case's own; cameras on a ring, from the seed."""
    rng = np.random.default_rng([case["views"], case["scenes"], case["tris_hi"]])
    cams = np.random.default_rng([int(seed), 7])
    views = []
    for _ in range(case["views"]):
        w, h = scenes.BATCH_RESOLUTIONS[int(rng.integers(len(scenes.BATCH_RESOLUTIONS)))]
        spp = int(scenes.BATCH_SPP[int(rng.integers(len(scenes.BATCH_SPP)))])
        nl = int(rng.integers(1, 9))
        while w * h * spp * nl > 4.0e7 and spp > 1:
            spp //= 4
        ang = cams.uniform(0, 2 * np.pi)
        views.append(dict(scene=int(rng.integers(case["scenes"])), w=w, h=h, spp=max(1, spp), lights=nl,
                          camera=Camera((55.0 * np.sin(ang), float(cams.uniform(12, 24)), 55.0 * np.cos(ang)),
                                        (0.0, 0.0, 0.0), 60.0)))
    return views


def _prepare_batch(case, seed, st, dev):
    rng = np.random.default_rng(seed)
    n = np.exp(rng.uniform(np.log(case["tris_lo"]), np.log(case["tris_hi"]), case["scenes"])).astype(int)
    ctxs = [_context(st["stream"], scenes.batch_scene(rng, int(k))) for k in n]
    views = _batch_plan(case, seed)
    for v in views:
        ctx = ctxs[v["scene"]]
        v["cam"] = v["camera"].rt_camera(v["w"], v["h"], 0.0)
        v["planes"] = ctx.gbuffer(v["cam"], v["w"], v["h"])
        v["hist"] = torch.zeros((v["lights"], v["h"], v["w"]), dtype=torch.uint8, device=dev)
        v["out_8"] = torch.empty((v["h"], v["w"], 4), dtype=torch.uint8, device=dev)
        ctx.forward(v["planes"], v["cam"], pass_config(1, 1, 1, 0), v["hist"], out_8=v["out_8"])
    st.update(ctxs=ctxs, views=views)


def _run_batch(st):
    st["frame"] += 1
    f, views = st["frame"], []
    for v in st["views"]:
        cam = v["cam"].copy()
        cam[32:36] = float(f)
        views.append(dict(scene=v["scene"], planes=v["planes"], camera=cam,
                          config=pass_config(v["spp"], 1, L.HY_RNG_DECORRELATED, f, L.HY_FLAG_NO_STATUS_SYNC),
                          hist=v["hist"], out_8=v["out_8"]))
    st["ctxs"][0].batch_forward(st["ctxs"], views, sync=False)
    return [(v["hist"], v["out_8"]) for v in st["views"]]


def _prepare_pathtrace(case, seed, st, dev):
    wl = _workload(case, seed)
    st.update(ctx=_context(st["stream"], wl.scene), cam=wl.camera(0.0), w=wl.width, h=wl.height,
              image=torch.zeros((wl.height, wl.width, 4), dtype=torch.uint8, device=dev))


def _run_pathtrace(st):
    c, cam = st["case"], _camera(st)
    cfg = pass_config(c["spp"], c["bounces"], c["rng"], 0, L.HY_FLAG_NO_STATUS_SYNC)
    image, _ = st["ctx"].pathtrace(cam, st["w"], st["h"], cfg, st["image"], stats=False)
    return image


def _prepare_fit(case, seed, st, dev):
    wl = _workload(case, seed)
    r = diffrender.DiffRenderer(wl.scene, wl.camera(0.0), wl.width, wl.height, spp=case["spp"],
                                max_bounces=case["bounces"])
    rng = np.random.default_rng([int(seed), 3])
    mp, lp = r.params0
    target, _ = r.render(np.clip(mp + rng.normal(0, 0.05, mp.shape), 0, 1).astype(np.float32),
                         (lp + rng.normal(0, 0.05, lp.shape)).astype(np.float32))
    st.update(r=r, mp=mp, lp=lp, target=target)


def _run_fit(st):
    r = st["r"]
    img, saved = r.render(st["mp"], st["lp"])
    grad = 2.0 * (img - st["target"])
    grad[..., 3] = 0.0
    gm, gl, _ = r.backward(saved, grad)
    return dict(image=img, materials=gm, lights=gl)


def _prepare_build(case, seed, st, dev):
    wl = _workload(case, seed)
    ctx = HybridContext(0, stream=st["stream"].cuda_stream)
    ctx.set_scene(wl.scene)
    if case["lbvh"]:
        ctx.set_build_mode(L.HY_BUILD_LBVH)
    st.update(ctx=ctx, wl=wl, rays=_rays(case, seed, dev))


def _hits(hits):
    """A query's results as a program reads them: distance, triangle id, barycentrics."""
    return dict(t=hits[:, 0], id=hits.view(torch.int32)[:, 1], b=hits[:, 2:4])


def _run_build(st):
    b = st["ctx"].build_bvh(instanced=st["case"]["instanced"])
    hits, _ = st["ctx"].trace(st["rays"], any_hit=False)
    return dict(nodes=b["num_bvh8_nodes"], depth=b["depth"], **_hits(hits))


def _prepare_refit(case, seed, st, dev):
    wl = _workload(case, seed)
    xf = wl.scene.pack()[3]
    st.update(ctx=_context(st["stream"], wl.scene, instanced=case["instanced"]), wl=wl, cam=wl.camera(0.0),
              xf=[_moved(xf, seed, k) for k in range(3)])


def _run_refit(st):
    xf = st["xf"][st["frame"] % len(st["xf"])]
    st["frame"] += 1
    st["ctx"].refit_bvh(xf)
    return st["ctx"].gbuffer(st["cam"], st["case"]["width"], st["case"]["height"])


def _prepare_trace(case, seed, st, dev):
    wl = _workload(case, seed)
    st.update(ctx=_context(st["stream"], wl.scene), wl=wl, rays=_rays(case, seed, dev))


def _run_trace(st):
    hits, _ = st["ctx"].trace(st["rays"], any_hit=st["case"]["any_hit"])
    if st["case"]["any_hit"]:  # which triangle stops an any-hit ray is not defined, whether one does is
        return dict(hit=hits.view(torch.int32)[:, 1] != -1)
    return _hits(hits)


def run(state):
    with torch.cuda.stream(state["stream"]):
        return globals()["_run_" + state["kind"]](state)


# ---- work ----------------------------------------------------------------------------------
def _tris(case):
    if case["kind"] == "fit":
        return 64 * 1280 + 2
    sc = case.get("scene", "hd")
    if sc == "hd":
        return 2 * (case["terrain"] - 1) ** 2 + case["spheres"] * 20 * 4 ** case["subdiv"]
    if sc == "large":
        return 2 * (case["terrain"] - 1) ** 2 + case["instances"] * 2024
    return 2 + 16 * 320


def _ray_flops(tris):
    """One ray: a node of 8 boxes per level of an 8-wide tree (8 x 12 operations), one triangle (50)."""
    return 96 * max(1.0, math.log(max(tris, 8), 8)) + 50


def work(case):
    k = case["kind"]
    if k == "batch":
        by = fl = 0.0
        tris = math.sqrt(case["tris_lo"] * case["tris_hi"])
        for v in _batch_plan(case, 0):
            px = v["w"] * v["h"]
            by += px * (88 + 4 + 2 * v["lights"])
            fl += px * 0.7 * v["lights"] * v["spp"] * _ray_flops(tris)
        return {"bytes": by + case["scenes"] * tris * 56, "flops": fl}
    tris = _tris(case)
    scene_bytes = 56.0 * tris  # packed triangles (48 B) and about 8 B of nodes each
    if k == "trace":
        return {"bytes": case["rays"] * 48 + scene_bytes, "flops": case["rays"] * _ray_flops(tris)}
    if k == "build":
        # vertices and indices in, nodes and packed triangles out; a sort-like n log n of box work
        return {"bytes": tris * (36 + 12) + scene_bytes + case["rays"] * 48,
                "flops": tris * math.log2(tris) * 30 + case["rays"] * _ray_flops(tris)}
    px = case["width"] * case["height"]
    if k == "refit":
        return {"bytes": tris * (36 + 12) + scene_bytes + px * 88, "flops": tris * 100 + px * _ray_flops(tris)}
    if k == "fit":
        # G-buffer and shadow images written and read, the image, the loss gradient
        return {"bytes": px * (2 * 88 + 2 * 4 * 8 + 16 * 3) + scene_bytes,
                "flops": px * (1 + 0.7 * 8 * case["spp"]) * _ray_flops(tris)}
    spp = case["spp"] if case["rng"] else 1
    shadow = px * 0.7 * case["lights"] * spp
    if k == "pathtrace":
        return {"bytes": px * 8 + scene_bytes, "flops": (px + shadow) * _ray_flops(tris)}
    texel = 36 if case["packed"] else 88
    hist = (4 if case.get("f32") else 1) * case["lights"]
    written = case.get("out", "8")
    out = (16 if "f" in written else 0) + (4 if "8" in written else 0) + (8 if case.get("post") else 0)
    return {"bytes": px * (texel + 2 * hist + out) + scene_bytes, "flops": shadow * _ray_flops(tris)}


# ---- exact -----------------------------------------------------------------------------------
MOST_PAIRS = 4.0e10  # ray-triangle pairs a plain 64-bit search takes within a few seconds


def _world(scene, xf=None):
    """World-space triangles (n, 3, 3) and what their hits need, in 64 bits."""
    verts, idx, prims, xf0, mats, _ = scene.pack()
    xf = xf0 if xf is None else xf
    pos, nrm, mat = [], [], []
    for first, count, vofs, material, tf, _ in prims:
        vi = idx[first:first + count].astype(np.int64) + int(vofs)
        m = xf[tf].astype(np.float64).reshape(4, 4).T
        p = verts[vi, 0:3].astype(np.float64) @ m[:3, :3].T + m[:3, 3]
        nm = np.linalg.inv(m).T[:3, :3]
        pos.append(p.reshape(-1, 3, 3))
        nrm.append((verts[vi, 3:6].astype(np.float64) @ nm.T).reshape(-1, 3, 3))
        mat.append(np.full(count // 3, material, np.int64))
    return np.concatenate(pos), np.concatenate(nrm), np.concatenate(mat), mats


def _closest(tri, org, dirs, tmin, tmax):
    """Closest hit of each ray by trying every triangle (Moeller-Trumbore): t, triangle or -1, b1, b2."""
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = torch.linalg.cross(e1, e2)
    out = []
    step = max(1, int(2.0e7 // len(tri)))
    for i in range(0, len(org), step):
        o, d = org[i:i + step], dirs[i:i + step]
        # t = (a - o).n / d.n; barycentrics as products of separate ray and triangle terms
        dn = d @ n.T
        m = torch.linalg.cross(o, d)                                       # Pluecker moment of the ray
        t = ((a * n).sum(1)[None] - o @ n.T) / dn
        u = ((d @ torch.linalg.cross(e2, a).T) - m @ e2.T) / dn
        v = (m @ e1.T - d @ torch.linalg.cross(e1, a).T) / dn
        ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t >= tmin) & (t <= tmax)
        t = torch.where(ok, t, torch.inf)
        best, k = t.min(1)
        hit = torch.isfinite(best)
        pick = lambda x: x.gather(1, k[:, None])[:, 0]  # noqa: E731
        zero = torch.zeros_like(best)
        out.append((torch.where(hit, best, zero), torch.where(hit, k, -1), torch.where(hit, pick(u), zero),
                    torch.where(hit, pick(v), zero)))
    return [torch.cat(x) for x in zip(*out)]


def exact(case, seed):
    k = case["kind"]
    if k not in ("trace", "build", "refit") or case.get("any_hit"):
        # images of a whole frame: a texel's shadow rays, and so its value, turn on single roundings
        return None
    tris = _tris(case)
    dev = torch.device("cuda", 0)
    if k == "refit":
        if tris * case["width"] * case["height"] > MOST_PAIRS:
            return None
        return _exact_gbuffer(case, int(seed), dev)
    if tris * case["rays"] > MOST_PAIRS:
        return None
    tri = torch.from_numpy(_world(_workload(case, int(seed)).scene)[0]).to(dev)
    r = _rays(case, seed, dev).double()
    t, _, b1, b2 = _closest(tri, r[:, 0:3], r[:, 4:7], 1e-3, 1000.0)
    out = dict(t=t, id=None, b=torch.stack([b1, b2], 1))
    return dict(nodes=None, depth=None, **out) if k == "build" else out


def _exact_gbuffer(case, seed, dev):
    """Planes of the primary-ray G-buffer after the first update of a refit case."""
    wl = _workload(case, seed)
    w, h = wl.width, wl.height
    xf = _moved(wl.scene.pack()[3], seed, 0)
    tri, nrm, mat, mats = (torch.from_numpy(np.asarray(x)).to(dev) for x in _world(wl.scene, xf))
    cam = torch.from_numpy(wl.camera(0.0)).to(dev).double()
    iv, ip = cam[0:16].reshape(4, 4).T, cam[16:32].reshape(4, 4).T
    y, x = torch.meshgrid(torch.arange(h, device=dev, dtype=torch.float64),
                          torch.arange(w, device=dev, dtype=torch.float64), indexing="ij")
    x, y = x.reshape(-1), y.reshape(-1)
    ndc = torch.stack([(x + 0.5) / w * 2 - 1, (y + 0.5) / h * 2 - 1, torch.ones_like(x), torch.ones_like(x)], 1)
    tgt = (ndc @ ip.T)[:, :3]
    d = (tgt / tgt.norm(dim=1, keepdim=True)) @ iv[:3, :3].T
    o = iv[:3, 3][None] + d * 1e-2
    t, k, b1, b2 = _closest(tri, o, d, 1e-3, 10000.0)
    hit = (k >= 0).double()[:, None]
    n = (nrm[k] * torch.stack([1 - b1 - b2, b1, b2], 1)[..., None]).sum(1)
    n = n / n.norm(dim=1, keepdim=True)
    m = mats.double()[mat[k]]
    one = torch.ones_like(t)[:, None]
    planes = [torch.cat([o + d * t[:, None], m[:, 11:12]], 1), torch.cat([n * 0.5 + 0.5, one], 1),
              torch.cat([m[:, 0:3], one], 1), torch.full((w * h, 2), 0.5, device=dev, dtype=torch.float64),
              torch.cat([0 * one, m[:, 10:11], m[:, 9:10], one], 1), torch.cat([0 * one, 0 * one, 0 * one, one], 1)]
    return [(p * hit).reshape(h, w, -1) for p in planes]
