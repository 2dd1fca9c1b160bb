"""One ray per pixel and light (REFERENCE RNG, or one sample): each lane walks its own
pixel's lights and prepares the next ray while it walks.  The images must be
those of one lane per pixel, over scenes large enough that rays of one warp
differ widely in length, for frames with partial tiles and light counts around
the run-ahead limit; histories and batches alike."""
import numpy as np
import pytest

from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300 import scenes
from vulkanhybridraytracer_gb300.scene import Light

pytestmark = pytest.mark.gpu


def _scene(n_lights):
    """Terrain and spheres (66k triangles) under n_lights lights, some directional, near or low."""
    rng = np.random.default_rng(n_lights)
    wl = scenes.hd(3, 203, 117, n_spheres=12, sphere_subdiv=4, terrain_n=48)
    wl.scene.lights = [Light(scenes.DIRECTIONAL_LIGHT, (1, 1, 1), (0.2, 1.0, 0.1), 1.0, 500.0, 0.1) if i % 11 == 4 else
                       Light(scenes.POINT_LIGHT, (1, 1, 1), (float(rng.uniform(-30, 30)), float(rng.uniform(-1, 14)),
                                                             float(rng.uniform(-30, 30))), 30.0,
                             float(rng.choice([20.0, 500.0])), 0.5) for i in range(n_lights)]
    return wl


@pytest.mark.parametrize("instanced", [False, True])
@pytest.mark.parametrize("rng_mode,spp", [(L.HY_RNG_REFERENCE, 5), (L.HY_RNG_DECORRELATED, 1)])
@pytest.mark.parametrize("n_lights", [1, 2, 9, 10, 33])
def test_one_ray_streams_equal_per_pixel_walk(gpu_lib, n_lights, rng_mode, spp, instanced):
    import torch
    from vulkanhybridraytracer_gb300.hybrid import HybridContext, pass_config
    wl = _scene(n_lights)
    w, h = wl.width, wl.height
    ctx = HybridContext(0)
    try:
        ctx.set_scene(wl.scene)
        ctx.build_bvh(instanced=instanced)
        cam = wl.camera(2.0)
        planes = ctx.gbuffer(cam, w, h)
        h0 = torch.randint(0, 256, (n_lights, h, w), dtype=torch.uint8, generator=torch.Generator().manual_seed(1))
        outs = []
        for flags, visits in ((L.HY_FLAG_PIXEL_PARALLEL, 0), (0, 0), (0, 1), (0, 16)):
            raw = torch.zeros((n_lights, h, w), dtype=torch.uint8, device="cuda")
            hist = h0.cuda()
            torch.cuda.synchronize()
            cfg = pass_config(spp, 1, rng_mode, 2, flags, visits_per_round=visits)
            st = ctx.shadow_pass(planes, cam, cfg, raw)
            ctx.forward(planes, cam, cfg, hist)
            outs.append((raw, hist, st["shadow_rays"]))
        for raw, hist, rays in outs[1:]:
            assert torch.equal(raw, outs[0][0]) and torch.equal(hist, outs[0][1]) and rays == outs[0][2] > 0
        assert 0.02 < float((outs[0][0] > 0).float().mean()) < 0.98
        # the same frame as a batch of views
        hists = [h0.cuda(), h0.cuda()]
        torch.cuda.synchronize()
        ctx.batch_forward([ctx], [dict(scene=0, planes=planes, camera=cam, config=pass_config(spp, 1, rng_mode, 2), hist=x)
                                  for x in hists])
        assert torch.equal(hists[0], outs[0][1]) and torch.equal(hists[1], outs[0][1])
    finally:
        ctx.close()


@pytest.mark.parametrize("w,h", [(1, 1), (64, 40), (1100, 700)])
@pytest.mark.parametrize("n_lights,spp", [(2, 1), (3, 4), (9, 3)])
def test_light_parts_equal_whole_tiles(gpu_lib, w, h, n_lights, spp):
    """The last tiles of a launch are handed out in parts of a tile's lights: frames that are
    all parts and frames that start with whole tiles write the same images as one lane
    per pixel (the RNG of a part's first light follows the lights traced before it)."""
    import torch
    from vulkanhybridraytracer_gb300.hybrid import HybridContext, pass_config
    wl = _scene(n_lights)
    ctx = HybridContext(0)
    try:
        ctx.set_scene(wl.scene)
        ctx.build_bvh()
        cam = wl.scene.camera.rt_camera(w, h, 5.0)
        planes = ctx.gbuffer(cam, w, h)
        outs = []
        for flags, chunk in ((L.HY_FLAG_PIXEL_PARALLEL, 0), (0, 0), (0, 5)):
            raw = torch.zeros((n_lights, h, w), dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            st = ctx.shadow_pass(planes, cam, pass_config(spp, 1, L.HY_RNG_DECORRELATED, 5, flags, queue_chunk=chunk), raw)
            outs.append((raw, st["shadow_rays"]))
        for raw, rays in outs[1:]:
            assert torch.equal(raw, outs[0][0]) and rays == outs[0][1]
    finally:
        ctx.close()
