"""The launch fields min_blocks and stack_depth select a compiled variant of the tile-stream
shadow kernel for passes with many samples per light and for passes with one ray per light
alike, and every variant gives the images of one lane per pixel."""
import ctypes as C

import pytest

from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300 import build, scenes

VARIANTS = [(5, 0), (6, 0), (7, 0), (8, 0), (8, 8)]  # min_blocks, stack_depth


@pytest.mark.parametrize("one", [False, True])
@pytest.mark.parametrize("count", [False, True])
@pytest.mark.parametrize("symbol", ["_ZN2hy17stream_kernel_rawEbibb", "_ZN2hy19stream_kernel_accumEbibb"])
def test_variants_are_distinct_kernels(symbol, count, one):
    """hy::stream_kernel_raw / _accum(count, min_blocks, short stack, one ray per light)"""
    build.build_cuda()
    f = getattr(C.CDLL(str(build.LIB)), symbol)
    f.restype, f.argtypes = C.c_void_p, [C.c_bool, C.c_int, C.c_bool, C.c_bool]
    kernels = [f(count, minb, depth == 8, one) for minb, depth in VARIANTS]
    assert all(kernels) and len(set(kernels)) == len(VARIANTS)


@pytest.mark.gpu
@pytest.mark.parametrize("rng_mode,spp", [(L.HY_RNG_REFERENCE, 4), (L.HY_RNG_DECORRELATED, 1)])
@pytest.mark.parametrize("w,h", [(37, 23), (320, 240)])
def test_one_ray_variants_equal_pixel_kernel(gpu_lib, rng_mode, spp, w, h):
    import torch
    from vulkanhybridraytracer_gb300.hybrid import HybridContext, pass_config
    wl = scenes.hd(2, w, h, n_spheres=9, sphere_subdiv=3, terrain_n=40)
    nl = len(wl.scene.lights)
    ctx = HybridContext(0)
    try:
        ctx.set_scene(wl.scene)
        ctx.build_bvh()
        cam = wl.camera(2.0)
        planes = ctx.gbuffer(cam, w, h)

        def images(flags, minb, depth):
            cfg = pass_config(spp, 1, rng_mode, 3, flags, min_blocks=minb, stack_depth=depth)
            raw = torch.zeros((nl, h, w), dtype=torch.uint8, device="cuda")
            hist = torch.full((nl, h, w), 90, dtype=torch.uint8, device="cuda")
            torch.cuda.synchronize()
            st = ctx.shadow_pass(planes, cam, cfg, raw)
            ctx.forward(planes, cam, cfg, hist)
            return raw, hist, st["shadow_rays"]

        want = images(L.HY_FLAG_PIXEL_PARALLEL, 0, 0)
        assert 0.02 < float((want[0] > 0).float().mean()) < 0.98 and want[2] > 0
        for minb, depth in VARIANTS:
            for flags in (0, L.HY_FLAG_COUNT_TRAVERSAL):
                got = images(flags, minb, depth)
                assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and got[2] == want[2]
    finally:
        ctx.close()
