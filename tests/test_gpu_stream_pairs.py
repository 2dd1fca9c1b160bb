"""The tile streams test a round's triangles together, as (ray, triangle) pairs
collected from all lanes of the warp: the images must be those of one lane per
pixel walking its rays alone, also where a visit reaches more triangles than
the warp's list holds, and a limit that runs out must be reported for exactly
the rays that the plain walk reports."""
import numpy as np
import pytest

from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300 import scenes
from vulkanhybridraytracer_gb300.scene import Mesh, Object

pytestmark = pytest.mark.gpu


def _torch():
    import torch
    return torch


def soup_workload(w, h, n=400):
    """The small scene under a soup of n large overlapping triangles with gaps: nodes whose
    boxes all overlap, so a visit reaches up to 8 leaves of 3 triangles on every lane."""
    rng = np.random.default_rng(12)
    wl = scenes.small(0, w, h)
    c = rng.uniform([-6, 2.0, -6], [6, 3.0, 6], (n, 1, 3))
    pos = (c + rng.uniform(-1.2, 1.2, (n, 3, 3)) * [1, 0.3, 1]).reshape(-1, 3)
    v = np.zeros((3 * n, 11), np.float32)
    v[:, 0:3] = pos
    v[:, 4] = 1.0
    v[:, 6:9] = 1.0
    wl.scene.entities.append(Object(Mesh(v, np.arange(3 * n, dtype=np.uint32)), 1))
    return wl


def make(wl, instanced):
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    ctx = HybridContext(0)
    ctx.set_scene(wl.scene)
    ctx.build_bvh(instanced=instanced)
    cam = wl.camera(3.0)
    return ctx, cam, ctx.gbuffer(cam, wl.width, wl.height)


def shadow(ctx, wl, cam, planes, spp, flags=0, visits=0):
    from vulkanhybridraytracer_gb300.hybrid import pass_config
    torch = _torch()
    out = torch.zeros((ctx.num_lights, wl.height, wl.width), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    st = ctx.shadow_pass(planes, cam, pass_config(spp, 1, L.HY_RNG_DECORRELATED, 3, flags, visits_per_round=visits), out)
    return out, st


@pytest.mark.parametrize("instanced", [False, True])
@pytest.mark.parametrize("spp,visits", [(1, 0), (16, 1), (16, 0), (16, 16), (37, 5)])
def test_pair_list_overflow_equals_plain_walk(gpu_lib, instanced, spp, visits):
    torch = _torch()
    wl = soup_workload(61, 37)
    ctx, cam, planes = make(wl, instanced)
    try:
        a, sa = shadow(ctx, wl, cam, planes, spp, visits=visits)
        b, sb = shadow(ctx, wl, cam, planes, spp, L.HY_FLAG_PIXEL_PARALLEL)
        assert torch.equal(a, b)
        assert sa["shadow_rays"] == sb["shadow_rays"] > 0 and sa["error_flags"] == 0
        assert 0 < int((a > 0).sum()) < a.numel()  # lit and occluded samples
    finally:
        ctx.close()


@pytest.mark.parametrize("instanced", [False, True])
def test_limits_reported_as_by_the_plain_walk(gpu_lib, instanced):
    """The smallest node-visit budget (and stack cap) under which one lane per pixel succeeds
    is enough for the tile streams, and one less is too little for both."""
    wl = soup_workload(40, 24)
    ctx, cam, planes = make(wl, instanced)
    lib = ctx.lib

    def code(limits, flags, visits=0):
        assert lib.hy_debug_set_traversal_limits(ctx.h, *limits) == L.HY_OK
        try:
            shadow(ctx, wl, cam, planes, 8, flags, visits)
        except L.HyError as e:
            return e.code
        return L.HY_OK

    try:
        for limit, lo, hi, err in ((lambda n: (n, 0), 1, 4096, L.HY_ERR_TIMEOUT),
                                   (lambda n: (0, n), 1, 64, L.HY_ERR_STACK_OVERFLOW)):
            while lo < hi:  # the plain walk's smallest sufficient limit
                mid = (lo + hi) // 2
                if code(limit(mid), L.HY_FLAG_PIXEL_PARALLEL) == L.HY_OK:
                    hi = mid
                else:
                    lo = mid + 1
            assert lo > 1
            for visits in (1, 0, 16):
                assert code(limit(lo), 0, visits) == L.HY_OK, (lo, visits)
                assert code(limit(lo - 1), 0, visits) == err, (lo, visits)
    finally:
        lib.hy_debug_set_traversal_limits(ctx.h, 0, 0)
        ctx.close()
