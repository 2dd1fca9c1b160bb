"""The automatic any-hit order on a one-level structure beyond L2: the default shadow
schedule walks far first while ray queries and counted passes go near first; the
images and histories are those of both set orders, counted or not."""
import pytest

from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_auto_order_beyond_l2_equals_both_orders(gpu_lib):
    import torch
    from vulkanhybridraytracer_gb300.hybrid import HybridContext, pass_config
    wl = scenes.hd(5, 203, 117, n_spheres=6, sphere_subdiv=4, terrain_n=1400)  # 3.9M triangles
    w, h = wl.width, wl.height
    ctx = HybridContext(0)
    try:
        ctx.set_scene(wl.scene)
        ctx.build_bvh()
        assert ctx.anyhit_order() == L.HY_ANYHIT_NEAR_FIRST
        cam = wl.camera(1.0)
        planes = ctx.gbuffer(cam, w, h)
        for rng_mode, spp in ((L.HY_RNG_REFERENCE, 1), (L.HY_RNG_DECORRELATED, 5)):
            outs = []
            for order in (L.HY_ANYHIT_AUTO, L.HY_ANYHIT_FAR_FIRST, L.HY_ANYHIT_NEAR_FIRST):
                ctx.set_anyhit_order(order)
                for flags in (0, L.HY_FLAG_COUNT_TRAVERSAL):
                    cfg = pass_config(spp, 1, rng_mode, 0, flags)
                    raw = torch.zeros((4, h, w), dtype=torch.uint8, device="cuda")
                    hist = torch.full((4, h, w), 100, dtype=torch.uint8, device="cuda")
                    torch.cuda.synchronize()
                    st = ctx.shadow_pass(planes, cam, cfg, raw)
                    ctx.forward(planes, cam, cfg, hist)
                    outs.append((raw, hist, st["nodes_visited"], st["shadow_rays"]))
            for raw, hist, _, rays in outs[1:]:
                assert torch.equal(raw, outs[0][0]) and torch.equal(hist, outs[0][1]) and rays == outs[0][3] > 0
            assert outs[1][2] == outs[5][2] > 0  # counted under AUTO: near first
            assert 0.02 < float((outs[0][0] > 0).float().mean()) < 0.98
    finally:
        ctx.close()
