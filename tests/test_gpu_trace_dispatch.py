"""Ray queries around the sizes where the kernel changes (rays resident at once at 5 and 8
blocks per SM, structures of few and many records): hits equal the oracle's, with and
without counters."""
import numpy as np
import pytest

import pyoracle as po
from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("few", [True, False])
@pytest.mark.parametrize("instanced", [False, True])
def test_hits_around_the_lines(gpu_lib, oracle_lib, instanced, few):
    import torch
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    wl = scenes.hd(5, 64, 64, n_spheres=9, sphere_subdiv=3, terrain_n=40 if few else 300)
    ctx, orc = HybridContext(0), po.OracleScene()
    try:
        ctx.set_scene(wl.scene)
        orc.set_scene(wl.scene)
        ctx.build_bvh(instanced=instanced)
        orc.build_bvh_instanced() if instanced else orc.build_bvh()
        assert (ctx.bvh_layout()["num_records"] < 100_000) == few
        wave = 128 * torch.cuda.get_device_properties(0).multi_processor_count
        n = 8 * wave + 33
        rng = np.random.default_rng(4)
        rays = np.zeros((n, 8), np.float32)
        rays[:, 0:3], rays[:, 4:7] = rng.uniform([-40, 0, -40], [40, 10, 40], (n, 3)), rng.normal(size=(n, 3))
        rays[:, 3], rays[:, 7] = 1e-3, 1000.0
        dev = torch.from_numpy(rays).cuda()
        for any_hit in (False, True):
            want, counts = orc.trace(rays, any_hit)
            want = want.view(np.uint32)
            for m in (5 * wave, 5 * wave + 1, 8 * wave, 8 * wave + 1, n):
                got, st = ctx.trace(dev[:m], any_hit, count=True)
                assert np.array_equal(got.cpu().numpy().view(np.uint32), want[:m])
                assert st["nodes_visited"] == int(counts[:m, 0].sum()) and st["tris_tested"] == int(counts[:m, 1].sum())
                plain = ctx.trace(dev[:m], any_hit)[0].cpu().numpy().view(np.uint32)
                if any_hit:
                    assert np.array_equal(plain[:, 1] != L.HY_NO_HIT, want[:m, 1] != L.HY_NO_HIT)
                else:
                    assert np.array_equal(plain, want[:m])
    finally:
        ctx.close()
