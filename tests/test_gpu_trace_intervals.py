"""Ray queries over every kind of ray interval: the node and triangle counts and
the hits of the GPU's box test equal the oracle's, bit for bit."""
import numpy as np
import pytest

import pyoracle as po
from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300 import scenes

pytestmark = pytest.mark.gpu

INTERVALS = {"usual": (1e-3, 1000.0), "from zero": (0.0, 50.0), "behind the origin": (-30.0, 30.0),
             "all behind": (-30.0, -1.0), "short": (2.0, 2.5), "a point": (3.0, 3.0), "empty": (5.0, 1.0),
             "empty by an ulp": (1.0, float(np.nextafter(np.float32(1.0), np.float32(0.0)))),
             "unbounded": (1e-3, np.inf), "both ways": (-np.inf, np.inf), "negative empty": (-1.0, -2.0)}


@pytest.mark.parametrize("instanced", [False, True])
@pytest.mark.parametrize("interval", list(INTERVALS))
def test_interval_counts_and_hits(gpu_lib, oracle_lib, interval, instanced):
    import torch
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    wl = scenes.small(0, 64, 64)
    ctx, orc = HybridContext(0), po.OracleScene()
    try:
        ctx.set_scene(wl.scene)
        orc.set_scene(wl.scene)
        ctx.build_bvh(instanced=instanced)
        orc.build_bvh_instanced() if instanced else orc.build_bvh()
        rng = np.random.default_rng(6)
        rays = np.zeros((6000, 8), np.float32)
        rays[:, 0:3] = rng.uniform([-8, -1, -8], [8, 4, 8], (6000, 3))
        d = rng.normal(size=(6000, 3))
        d[::7] = np.eye(3)[rng.integers(0, 3, len(d[::7]))] * rng.choice([-1, 1], (len(d[::7]), 1))  # along the axes
        rays[:, 4:7] = d
        rays[:, 3], rays[:, 7] = INTERVALS[interval]
        for any_hit in (False, True):
            hg, sg = ctx.trace(torch.from_numpy(rays).cuda(), any_hit, count=True)
            ho, co = orc.trace(rays, any_hit)
            assert np.array_equal(hg.cpu().numpy().view(np.uint32), ho.view(np.uint32))
            assert sg["nodes_visited"] == int(co[:, 0].sum()) and sg["tris_tested"] == int(co[:, 1].sum())
            hn, _ = ctx.trace(torch.from_numpy(rays).cuda(), any_hit)  # the kernel without counters
            if any_hit:
                got, want = (x[:, 1] != L.HY_NO_HIT for x in (hn.cpu().numpy().view(np.uint32), ho.view(np.uint32)))
                assert np.array_equal(got, want)
            else:
                assert np.array_equal(hn.cpu().numpy().view(np.uint32), ho.view(np.uint32))
    finally:
        ctx.close()
