"""Structures over coordinates near the largest float, where sums of box corners, areas and
child costs overflow to infinities and NaN: builds, refits and instanced builds equal the
oracle's array for array, in both builds."""
import numpy as np
import pytest

import pyoracle as po
from test_gpu_climb import _arrays
from vulkanhybridraytracer_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def _scaled(n, scale):
    v, idx, prims, xf, mats, lights = _arrays(n, "random")
    v[:, 0:3] = np.clip(v[:, 0:3].astype(np.float64) * scale, -3.4e38, 3.4e38).astype(np.float32)
    return v, idx, prims, xf, mats, lights


def _equal(got, want):
    return [a.shape == b.shape and np.array_equal(a.view(np.uint32), b.view(np.uint32)) for a, b in zip(got, want)]


@pytest.mark.parametrize("mode", [L.HY_BUILD_SAH, L.HY_BUILD_LBVH])
@pytest.mark.parametrize("scale", [1e19, 1.5e38, 3e38, 1.2e39])
@pytest.mark.parametrize("n", [9, 40, 300, 3000])
def test_build_and_refit_equal_oracle(gpu_lib, oracle_lib, n, scale, mode):
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    arrays = _scaled(n, scale)
    ctx, o = HybridContext(0), po.OracleScene()
    try:
        for s in (ctx, o):
            s.set_scene_arrays(*arrays)
            s.set_build_mode(mode)
        gi, oi = ctx.build_bvh(), o.build_bvh()
        assert gi["num_bvh8_nodes"] == oi["num_bvh8_nodes"]
        moved = arrays[3].copy()
        moved[1, 0:12] = np.float32([0.8, 0.1, 0, 0, 0.05, 1.3, -0.2, 0, 0, 0.4, 0.9, 0])
        for xf in (None, moved):
            if xf is not None:
                ctx.refit_bvh(xf)
                o.refit_bvh(xf)
            assert all(_equal(ctx.download_bvh(gi["num_bvh8_nodes"]), o.download_bvh(gi["num_bvh8_nodes"])))
    finally:
        ctx.close()


@pytest.mark.parametrize("mode", [L.HY_BUILD_SAH, L.HY_BUILD_LBVH])
@pytest.mark.parametrize("scale", [1.5e38, 3e38])
def test_instanced_build_equals_oracle(gpu_lib, oracle_lib, scale, mode):
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    arrays = _scaled(3000, scale)
    ctx, o = HybridContext(0), po.OracleScene()
    try:
        for s in (ctx, o):
            s.set_scene_arrays(*arrays)
            s.set_build_mode(mode)
        ctx.build_bvh(instanced=True)
        o.build_bvh_instanced()
        got, want = ctx.download_bvh_instanced(), o.download_bvh_instanced()
        assert got[0]["num_nodes"] == want[0]["num_nodes"] and all(_equal(got[1:], want[1:]))
    finally:
        ctx.close()
