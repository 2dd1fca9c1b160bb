"""Boxes and slot budgets climb from blocks of 256 leaves: builds and refits around the
block edges equal the oracle's array for array, in both builds, for random
triangles and for coincident and exponentially spaced ones (deep trees)."""
import numpy as np
import pytest

import pyoracle as po
from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300.scene import Material

pytestmark = pytest.mark.gpu


def _arrays(n, kind):
    rng = np.random.default_rng(n)
    cen = rng.uniform(-1, 1, (n, 3))
    if kind == "same":
        cen[n // 3:] = cen[0]
    elif kind == "line":
        cen[:, 0] = 2.0 ** np.linspace(-60, 20, n)
        cen[:, 1:] = 0
    v = np.zeros((3 * n, 11), np.float32)
    v[:, 0:3] = np.repeat(cen, 3, 0) + rng.uniform(-0.05, 0.05, (3 * n, 3))
    v[:, 4] = 1
    first = n // 3 + 1 if n > 1 else n  # two instances of their own transforms, the second's indices reversed
    idx = np.arange(3 * n, dtype=np.uint32)
    idx[3 * first:] = np.arange(3 * (n - first), dtype=np.uint32)[::-1]
    prims = [[0, 3 * first, 0, 0, 0, 0]]
    if n > first:
        prims.append([3 * first, 3 * (n - first), 3 * first, 0, 1, 1])
    xf = np.tile(np.eye(4, dtype=np.float32).reshape(1, 16), (2, 1))
    return v, idx, np.array(prims, np.uint32), xf, Material().to_shader(0)[None], np.zeros((0, 12), np.float32)


@pytest.mark.parametrize("mode", [L.HY_BUILD_SAH, L.HY_BUILD_LBVH])
@pytest.mark.parametrize("kind", ["random", "same", "line"])
@pytest.mark.parametrize("n", [1, 2, 3, 255, 256, 257, 511, 512, 513, 1025, 70000])
def test_build_and_refit_equal_oracle(gpu_lib, oracle_lib, n, kind, mode):
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    arrays = _arrays(n, kind)
    xf = arrays[3]
    ctx, o = HybridContext(0), po.OracleScene()
    try:
        ctx.set_scene_arrays(*arrays)
        o.set_scene_arrays(*arrays)
        ctx.set_build_mode(mode)
        o.set_build_mode(mode)
        gi, oi = ctx.build_bvh(), o.build_bvh()
        assert gi["num_bvh8_nodes"] == oi["num_bvh8_nodes"]
        moved = xf.copy()
        moved[0, 12:15] = 0.3, -0.2, 0.1
        moved[1, 0:12] = np.float32([0.8, 0.1, 0, 0, 0.05, 1.3, -0.2, 0, 0, 0.4, 0.9, 0])
        for step in (None, moved, xf):
            if step is not None:
                ctx.refit_bvh(step)
                o.refit_bvh(step)
            g, r = ctx.download_bvh(gi["num_bvh8_nodes"]), o.download_bvh(gi["num_bvh8_nodes"])
            for name, a, b in zip(["morton", "order", "bvh2", "bvh8", "tris"], g, r):
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), name
    finally:
        ctx.close()
