"""Device memory of a build: the budgets (max_device_bytes) that builds once fitted in still
hold, in both builds, one and two levels."""
import numpy as np
import pytest

from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300.scene import Material

pytestmark = pytest.mark.gpu

# triangles, build, two levels, bytes
BUDGETS = [(200, L.HY_BUILD_SAH, False, 155520), (200, L.HY_BUILD_LBVH, True, 134936),
           (5000, L.HY_BUILD_SAH, True, 3663056), (5000, L.HY_BUILD_LBVH, False, 3311532),
           (100000, L.HY_BUILD_SAH, False, 73142900), (100000, L.HY_BUILD_LBVH, False, 66200764),
           (100000, L.HY_BUILD_LBVH, True, 66205736)]


@pytest.mark.parametrize("n,mode,instanced,budget", BUDGETS)
def test_build_fits(gpu_lib, n, mode, instanced, budget):
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    rng = np.random.default_rng(n)
    v = np.zeros((3 * n, 11), np.float32)
    v[:, 0:3] = np.repeat(rng.uniform(-1, 1, (n, 3)), 3, 0) + rng.uniform(-0.05, 0.05, (3 * n, 3))
    ctx = HybridContext(0, max_device_bytes=budget)
    try:
        ctx.set_scene_arrays(v, np.arange(3 * n, dtype=np.uint32), np.array([[0, 3 * n, 0, 0, 0, 0]], np.uint32),
                             np.eye(4, dtype=np.float32).reshape(1, 16), Material().to_shader(0)[None],
                             np.zeros((0, 12), np.float32))
        ctx.set_build_mode(mode)
        assert ctx.build_bvh(instanced=instanced)["num_tris"] == n
    finally:
        ctx.close()
