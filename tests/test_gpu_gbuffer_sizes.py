"""Primary rays over two levels around the frame size where the kernel changes, and at
ragged sizes: the G-buffer equals the oracle's over the same structure."""
import numpy as np
import pytest

import pyoracle as po
from vulkanhybridraytracer_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 1), (17, 9), (33, 3), (333, 171), "line", "above"])
@pytest.mark.parametrize("instanced", [False, True])
def test_gbuffer_equals_oracle(gpu_lib, oracle_lib, instanced, size):
    import torch
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    line = 6 * 5 * 128 * torch.cuda.get_device_properties(0).multi_processor_count
    w, h = {"line": (line // 640, 640), "above": (line // 640 + 1, 641)}.get(size, size)
    wl = scenes.small(0, 64, 64)
    ctx, orc = HybridContext(0), po.OracleScene()
    try:
        ctx.set_scene(wl.scene)
        orc.set_scene(wl.scene)
        ctx.build_bvh(instanced=instanced)
        orc.build_bvh_instanced() if instanced else orc.build_bvh()
        cam = wl.scene.camera.rt_camera(w, h, 0.0)
        got, want = [p.cpu().numpy() for p in ctx.gbuffer(cam, w, h)], orc.gbuffer(cam, w, h)
        for i in (0, 2, 3, 4, 5):
            assert np.array_equal(got[i], want[i]), f"plane {i}"
        np.testing.assert_allclose(got[1], want[1], atol=2e-6)
    finally:
        ctx.close()
