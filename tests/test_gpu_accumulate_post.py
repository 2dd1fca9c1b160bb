"""The accumulation kernel's block edges (one block, partial blocks, several) for both
history formats, and the post resolve's table against its float path and the
rounding of every 8-bit value."""
import numpy as np
import pytest

import pyoracle as po
from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def pair(gpu_lib, oracle_lib):
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    c, o = HybridContext(0), po.OracleScene()
    wl = scenes.small(0, 32, 32)
    c.set_scene(wl.scene)
    c.build_bvh()
    o.set_scene(wl.scene)
    o.build_bvh()
    yield c, o
    c.close()


@pytest.mark.parametrize("w,h", [(1, 1), (32, 16), (33, 17), (31, 15), (64, 49), (97, 130)])
@pytest.mark.parametrize("fmt", [L.HY_ACCUM_U8, L.HY_ACCUM_F32])
@pytest.mark.parametrize("frame", [0, 5])
def test_accumulate_block_edges(pair, w, h, fmt, frame):
    import torch
    from vulkanhybridraytracer_gb300.hybrid import pass_config
    ctx, orc = pair
    rng = np.random.default_rng(w * 1000 + h)
    planes = [np.zeros((h, w, 4), np.float32) for _ in range(6)]
    planes[3] = (0.5 + rng.uniform(-0.2, 0.2, (h, w, 2))).astype(np.float32)
    raw = rng.integers(0, 256, (2, h, w)).astype(np.uint8)
    hist = rng.integers(0, 256, (2, h, w)).astype(np.uint8)
    if fmt == L.HY_ACCUM_F32:
        raw, hist = (raw / 255).astype(np.float32), (hist / 255).astype(np.float32)
    for flags in (0, L.HY_FLAG_FULL_BLUR_DISPATCH):
        got = torch.from_numpy(hist.copy()).cuda()
        p, r = [torch.from_numpy(x).cuda() for x in planes], torch.from_numpy(raw).cuda()
        torch.cuda.synchronize()
        ctx.accumulate_pass(p, pass_config(accum_frame=frame, flags=flags), r, got, fmt)
        want = hist.copy()
        orc.accumulate(planes, po.cfg_dict(accum_frame=frame, flags=flags), raw, want, fmt)
        assert np.array_equal(got.cpu().numpy(), want), flags


@pytest.mark.parametrize("n", [1, 2047, 2048, 2049, 10_000])
def test_post_table_equals_float_path(pair, n):
    import torch
    ctx, _ = pair
    img = torch.randint(0, 256, (1, n, 4), dtype=torch.uint8, generator=torch.Generator().manual_seed(n)).cuda()
    flt = (img.float() / 255.0)[..., [2, 1, 0, 3]].contiguous()
    torch.cuda.synchronize()
    a, b = ctx.post(img), ctx.post(flt)
    assert torch.equal(a, b) and torch.equal(a[..., 3], img[..., 3])
