"""Ray queries with infinite, NaN, huge and subnormal components and with empty intervals:
hits and counts equal the oracle's, and an empty ray's walk is the root's visit and the step
that ends it, in the kernels with and without counters."""
import numpy as np
import pytest

import pyoracle as po
from test_gpu_trace_planes import _scene
from vulkanhybridraytracer_gb300 import _lib as L

pytestmark = pytest.mark.gpu

VALUES = np.float32([0, -0.0, np.inf, -np.inf, np.nan, 3e38, -3e38, 1e-40, -1e-40, 1e20, -1e20, 1, -1])


def _rays(rng, n=40000):
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3], rays[:, 4:7] = rng.uniform([-7, -2, -7], [8, 7, 8], (n, 3)), rng.normal(size=(n, 3))
    rays[:, 3], rays[:, 7] = 1e-3, 50.0
    for k in range(8):
        m = rng.random(n) < 0.12
        rays[m, k] = rng.choice(VALUES, m.sum())
    rays[::9, 3] = rays[::9, 7] + 1  # empty
    return rays


@pytest.fixture(params=[False, True], ids=["flat", "instanced"])
def traced(request, gpu_lib, oracle_lib):
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    scene = _scene()
    ctx, orc = HybridContext(0), po.OracleScene()
    try:
        ctx.set_scene(scene)
        orc.set_scene(scene)
        ctx.build_bvh(instanced=request.param)
        orc.build_bvh_instanced() if request.param else orc.build_bvh()
        yield ctx, orc
    finally:
        ctx.close()


@pytest.mark.parametrize("any_hit", [False, True])
def test_special_components_and_empty_intervals(traced, any_hit):
    import torch
    ctx, orc = traced
    rays = _rays(np.random.default_rng(8))
    dev = torch.from_numpy(rays).cuda()
    want, counts = orc.trace(rays, any_hit)
    found = want.view(np.uint32)[:, 1] != L.HY_NO_HIT
    assert 0.1 < found.mean() < 0.9
    got, st = ctx.trace(dev, any_hit, count=True)
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert st["nodes_visited"] == int(counts[:, 0].sum()) and st["tris_tested"] == int(counts[:, 1].sum())
    plain = ctx.trace(dev, any_hit)[0].cpu().numpy().view(np.uint32)  # the kernels without counters
    if any_hit:
        assert np.array_equal(plain[:, 1] != L.HY_NO_HIT, found)
    else:
        assert np.array_equal(plain, want.view(np.uint32))


def test_empty_intervals_under_limits(traced):
    import torch
    ctx = traced[0]
    rays = torch.from_numpy(_rays(np.random.default_rng(9))[::9].copy())
    keep = torch.isfinite(rays[:, 3]) & (rays[:, 3] > rays[:, 7] * 1.001 + 1e-3) & (rays[:, 7] > -1e30)
    rays = rays[keep].cuda()
    assert len(rays) > 1000
    try:
        for limit, code in ((1, L.HY_ERR_TIMEOUT), (2, L.HY_OK)):
            assert ctx.lib.hy_debug_set_traversal_limits(ctx.h, limit, 1) == L.HY_OK
            for any_hit in (False, True):
                for count in (False, True):
                    try:
                        hits, st = ctx.trace(rays, any_hit, count=count)
                        assert bool((hits.view(torch.int32)[:, 1] == -1).all())
                        assert not count or (st["nodes_visited"], st["tris_tested"]) == (len(rays), 0)
                        got = L.HY_OK
                    except L.HyError as e:
                        got = e.code
                    assert got == code
    finally:
        ctx.lib.hy_debug_set_traversal_limits(ctx.h, 0, 0)


def test_hits_at_a_negative_start(gpu_lib, oracle_lib):
    """Closest hits at exactly tmin < 0: from there on the interval is empty up to the box
    test's slack, and the nodes left make no more visits than the comparing walk's."""
    import torch
    from vulkanhybridraytracer_gb300 import scenes
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    n, rng = 400_000, np.random.default_rng(1)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = rng.uniform([-7, -2, -7], [8, 7, 8], (n, 3))
    axis, k = rng.integers(0, 3, n), np.arange(n)
    rays[k, axis] = rng.integers(-7, 8, n)
    rays[:, 4:7] = rng.uniform(-0.5, 0.5, (n, 3)) * (rng.random((n, 1)) < 0.7)
    rays[k, 4 + axis] = rng.choice([-1.0, 1.0], n)
    rays[:, 3], rays[:, 7] = -rng.integers(1, 6, n), 50
    wl = scenes.small(0, 64, 64)
    ctx, orc = HybridContext(0), po.OracleScene()
    try:
        ctx.set_scene(wl.scene)
        orc.set_scene(wl.scene)
        ctx.build_bvh()
        orc.build_bvh()
        want, counts = orc.trace(rays, False)
        assert ((want.view(np.uint32)[:, 1] != L.HY_NO_HIT) & (want[:, 0] == rays[:, 3])).sum() > 1000
        dev = torch.from_numpy(rays).cuda()
        got, st = ctx.trace(dev, False, count=True)
        assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))
        assert st["nodes_visited"] == int(counts[:, 0].sum()) and st["tris_tested"] == int(counts[:, 1].sum())
        assert np.array_equal(ctx.trace(dev, False)[0].cpu().numpy().view(np.uint32), want.view(np.uint32))
    finally:
        ctx.close()


@pytest.mark.parametrize("length", [3e38, 1e30, 2.0 ** 41, 2.0 ** 39, 2.0 ** -39, 2.0 ** -41, 1e-21, 1e-38])
@pytest.mark.parametrize("instanced", [False, True])
def test_direction_lengths(gpu_lib, oracle_lib, instanced, length):
    """Closest hits along directions so long or short that distances underflow or box and
    triangle distances part: the queries without counters give the plain walk's hits."""
    import torch
    from vulkanhybridraytracer_gb300 import scenes
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    n, rng = 200_000, np.random.default_rng(2)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3] = rng.uniform([-10, -1, -10], [10, 5, 10], (n, 3))
    d = rng.uniform(-1, 1, (n, 3))
    rays[:, 4:7] = d / np.abs(d).max(axis=1, keepdims=True) * length
    rays[::2, 4] = rng.uniform(-0.5, 0.5, len(rays[::2]))
    rays[:, 3], rays[:, 7] = rng.choice([0.0, -3e38, -np.inf], n), np.inf if length < 1e-35 else 1000.0 * max(1.0, 1.0 / length)
    ctx = HybridContext(0)
    try:
        ctx.set_scene(scenes.diff(3, 64, 64).scene)
        ctx.build_bvh(instanced=instanced)
        dev = torch.from_numpy(rays).cuda()
        plain, _ = ctx.trace(dev, False, count=True)
        queued, _ = ctx.trace(dev, False)
        assert torch.equal(plain.view(torch.int32), queued.view(torch.int32))
    finally:
        ctx.close()
