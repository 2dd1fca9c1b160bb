"""Closest-hit queries without counters run as a queue of rays over persistent warps
that test a round's triangles together: hits (distance, id, barycentrics) equal the
plain walk's (the counting kernel's) bit for bit, for any number of rays and for
buffers that are only 4-byte aligned, and a limit that runs out is reported for
exactly the rays the plain walk reports."""
import numpy as np
import pytest

from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[False, True], ids=["flat", "instanced"])
def ctx(request, gpu_lib):
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    c = HybridContext(0)
    c.set_scene(scenes.hd(5, 64, 64, n_spheres=9, sphere_subdiv=4, terrain_n=40).scene)
    c.build_bvh(instanced=request.param)
    yield c
    c.close()


def _rays(n, offset=0):
    import torch
    rng = np.random.default_rng(n)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform([-40, 0, -40], [40, 10, 40], (n, 3))
    r[:, 4:7] = rng.normal(size=(n, 3))
    r[::5, 5] = 0.0  # along planes of the boxes
    r[:, 3], r[:, 7] = 1e-3, 1000.0
    flat = torch.zeros(n * 8 + offset, device="cuda")
    t = flat[offset:].view(n, 8)
    t.copy_(torch.from_numpy(r))
    torch.cuda.synchronize()
    return t


@pytest.mark.parametrize("n,offset", [(1, 0), (31, 0), (33, 0), (4097, 0), (300_001, 0), (5000, 1)])
def test_queue_hits_equal_plain_walk(ctx, n, offset):
    rays = _rays(n, offset)
    plain, _ = ctx.trace(rays, False, count=True)
    queued, _ = ctx.trace(rays, False)
    a, b = plain.cpu().numpy().view(np.uint32), queued.cpu().numpy().view(np.uint32)
    assert np.array_equal(a, b)
    assert n < 100 or 0.05 < (a[:, 1] != L.HY_NO_HIT).mean() < 0.95


def test_queue_limits_equal_plain_walk(ctx):
    rays = _rays(3000)

    def code(limits, count):
        assert ctx.lib.hy_debug_set_traversal_limits(ctx.h, *limits) == L.HY_OK
        try:
            ctx.trace(rays, False, count=count)
        except L.HyError as e:
            return e.code
        return L.HY_OK

    try:
        for limit, hi, err in ((lambda v: (v, 0), 4096, L.HY_ERR_TIMEOUT), (lambda v: (0, v), 64, L.HY_ERR_STACK_OVERFLOW)):
            lo = 1
            while lo < hi:
                mid = (lo + hi) // 2
                lo, hi = (lo, mid) if code(limit(mid), True) == L.HY_OK else (mid + 1, hi)
            assert lo > 1 and code(limit(lo), False) == L.HY_OK and code(limit(lo - 1), False) == err
    finally:
        ctx.lib.hy_debug_set_traversal_limits(ctx.h, 0, 0)
