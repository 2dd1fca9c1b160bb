"""Ray queries that start on the planes of boxes and triangles, where a plane distance
is a zero of either sign: a floor, walls and boxes on whole coordinates, origins on their
faces, edges and corners and on the corners of the structure's nodes, directions in all
octants and along the axes with components +0 and -0, intervals that begin or end at
zero.  Hits and counts equal the oracle's, whose box test compares its distances."""
import numpy as np
import pytest

import pyoracle as po
from vulkanhybridraytracer_gb300 import _lib as L
from vulkanhybridraytracer_gb300.scene import Light, Material, Mesh, Object, Scene

pytestmark = pytest.mark.gpu

TMIN, TMAX = (0.0, -0.0, 1e-3, -1.0), (0.0, -0.0, 50.0)


def _mesh(pos, tri):
    v = np.zeros((len(pos), 11), np.float32)
    v[:, 0:3] = pos
    v[:, 4] = 1.0
    return Mesh(v, np.asarray(tri, np.uint32).reshape(-1))


def _sheet(n, axis):
    """n x n unit squares in the plane coordinate `axis` = 0"""
    g = np.arange(n + 1)
    a, b = (k for k in range(3) if k != axis)
    pos = np.zeros(((n + 1) ** 2, 3))
    pos[:, a], pos[:, b] = np.repeat(g, n + 1), np.tile(g, n + 1)
    c = (np.repeat(np.arange(n), n) * (n + 1) + np.tile(np.arange(n), n))[:, None]
    return _mesh(pos, np.concatenate([c + [0, 1, n + 2], c + [0, n + 2, n + 1]]))


def _box():
    pos = [(i & 1, i >> 1 & 1, i >> 2) for i in range(8)]
    faces = [(0, 1, 3, 2), (4, 5, 7, 6), (0, 1, 5, 4), (2, 3, 7, 6), (0, 2, 6, 4), (1, 3, 7, 5)]
    return _mesh(pos, [t for f in faces for t in ((f[0], f[1], f[2]), (f[0], f[2], f[3]))])


def _at(x, y, z):
    m = np.eye(4, dtype=np.float32)
    m[3, :3] = (x, y, z)  # [col][row]
    return m


def _scene():
    box = _box()
    ents = [Object(_sheet(12, axis), 0, _at(-6, 0, -6) if axis == 1 else _at(-6, -2, -6)) for axis in range(3)]
    rng = np.random.default_rng(11)
    ents += [Object(box, 0, _at(*p)) for p in rng.integers([-6, 0, -6], [6, 5, 6], (40, 3))]
    return Scene(entities=ents, lights=[Light(position=(0.0, 9.0, 0.0))], materials=[Material()])


def _rays(rng, corners, n=24000):
    org = rng.integers([-7, -2, -7], [8, 7, 8], (n, 3)).astype(np.float32)
    half = rng.random((n, 3)) < 0.3
    org[half] += rng.choice([0.25, 0.5], half.sum())
    org[::5] = corners[rng.integers(0, len(corners), len(org[::5]))]
    loose = rng.random((n, 3)) < 0.2
    org[loose] += rng.uniform(-3, 3, loose.sum()).astype(np.float32)
    d = rng.choice([-1.0, -0.5, -0.2, -0.0, 0.0, 0.2, 0.5, 1.0], (n, 3)).astype(np.float32)
    axis = rng.integers(0, 3, n)
    straight = rng.random(n) < 0.4
    d[straight] = np.copysign(np.float32(0.0), d[straight])
    d[np.arange(n), axis] = np.where(rng.random(n) < 0.5, -1.0, 1.0)
    rays = np.zeros((n, 8), np.float32)
    rays[:, 0:3], rays[:, 4:7] = org, d
    rays[:, 3], rays[:, 7] = rng.choice(TMIN, n), rng.choice(TMAX, n, p=(0.1, 0.1, 0.8))
    return rays


@pytest.mark.parametrize("instanced", [False, True])
def test_rays_from_planes(gpu_lib, oracle_lib, instanced):
    import torch
    from vulkanhybridraytracer_gb300.hybrid import HybridContext
    scene = _scene()
    ctx, orc = HybridContext(0), po.OracleScene()
    try:
        ctx.set_scene(scene)
        orc.set_scene(scene)
        ctx.build_bvh(instanced=instanced)
        if instanced:
            orc.build_bvh_instanced()
            nodes = orc.download_bvh_instanced()[1]
        else:
            nodes = orc.download_bvh(orc.build_bvh()["num_bvh8_nodes"])[3]
        rays = _rays(np.random.default_rng(3), nodes[:, 0:3].copy().view(np.float32))
        dev = torch.from_numpy(rays).cuda()
        for any_hit in (False, True):
            want, counts = orc.trace(rays, any_hit)
            found = want.view(np.uint32)[:, 1] != L.HY_NO_HIT
            assert 0.2 < found.mean() < 0.9 and (found & (want[:, 0] == 0.0)).sum() > 500
            got, st = ctx.trace(dev, any_hit, count=True)
            assert np.array_equal(got.cpu().numpy().view(np.uint32), want.view(np.uint32))
            assert st["nodes_visited"] == int(counts[:, 0].sum()) and st["tris_tested"] == int(counts[:, 1].sum())
            plain = ctx.trace(dev, any_hit)[0].cpu().numpy().view(np.uint32)  # the kernels without counters
            if any_hit:
                assert np.array_equal(plain[:, 1] != L.HY_NO_HIT, found)
            else:
                assert np.array_equal(plain, want.view(np.uint32))
    finally:
        ctx.close()
