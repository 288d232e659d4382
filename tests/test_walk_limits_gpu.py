"""The walks' distance limit and tie rule where they can go wrong: coincident primitives (equal
distances), negative and zero distances (tmin below zero), and a tmax just above a hit."""
from __future__ import annotations

import numpy as np
import pytest

import ptb200 as pt
from oracle_bind import Oracle

pytestmark = pytest.mark.gpu


def stacked_scene(copies: int) -> pt.FlatScene:
    """Unit squares at z = -1, 0 and 1, each stored `copies` times (every hit is an exact tie), and two equal spheres."""
    tri = np.zeros(6 * copies, pt.TRIANGLE)
    for k in range(3 * copies):
        z = float(k % 3 - 1)
        tri[2 * k]["v0"], tri[2 * k]["v1"], tri[2 * k]["v2"] = (0, 0, z), (1, 0, z), (0, 1, z)
        tri[2 * k + 1]["v0"], tri[2 * k + 1]["v1"], tri[2 * k + 1]["v2"] = (1, 1, z), (0, 1, z), (1, 0, z)
    spheres = np.zeros(2, pt.SPHERE)
    spheres["center"], spheres["radius"] = (0.5, 0.5, 3.0), 0.5
    mats = np.zeros(1, pt.MATERIAL)
    tex = np.zeros(1, pt.TEXTURE)
    return pt.FlatScene(tri, spheres, None, mats, tex).build_bvh()


@pytest.mark.parametrize("wide,speculative,persistent", [(1, 1, 1), (1, 0, 1), (0, 1, 1), (0, 1, 0)])
@pytest.mark.parametrize("copies", [1, 7])
@pytest.mark.parametrize("tmin", [-10.0, -0.5, 0.0, 0.001])
def test_ties_and_signed_distances_match_oracle(wide, speculative, persistent, copies, tmin):
    scene = stacked_scene(copies)
    g = np.random.default_rng(5)
    n = 700
    rays = np.zeros(n, pt.RAY)
    rays["origin"] = np.c_[g.uniform(0.05, 0.95, (n, 2)), g.choice([-2.0, -1.0, 0.0, 0.25, 2.0], n)]
    rays["direction"] = (0, 0, 1)
    rays["direction"][n // 2:] = g.normal(size=(n - n // 2, 3))
    tmax = np.full(n, np.finfo(np.float32).max, np.float32)
    tmax[::3] = np.nextafter(np.float32(1.0), np.float32(2.0))     # just above the square one unit away
    tmax[1::3] = 1.0                                               # and exactly at it (not a hit)
    oracle = Oracle()
    pt.query_layout(wide)
    pt.query_walk(speculative)
    pt.query_tuning(persistent, 24, 0)
    try:
        dev = pt.Scene(scene)
        for t in (None, tmax):
            got, want = dev.query(rays, tmin=tmin, tmax=t), oracle.query(scene, rays, tmin=tmin, tmax=t)
            assert got.tobytes() == want.tobytes()
            blocked = dev.query(rays, mode=pt.QUERY_ANY, tmin=tmin, tmax=t)
            assert ((blocked["primitive_type"] != 0) == (want["primitive_type"] != 0)).all()
    finally:
        pt.query_layout(1)
        pt.query_walk(1)
        pt.query_tuning(1, 24, 0)


@pytest.mark.parametrize("mode", [pt.QUERY_CLOSEST, pt.QUERY_ANY])
def test_batches_of_every_size_class(mode):
    """Around the counts where a warp takes 4, 8 or 32 rays of its own and where the shared counter starts, for
    every walk form: each prefix of a batch has the prefix of its answers."""
    import torch
    scene, cam = pt.procedural_scene(512, 400, sphere_count=4, segments=24, rings=13, seed=2)
    dev = pt.Scene(scene)
    total = 204_800
    rays = torch.empty((total, 7), dtype=torch.float32, device="cuda")
    pt.camera_rays_device(cam, 512, 400, 3, 0, total, rays)

    def query(n):
        out = torch.full((n, 4), -7, dtype=torch.int32, device="cuda")
        dev.query_device(rays, n, out, mode=mode)
        torch.cuda.synchronize()
        return (out[:, 2] != 0) if mode == pt.QUERY_ANY else out

    try:
        for wide, speculative in ((1, 1), (1, 0), (0, 1)):
            pt.query_layout(wide)
            pt.query_walk(speculative)
            whole = query(total)                       # more rays than the grid holds: the shared counter
            assert (whole != 0).any()
            for n in (1, 3, 4, 5, 31, 33, 127, 129, 4735, 4736, 4737, 18_943, 18_945, 75_777, 151_551, 151_552, 151_553):
                assert torch.equal(query(n), whole[:n]), (wide, speculative, n)
    finally:
        pt.query_layout(1)
        pt.query_walk(1)
