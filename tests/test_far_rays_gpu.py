"""Closest-hit and any-hit queries of small scenes by rays that start far away, against the brute-force scan.

Triangles of unit size, flat along one axis, lie 4 units apart.  Rays aim at their centroids from up to 10^6
scene sizes.  With u = 2^-24 and D the distance, the rounded ray passes within 3 u D of the centroid and the
triangle test is off by at most 4 u D / 0.4 within the triangle's plane, so a triangle other than the aimed one
could only be hit, in either form, where the boxes' widening by 8 u D takes in all of them anyway."""
from __future__ import annotations

import numpy as np
import pytest

import ptb200 as pt

pytestmark = pytest.mark.gpu


def plates(count: int) -> tuple[pt.FlatScene, np.ndarray]:
    g = np.random.default_rng(count)
    tri = np.zeros(count, pt.TRIANGLE)
    corner = 4.0 * np.stack([np.arange(count) % 4, np.arange(count) // 4 % 3, np.arange(count) // 12], axis=1)
    v = np.repeat(corner[:, None], 3, axis=1)
    for k in range(count):
        a = k % 3                                        # the flat axis
        v[k, 1, (a + 1) % 3] += 1
        v[k, 2, (a + 2) % 3] += 1
    v = (v + g.uniform(-0.3, 0.3, (count, 1, 3))).astype(np.float32)
    tri["v0"], tri["v1"], tri["v2"] = v[:, 0], v[:, 1], v[:, 2]
    mats = np.zeros(1, pt.MATERIAL)
    mats["texture_id"], mats["ref_idx"] = 0, 1
    tex = np.zeros(1, pt.TEXTURE)
    tex["color"], tex["scale"], tex["image_id"], tex["clamp"] = (1, 1, 1), (1, 1, 0), -1, 1
    return pt.FlatScene(tri, None, None, mats, tex).build_bvh(), v.mean(axis=1, dtype=np.float64)


@pytest.mark.parametrize("count", [1, 2, 3, 31, 32])
@pytest.mark.parametrize("sizes", [1e2, 1e4, 1e5, 1e6])
@pytest.mark.parametrize("parallel", [True, False], ids=["axis-parallel", "oblique"])
def test_far_rays_equal_brute_force(count, sizes, parallel):
    import torch
    scene, centers = plates(count)
    n = 4096
    g = np.random.default_rng(count + 1)
    aim = np.arange(n) % count
    sign = g.choice([-1.0, 1.0], (n, 3))
    if parallel:
        d = np.zeros((n, 3))
        d[np.arange(n), aim % 3] = sign[:, 0]            # across the plate's plane
    else:
        d = g.uniform(0.45, 1.0, (n, 3)) * sign
        d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.zeros(n, pt.RAY)
    rays["origin"] = centers[aim] - 16.0 * sizes * d
    rays["direction"] = d
    on_device = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    dev = pt.Scene(scene)

    def query(mode, brute):
        out = torch.full((n * 16,), 255, dtype=torch.uint8, device="cuda")
        dev.query_device(on_device, n, out, mode=mode, brute=brute)
        torch.cuda.synchronize()
        return out.cpu().numpy().view(pt.HIT)

    want = query(pt.QUERY_CLOSEST, True)
    if parallel:
        assert (want["primitive_type"] != 0).all()
    assert query(pt.QUERY_CLOSEST, False).tobytes() == want.tobytes()
    assert ((query(pt.QUERY_ANY, False)["primitive_type"] != 0) == (want["primitive_type"] != 0)).all()
