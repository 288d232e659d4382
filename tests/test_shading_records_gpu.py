"""Shading through the per-triangle and per-emitter records: smooth faces, image and mapped textures on
triangles and spheres, textured triangle and sphere emitters, against the oracle.

At bounce limit 0 with textures on emitters only, a pixel is an emitted texel: the triangle half of
the image is the oracle's bit for bit (no transcendental function is involved); on spheres atan2f and
asinf may differ from glibc's in the last place, which can move a texel lookup to its neighbour, so
fewer than 1 % of the pixels may differ.  At bounce limit 2 the bar is the repository's statistical one."""
from __future__ import annotations

import numpy as np
import pytest

import ptb200 as pt
from oracle_bind import Oracle

pytestmark = pytest.mark.gpu


def textured_scene(emit: bool, smooth: bool, spheres: bool) -> pt.FlatScene:
    g = np.random.default_rng(11)
    tri = np.zeros(8, pt.TRIANGLE)
    c = np.array([(-2, -1, 0), (2, -1, 0), (2, 1, 0), (-2, 1, 0)], np.float32)
    for k, (a, b, d) in enumerate([(0, 1, 2), (0, 2, 3)]):
        tri[k]["v0"], tri[k]["v1"], tri[k]["v2"] = c[a], c[b], c[d]
        tri[k]["uv0"], tri[k]["uv1"], tri[k]["uv2"] = [((c[i] + (2, 1, 0)) / (4, 2, 1)) for i in (a, b, d)]
    tri[2:]["v0"] = g.uniform(-1, 1, (6, 3)) + (0, 0, 1)
    tri[2:]["v1"] = tri[2:]["v0"] + g.normal(0, 0.4, (6, 3))
    tri[2:]["v2"] = tri[2:]["v0"] + g.normal(0, 0.4, (6, 3))
    tri["uv1"][2:], tri["uv2"][2:] = (1, 0, 0), (0.3, 1, 0)
    tri["material_id"] = np.r_[0, 1, 0, 1, 2, 0, 1, 3]
    if smooth:
        tri["smooth"] = 1
        for k in ("n0", "n1", "n2"):
            tri[k] = np.float32([0, 0, 1]) + g.normal(0, 0.2, (8, 3)).astype(np.float32)
    sph = np.zeros(2 if spheres else 0, pt.SPHERE)
    if spheres:
        sph["center"], sph["radius"], sph["material_id"] = [(-0.8, 0.3, 1.5), (0.9, -0.2, 1.2)], 0.4, [3, 1]
    mats = np.zeros(4, pt.MATERIAL)
    mats["type"] = 3 if emit else 0
    mats["type"][3] = 3
    mats["texture_id"] = (0, 1, 2, 1)
    mats["ref_idx"] = 1
    tex = np.zeros(4, pt.TEXTURE)
    tex["type"] = (pt.TEX_IMAGE if hasattr(pt, "TEX_IMAGE") else 1, 2, 0, 1)
    tex["color"] = ((1, 1, 1), (0.9, 0.5, 0.7), (0.2, 0.4, 0.6), (1, 1, 1))
    tex["scale"], tex["offset"] = (3, 2, 0), (0.25, 0.5, 0)
    tex["image_id"] = (-1, 3, -1, -1)
    tex["width"], tex["height"] = (5, 0, 0, 4), (3, 0, 0, 7)
    tex["byte_offset"] = (0, 0, 0, 45)
    tex["clamp"] = (1, 0, 1, 1)
    pixels = g.integers(0, 256, 45 + 84).astype(np.uint8)
    return pt.FlatScene(tri, sph, None, mats, tex, pixels).build_bvh()


CAMERA = ((0, 0, 6), (0, 0, 0))


@pytest.mark.parametrize("tail", [None, 0])
@pytest.mark.parametrize("spheres", [False, True])
def test_emitted_texels_match_oracle(spheres, tail):
    scene = textured_scene(True, False, spheres)
    oracle = Oracle()
    assert oracle.validate(scene)
    cam = pt.make_camera(*CAMERA, vfov=35.0, aspect=1.6)
    r = pt.CudaRenderer(scene, cam, 80, 50, 3, max_depth=0)
    if tail is not None:
        r.set_tail_paths(tail)
    r.add_samples(2)
    want, _, _ = oracle.render(scene, cam, 80, 50, 3, [2], max_depth=0)
    differ = (r.sums().reshape(-1, 3) != np.asarray(want, np.float32).reshape(-1, 3)).any(axis=1).mean()
    assert differ < (0.01 if spheres else 1e-12)
    assert r.sums().max() > 0


@pytest.mark.parametrize("smooth", [False, True])
@pytest.mark.parametrize("mis", [True, False])
def test_textured_scatter_is_statistically_the_oracles(smooth, mis):
    scene = textured_scene(False, smooth, True)
    cam = pt.make_camera(*CAMERA, vfov=35.0, aspect=1.6)
    r = pt.CudaRenderer(scene, cam, 80, 50, 5, direct_light=mis, max_depth=2)
    r.add_samples(4)
    want, _, rays = Oracle().render(scene, cam, 80, 50, 5, [4], max_depth=2, mis=mis)
    a, b = r.sums().reshape(-1, 3).astype(np.float64) / 4, np.asarray(want).reshape(-1, 3).astype(np.float64) / 4
    d = (a - b).mean(axis=1)
    assert abs(d.mean()) <= 4 * d.std() / np.sqrt(len(d)) + 1e-7
    assert abs(int(r.rays_traced()) - int(rays)) <= 0.01 * rays
