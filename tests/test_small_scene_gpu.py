"""Scenes held whole in shared memory (at most 32 primitives) against the general kernels and the
oracle: sums, streams and ray counts are the same bits whichever kernel ran."""
from __future__ import annotations

import numpy as np
import pytest

import ptb200 as pt
from oracle_bind import Oracle

pytestmark = pytest.mark.gpu


def box_scene(primitives: int) -> pt.FlatScene:
    """`primitives` primitives: an emitting quad, then spheres (all materials) and small triangles in turn."""
    g = np.random.default_rng(primitives)
    ntri = max(1, primitives - primitives // 2)
    tri = np.zeros(ntri, pt.TRIANGLE)
    c = g.uniform(-1, 1, (ntri, 3)).astype(np.float32)
    tri["v0"], tri["v1"], tri["v2"] = c, c + g.normal(0, 0.5, (ntri, 3)).astype(np.float32), c + g.normal(0, 0.5, (ntri, 3)).astype(np.float32)
    tri[0]["v0"], tri[0]["v1"], tri[0]["v2"] = (-2, 3, -2), (2, 3, -2), (0, 3, 3)
    tri["uv1"], tri["uv2"] = (1, 0, 0), (0, 1, 0)
    tri["material_id"] = np.r_[4, g.integers(0, 4, ntri - 1)]
    nsph = primitives - ntri
    sph = np.zeros(nsph, pt.SPHERE)
    sph["center"], sph["radius"] = g.uniform(-1, 1, (nsph, 3)), g.uniform(0.1, 0.5, nsph)
    sph["material_id"] = g.integers(0, 4, nsph)
    mats = np.zeros(5, pt.MATERIAL)
    mats["type"] = (0, 1, 2, 0, 3)
    mats["albedo"], mats["fuzz"], mats["ref_idx"] = (0.7, 0.6, 0.5), 0.1, 1.5
    mats["texture_id"] = (0, -1, -1, 1, 2)
    tex = np.zeros(3, pt.TEXTURE)
    tex["color"] = ((0.8, 0.3, 0.2), (0.2, 0.7, 0.4), (6, 6, 6))
    tex["scale"], tex["image_id"], tex["clamp"] = (1, 1, 0), -1, 1
    return pt.FlatScene(tri, sph if nsph else None, None, mats, tex).build_bvh()


@pytest.mark.parametrize("primitives", [1, 2, 3, 31, 32, 33])
@pytest.mark.parametrize("width,height,samples,mis", [(1, 1, 5, True), (33, 7, 3, True), (96, 61, 2, False), (400, 250, 1, True)])
def test_render_equals_general_kernels(primitives, width, height, samples, mis):
    scene = box_scene(primitives)
    cam = pt.make_camera((0, 0.5, 4), (0, 0, 0), vfov=50.0, aspect=width / height, aperture=0.05, focus_dist=4.0)
    results = []
    for tail in (None, 0, 1 << 30):      # None: the default kernel for the scene
        r = pt.CudaRenderer(scene, cam, width, height, 7, direct_light=mis, max_depth=6)
        if tail is not None:
            r.set_tail_paths(tail)
        r.add_samples(samples)
        r.add_samples(1)
        results.append((r.sums().tobytes(), r.rng_state().tobytes(), r.rays_traced()))
    assert results[0] == results[1] == results[2]


def test_parallel_and_degenerate_camera_rays():
    """Axis-parallel rays (infinite inverse directions) and origins on box planes."""
    scene, _ = pt.cornell_box(16, 16)
    cam = pt.make_camera((0.5, 0.5, 0.9), (0.5, 0.5, 0.0), vfov=1e-3, aspect=1.0)
    a = pt.CudaRenderer(scene, cam, 16, 16, 3, max_depth=4)
    b = pt.CudaRenderer(scene, cam, 16, 16, 3, max_depth=4)
    b.set_tail_paths(0)
    for r in (a, b):
        r.add_samples(4)
    assert a.sums().tobytes() == b.sums().tobytes() and a.rays_traced() == b.rays_traced()
    assert Oracle().validate(scene)
