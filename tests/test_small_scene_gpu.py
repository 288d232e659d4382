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


def flat_boxes(scene: pt.FlatScene) -> pt.FlatScene:
    """The same tree with every box shrunk to its primitives' bounds (flat for axis-aligned triangles)."""
    s = scene.copy()
    lo, hi = np.zeros((len(s.nodes), 3), np.float32), np.zeros((len(s.nodes), 3), np.float32)

    def fit(k):
        n = s.nodes[k]
        if n["type"] == 0:
            a, b = fit(int(n["left"])), fit(int(n["right"]))
            lo[k], hi[k] = np.minimum(a[0], b[0]), np.maximum(a[1], b[1])
        elif n["type"] == 1:
            t = s.triangles[n["primitive"]]
            v = np.stack([t["v0"], t["v1"], t["v2"]])
            lo[k], hi[k] = v.min(axis=0), v.max(axis=0)
        else:
            p = s.spheres[n["primitive"]]
            r = np.nextafter(p["radius"], np.float32(np.inf)) * np.float32(1.000001)
            lo[k], hi[k] = p["center"] - r, p["center"] + r
        return lo[k], hi[k]

    fit(s.root)
    s.nodes["minimum"], s.nodes["maximum"] = lo, hi
    return s


@pytest.mark.parametrize("primitives", [1, 2, 3, 31, 32, 33])
@pytest.mark.parametrize("flat", [False, True])
@pytest.mark.parametrize("count", [1, 31, 64, 1000, 200_001])
def test_query_equals_general_walk_and_brute_force(primitives, flat, count):
    """Random and axis-parallel rays; the single-loop walk and the brute-force scan never use the shared-memory form.
    200,001 rays are more than the resident grid of either kernel holds at once."""
    import torch
    scene = box_scene(primitives)
    scene.triangles["v1"][0::2, 1] = scene.triangles["v0"][0::2, 1]      # every other triangle axis-aligned
    scene.triangles["v2"][0::2, 1] = scene.triangles["v0"][0::2, 1]
    scene = scene.build_bvh()
    if flat:
        scene = flat_boxes(scene)
    assert Oracle().validate(scene)
    g = np.random.default_rng(count)
    rays = np.zeros(count, pt.RAY)
    rays["origin"] = g.uniform(-2, 2, (count, 3))
    rays["direction"] = g.normal(size=(count, 3))
    rays["direction"][::5, 0] = 0
    rays["direction"][::7, 2] = 0
    rays["direction"][::35, 1] = 0                                       # some have no direction at all
    d = torch.from_numpy(rays.view(np.uint8).copy()).cuda()
    tmax = torch.from_numpy(g.uniform(0.1, 5, count).astype(np.float32)).cuda()
    dev = pt.Scene(scene)

    def query(mode, t, brute=False):
        out = torch.full((count * 16,), 255, dtype=torch.uint8, device="cuda")
        dev.query_device(d, count, out, mode=mode, tmax=t, brute=brute)
        torch.cuda.synchronize()
        return out.cpu().numpy().view(pt.HIT)

    for t in (None, tmax):
        got, brute = query(pt.QUERY_CLOSEST, t), query(pt.QUERY_CLOSEST, t, True)
        blocked = query(pt.QUERY_ANY, t)["primitive_type"] != 0
        pt.query_walk(0)
        try:
            walk = query(pt.QUERY_CLOSEST, t)
        finally:
            pt.query_walk(1)
        assert got.tobytes() == walk.tobytes() == brute.tobytes()
        assert (blocked == (got["primitive_type"] != 0)).all()
