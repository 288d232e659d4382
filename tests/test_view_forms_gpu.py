"""Which kernels render an image of ordinary size: the one that walks and shades where most paths end early, the
wavefront where they go on (csrc/pt_forms.h).  Inside a room the former took up to 1.7 times as long as the latter.

Told by memory: the wavefront's records, some 70 bytes a pixel, are allocated by the first call that needs them."""
from __future__ import annotations

import numpy as np
import pytest

import ptb200 as pt

pytestmark = pytest.mark.gpu
WIDTH, HEIGHT = 1280, 720            # 921,600 pixels
RECORDS = 40 << 20


def free() -> int:
    import torch
    return torch.cuda.mem_get_info()[0]


def room(width=WIDTH, height=HEIGHT):
    """The Cornell box, every triangle split into sixteen."""
    flat, cam = pt.cornell_box(width, height)
    t = flat.triangles
    for _ in range(2):
        a, b, c = t["v0"], t["v1"], t["v2"]
        ab, bc, ca = (a + b) / 2, (b + c) / 2, (c + a) / 2
        parts = []
        for corners in ((a, ab, ca), (ab, b, bc), (ca, bc, c), (ab, bc, ca)):
            q = t.copy()
            q["v0"], q["v1"], q["v2"] = corners
            parts.append(q)
        t = np.concatenate(parts)
    return pt.FlatScene(t, flat.spheres, None, flat.materials, flat.textures, flat.pixels).build_bvh(), cam


def spheres(width=WIDTH, height=HEIGHT):
    return pt.procedural_scene(width, height, sphere_count=4, segments=24, rings=13, seed=2)


@pytest.mark.parametrize("view,loop", [(room, True), (spheres, False)], ids=["room", "open"])
def test_renderer_form(view, loop):
    flat, cam = view()
    r = pt.CudaRenderer(flat, cam, WIDTH, HEIGHT, 3, max_depth=6)
    r.add_samples(2)
    want, before = r.sums().tobytes(), free()
    r.set_tail_paths(WIDTH * HEIGHT // 4)
    r.reset(cam)
    r.add_samples(2)
    assert (before - free() < RECORDS) == loop
    assert r.sums().tobytes() == want


@pytest.mark.parametrize("view,loop", [(room, True), (spheres, False)], ids=["room", "open"])
def test_batch_form(view, loop):
    flat, cam = view()
    b = pt.Batch([flat], [dict(scene=0, camera=cam, width=WIDTH, height=HEIGHT, samples=2, max_depth=6, seed=3)])
    b.run()
    want, before = b.sums(0).tobytes(), free()
    b.tuning(tail_paths=20000)
    b.run()
    assert (before - free() < RECORDS) == loop
    assert b.sums(0).tobytes() == want


@pytest.mark.parametrize("view,loop", [(room, True), (spheres, False)], ids=["room", "open"])
def test_cached_form(view, loop):
    flat, cam = view()
    r = pt.CachedRenderer(flat, cam, WIDTH, HEIGHT, seed=3, max_depth=6, samples_per_frame=2)
    r.frames(1)
    before = free()
    r.train(1)                       # training-only frames run in the wavefront
    assert (before - free() < RECORDS) == loop


def test_reset_looks_at_the_new_view():
    flat, inside = room()
    away = pt.make_camera((40, 0.5, 0.5), (60, 0.5, 0.5), (0, 1, 0), 40.0, WIDTH / HEIGHT)
    r = pt.CudaRenderer(flat, away, WIDTH, HEIGHT, 3, max_depth=6)
    r.add_samples(2)
    before = free()
    r.reset(inside)
    r.add_samples(4)                 # a call of few samples would not wait for the look
    assert before - free() >= RECORDS
    want = pt.CudaRenderer(flat, inside, WIDTH, HEIGHT, 3, max_depth=6)
    want.add_samples(4)
    assert r.sums().tobytes() == want.sums().tobytes()
    r.reset(away)
    r.add_samples(1)
    r.reset(inside)
    r.add_samples(1)
    r.add_samples(3)
    assert r.sums().tobytes() == want.sums().tobytes()


def test_batch_of_rooms_and_open_views():
    """Two rooms of 20,000 pixels among 600,000 of an open scene, and against a lone renderer each."""
    a, cam_a = room(200, 100)
    b, cam_b = spheres(1000, 600)
    jobs = [dict(scene=0, camera=cam_a, width=200, height=100, samples=3, max_depth=6, seed=1),
            dict(scene=1, camera=cam_b, width=1000, height=600, samples=1, max_depth=4, seed=2),
            dict(scene=0, camera=cam_a, width=200, height=100, samples=2, max_depth=9, seed=3)]
    batch = pt.Batch([a, b], jobs)
    batch.run()
    before = free()
    for k, j in enumerate(jobs):
        r = pt.CudaRenderer((a, b)[j["scene"]], j["camera"], j["width"], j["height"], j["seed"], direct_light=True, max_depth=j["max_depth"])
        r.add_samples(j["samples"])
        assert batch.sums(k).tobytes() == r.sums().tobytes()
        r.close()
    before = free()
    batch.tuning(tail_paths=20000)
    batch.run()
    assert before - free() >= RECORDS // 2


@pytest.mark.parametrize("segments,rings", [(5, 5), (6, 6), (8, 8), (10, 10)])
@pytest.mark.parametrize("width,height", [(64, 40), (640, 400), (1280, 720)])
def test_trees_of_a_few_nodes(segments, rings, width, height):
    """Scenes of 33 to some 190 triangles: the forms of larger scenes, and the wavefront's own when asked for."""
    flat, cam = pt.procedural_scene(width, height, sphere_count=1, segments=segments, rings=rings, seed=4)
    r = pt.CudaRenderer(flat, cam, width, height, 3, max_depth=6)
    r.add_samples(3)
    want, rays, before = r.sums().tobytes(), r.rays_traced(), free()
    r.set_tail_paths(500)
    r.reset(cam)
    r.add_samples(3)
    assert r.sums().tobytes() == want and r.rays_traced() == rays
    if width == WIDTH:
        assert before - free() >= RECORDS
    brute = pt.CudaRenderer(flat, cam, width, height, 3, max_depth=6, brute=True)
    brute.add_samples(3)
    assert brute.rays_traced() == rays and brute.sums().tobytes() == want


def test_small_room():
    """80 triangles in a room: the two-lane kernel alone for a small image, the two-wide wavefront for a large one."""
    flat, cam = pt.cornell_box(320, 200)
    t = flat.triangles
    parts = [t.copy() for _ in range(4)]
    mid = (t["v0"] + t["v1"] + t["v2"]) / np.float32(3)
    flat = pt.FlatScene(np.concatenate(parts), flat.spheres, None, flat.materials, flat.textures, flat.pixels)
    for k, (a, b) in enumerate((("v0", "v1"), ("v1", "v2"), ("v2", "v0"))):      # three parts around the centroid
        part = flat.triangles[k * len(t):(k + 1) * len(t)]
        part["v0"], part["v1"], part["v2"] = t[a], t[b], mid
    flat = pt.FlatScene(flat.triangles[:3 * len(t)], flat.spheres, None, flat.materials, flat.textures, flat.pixels).build_bvh()
    for width, height in ((320, 200), (900, 560)):
        _, cam = pt.cornell_box(width, height)
        r = pt.CudaRenderer(flat, cam, width, height, 3, max_depth=6)
        r.add_samples(2)
        want = r.sums().tobytes()
        r.set_tail_paths(500)
        r.reset(cam)
        r.add_samples(2)
        assert r.sums().tobytes() == want


@pytest.mark.parametrize("samples", [3, 4])
def test_open_view_of_few_pixels_and_samples(samples):
    """256,000 pixels of an open scene: the tail kernel alone from four samples, one call or split."""
    flat, cam = spheres(640, 400)
    r = pt.CudaRenderer(flat, cam, 640, 400, 3, max_depth=6)
    r.add_samples(samples)
    want, rays = r.sums().tobytes(), r.rays_traced()
    r.reset(cam)
    r.add_samples(1)
    r.add_samples(samples - 1)
    assert r.sums().tobytes() == want and r.rays_traced() == rays
    r.set_tail_paths(500)
    r.reset(cam)
    r.add_samples(samples)
    assert r.sums().tobytes() == want
