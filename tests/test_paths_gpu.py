"""The one-kernel render of four-wide trees (paths carried by persistent warps, samples of a pixel claimed
one by one) against the wavefront form: sums, streams and ray counts are the same bits."""
from __future__ import annotations

import numpy as np
import pytest

import ptb200 as pt

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene():
    flat, _ = pt.procedural_scene(64, 40, sphere_count=6, segments=24, rings=13, seed=3, metal_fraction=0.3, glass_fraction=0.4)
    return flat, pt.Scene(flat)


def render(scene, width, height, batches, depth, mis, tail):
    flat, dev = scene
    _, cam = pt.procedural_scene(width, height, sphere_count=6, segments=24, rings=13, seed=3)
    r = pt.CudaRenderer(dev, cam, width, height, 11, direct_light=mis, max_depth=depth)
    if tail is not None:
        r.set_tail_paths(tail)
    for n in batches:
        r.add_samples(n)
    return r.sums().tobytes(), r.rng_state().tobytes(), r.rays_traced()


# from a single pixel past two per resident thread (each side of the change from the tail kernel alone to the one
# kernel with hand-over); queues shorter and longer than the tail kernel's warps; one to many samples; several calls
@pytest.mark.parametrize("width,height,batches", [(1, 1, [2]), (1, 1, [1, 1, 2]), (31, 1, [2]), (33, 7, [1, 2]), (320, 240, [3]), (430, 260, [3]),
                                                  (400, 200, [1, 5, 2]), (401, 199, [24]), (512, 300, [4, 1]), (479, 395, [3]), (479, 396, [3]), (600, 331, [1, 7])])
@pytest.mark.parametrize("depth,mis", [(0, True), (3, False), (12, True)])
def test_equals_wavefront(scene, width, height, batches, depth, mis):
    assert render(scene, width, height, batches, depth, mis, None) == render(scene, width, height, batches, depth, mis, 0)


def test_equals_wavefront_after_reset_and_on_a_large_image(scene):
    flat, dev = scene
    _, cam = pt.procedural_scene(2100, 1500, sphere_count=6, segments=24, rings=13, seed=3)
    results = []
    for tail in (None, 1 << 20):
        r = pt.CudaRenderer(dev, cam, 2100, 1500, 5, max_depth=4)      # 3.15M pixels
        if tail is not None:
            r.set_tail_paths(tail)
        r.add_samples(1)
        r.reset(cam)
        r.add_samples(3)
        results.append((r.sums().tobytes(), r.rays_traced()))
    assert results[0] == results[1]
    assert np.frombuffer(results[0][0], np.float32).max() > 0


@pytest.mark.parametrize("k", [1, 2])
def test_batch_in_one_kernel_equals_its_graph_form_and_lone_renderers(k):
    """Uneven jobs (1 to 9 samples, an empty scene, a scene without emitters) below and past two pixels per resident thread."""
    a, cam_a = pt.procedural_scene(300 * k, 200 * k, sphere_count=4, segments=24, rings=13, seed=2, glass_fraction=0.5)
    b, cam_b = pt.cornell_box(180 * k, 150 * k)
    c, cam_c = pt.procedural_scene(90, 70, sphere_count=2, segments=16, rings=9, seed=7, light_fraction=0.0)
    scenes = [a, b, c, pt.FlatScene()]
    jobs = [dict(scene=0, camera=cam_a, width=300 * k, height=200 * k, samples=9, max_depth=9, seed=1),
            dict(scene=1, camera=cam_b, width=180 * k, height=150 * k, samples=2, max_depth=6, seed=2),
            dict(scene=2, camera=cam_c, width=90, height=70, samples=1, max_depth=3, seed=3),
            dict(scene=3, camera=cam_c, width=33, height=5, samples=4, max_depth=2, seed=4),
            dict(scene=0, camera=cam_a, width=300 * k, height=200 * k, samples=3, max_depth=0, seed=5)]
    batch = pt.Batch(scenes, jobs)
    forms = []
    for capacity in (0, 40000, 0):         # all pixels have a slot; a pool of 40,000 (graph loop); again after it
        batch.tuning(path_capacity=capacity)
        for _ in range(2):                 # a second run starts from a fresh state
            batch.run()
        ms, rays, done = batch.stats()
        assert (done > 0).all() and (done <= ms * 1.01 + 0.1).all()
        forms.append(([batch.sums(k).tobytes() for k in range(len(jobs))], rays))
    assert forms[0] == forms[1] == forms[2]
    for k, j in enumerate(jobs):
        if j["scene"] == 3:
            assert not np.frombuffer(forms[0][0][k], np.float32).any()
            continue
        r = pt.CudaRenderer(scenes[j["scene"]], j["camera"], j["width"], j["height"], j["seed"], max_depth=j["max_depth"])
        r.set_tail_paths(0)
        r.add_samples(j["samples"])
        assert r.sums().tobytes() == forms[0][0][k]


@pytest.mark.parametrize("width,height,spf,depth", [(64, 40, 1, 9), (400, 200, 1, 5), (401, 203, 3, 9), (320, 260, 8, 3), (31, 1, 1, 4), (655, 433, 2, 6), (656, 435, 2, 6), (800, 401, 1, 9)])
@pytest.mark.parametrize("use_cache,graph", [(True, True), (True, False), (False, True)])
def test_cached_frames_in_one_kernel_equal_the_wavefront(scene, width, height, spf, depth, use_cache, graph):
    """A frozen network: frames are the same bits whichever kernels ran them (a tail length asks for the wavefront)."""
    flat, dev = scene
    _, cam = pt.procedural_scene(width, height, sphere_count=6, segments=24, rings=13, seed=3)
    results = []
    for tail in (0, 20000):
        r = pt.CachedRenderer(dev, cam, width, height, seed=4, max_depth=depth, samples_per_frame=spf, train=False, use_cache=use_cache,
                              use_graph=graph, tail_paths=tail)
        for k in range(3):
            if k == 2:
                r.clear()
            r.frames(1)
        s = r.stats()
        results.append((r.sums().tobytes(), s["rays"], s["queries"], s["frames"]))
    assert results[0] == results[1]
    assert np.frombuffer(results[0][0], np.float32).max() > 0
    # none of the strip's 31 paths, in either form, ends at the cache
    assert (results[0][2] > 0) == (use_cache and height > 1)


@pytest.mark.parametrize("width,height", [(400, 220), (700, 420)])
def test_cached_training_in_one_kernel(scene, width, height):
    """Online training: the first frame's image uses the initial weights, so it and the counts are the wavefront's; the
    loss falls as it does there, and training-only frames mix with image frames."""
    flat, dev = scene
    _, cam = pt.procedural_scene(width, height, sphere_count=6, segments=24, rings=13, seed=3)
    first, last = [], []
    for tail in (0, 20000):
        r = pt.CachedRenderer(dev, cam, width, height, seed=4, max_depth=8, samples_per_frame=2, training_paths=8192, tail_paths=tail)
        r.frames(1)
        s = r.stats()
        first.append((r.sums().tobytes(), s["rays"], s["queries"], s["samples"]))
        r.train(20)
        r.frames(10)
        last.append(r.stats())
    assert first[0] == first[1] and first[0][3] > 0
    for s in last:
        assert np.isfinite(s["loss"]) and s["frames"] == 22
    # the same number of training samples within the scatter of two differently trained networks' path ends
    assert abs(last[0]["samples"] - last[1]["samples"]) <= 0.02 * last[1]["samples"]
    assert abs(last[0]["loss"] - last[1]["loss"]) <= 0.25 * last[1]["loss"]
