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


# pixels below, at and above the resident threads; one to many samples (each side of the hand-over to the
# tail kernel, and of the samples below which few pixels run in one kernel); single pixels; several calls
@pytest.mark.parametrize("width,height,batches", [(1, 1, [2]), (1, 1, [1, 1, 2]), (31, 1, [2]), (33, 7, [1, 2]), (320, 240, [3]),
                                                  (400, 200, [1, 5, 2]), (401, 199, [24]), (512, 300, [4, 1])])
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
