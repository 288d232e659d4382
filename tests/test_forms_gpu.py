"""The loop forms of batches and cached frames that the sizes of the other tests no longer reach by
default: a tail length other than the default asks for them."""
from __future__ import annotations

import pytest

import ptb200 as pt

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def job():
    flat, _ = pt.procedural_scene(64, 40, sphere_count=4, segments=24, rings=13, seed=2, glass_fraction=0.5)

    def make(width, height, samples):
        _, cam = pt.procedural_scene(width, height, sphere_count=4, segments=24, rings=13, seed=2)
        return [flat], [dict(scene=0, camera=cam, width=width, height=height, samples=samples, max_depth=6, seed=3)]
    return make


def alone(scenes, j, mis):
    r = pt.CudaRenderer(scenes[0], j["camera"], j["width"], j["height"], j["seed"], direct_light=mis, max_depth=j["max_depth"])
    r.set_tail_paths(0)
    r.add_samples(j["samples"])
    return r.sums().tobytes(), r.rays_traced()


# 6,000 pixels: the tail kernel alone by default; 208,000: one kernel by default
@pytest.mark.parametrize("width,height", [(100, 60), (520, 400)])
def test_batch_tail_setting_asks_for_the_loop(job, width, height):
    """The loop's records (over 60 bytes a slot) are allocated with the first run that needs them."""
    import torch
    b = pt.Batch(*job(width, height, 2))
    b.tuning(tail_paths=16384)
    b.run()
    first = torch.cuda.mem_get_info()[0]
    b.run()
    assert torch.cuda.mem_get_info()[0] == first
    hold = torch.cuda.mem_get_info()[0]
    b.tuning(tail_paths=20000)
    b.run()
    if width * height > 100_000:
        assert hold - torch.cuda.mem_get_info()[0] > 8 << 20
    b.tuning(tail_paths=16384)
    held = torch.cuda.mem_get_info()[0]
    b.run()
    assert torch.cuda.mem_get_info()[0] == held


@pytest.mark.parametrize("width,height", [(100, 60), (520, 400)])
@pytest.mark.parametrize("mis", [True, False])
def test_batch_forms_equal_a_lone_renderer(job, width, height, mis):
    scenes, jobs = job(width, height, 3)
    want, rays = alone(scenes, jobs[0], mis)
    b = pt.Batch(scenes, jobs, direct_light=mis)
    for tail in (16384, 0, 5000, 1 << 30):               # the form of the size; the loop to its end, with a tail, one round of it
        for graph in (1, 0):
            b.tuning(tail_paths=tail, use_graph=graph)
            b.run()
            assert b.sums(0).tobytes() == want, (tail, graph)
            assert b.stats()[1] == rays


def test_cached_loop_graph_equals_launches():
    flat, cam = pt.cornell_box(96, 64)
    out = []
    for graph in (1, 0):
        r = pt.CachedRenderer(flat, cam, 96, 64, seed=5, max_depth=8, train=0, use_graph=graph, tail_paths=500)
        r.frames(4)
        assert r.stats()["queries"] > 0
        out.append(r.sums().tobytes())
    assert out[0] == out[1]


def test_autotune_keeps_the_answer_and_the_sample_counts(job):
    scenes, jobs = job(520, 400, 3)
    b = pt.Batch(scenes, jobs)
    best = b.autotune(probe_samples=1)
    assert best[3] in (0, 1) and best[4] in (0, 1)
    b.run()
    assert b.sums(0).tobytes() == alone(scenes, jobs[0], True)[0]
