"""A batch whose records cannot be had: the call fails with an error, and the next run, once there is memory
again, allocates them anew instead of using what the failed call had freed."""
from __future__ import annotations

import pytest

import ptb200 as pt

pytestmark = pytest.mark.gpu
WIDTH, HEIGHT = 1000, 900            # one kernel by default; the loop's records take some 140 MB


@pytest.fixture(scope="module")
def made():
    flat, _ = pt.procedural_scene(64, 40, sphere_count=2, segments=24, rings=13, seed=2)
    _, cam = pt.procedural_scene(WIDTH, HEIGHT, sphere_count=2, segments=24, rings=13, seed=2)
    jobs = [dict(scene=0, camera=cam, width=WIDTH, height=HEIGHT, samples=1, max_depth=3, seed=3)]
    b = pt.Batch([flat], jobs)       # every kernel has run once: what a run allocates after this is its records
    for tail in (0, 16384):
        b.tuning(tail_paths=tail)
        b.run()
    want = b.sums(0).tobytes()
    b.close()
    return [flat], jobs, want


@pytest.mark.parametrize("setting", [dict(tail_paths=0), dict(path_capacity=WIDTH * HEIGHT - 1, tail_paths=0)],
                         ids=["tail length", "capacity"])
def test_run_after_a_failed_allocation(made, setting):
    import torch
    scenes, jobs, want = made
    b = pt.Batch(scenes, jobs)
    b.run()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - (64 << 20), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(pt.PtError):
            b.tuning(**setting)
            b.run()
        with pytest.raises(pt.PtError):
            b.run()
    finally:
        del held
        torch.cuda.empty_cache()
    b.run()
    assert b.sums(0).tobytes() == want
    b.tuning()
    b.run()
    assert b.sums(0).tobytes() == want
