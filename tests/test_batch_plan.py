"""The order in which a batch's samples are drawn (csrc/pt_batch_plan.h): every pixel gets its job's samples and
no item is drawn for nothing; and batches of very uneven jobs equal lone renderers."""
from __future__ import annotations

import subprocess
from pathlib import Path

import numpy as np
import pytest

import ptb200 as pt

CSRC = Path(pt.__file__).resolve().parents[1] / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "pt_batch_plan.h"
// stdin: few, jobs, then pixels and samples per job; stdout: items, then per job's pixel the samples it was given
int main() {
    long long few; int n;
    if (scanf("%lld %d", &few, &n) != 2) return 1;
    std::vector<int32_t> pixels(n), samples(n);
    for (int k = 0; k < n; k++) if (scanf("%d %d", &pixels[k], &samples[k]) != 2) return 1;
    const ptb::BatchPlan p = ptb::batch_plan(pixels, samples, few);
    std::vector<std::vector<long long>> given(n);
    for (int k = 0; k < n; k++) given[k].assign(pixels[k], 0);
    int dropped = 0;
    for (unsigned long long i = 0; i < p.items; i++) {
        const ptb::BatchItem at = ptb::batch_item(p.levels.data(), int(p.levels.size()), i);
        const int k = ptb::batch_job_at(p.first.data(), n, at.place), job = p.order[k];
        const unsigned in = at.place - p.first[k];
        if (in >= unsigned(pixels[job])) { dropped++; continue; }
        const int taken = at.drawn < 0 ? 1 : samples[job] - at.drawn;
        if (taken < 1) dropped++;
        if (at.drawn >= 0 && given[job][in] != at.drawn) dropped++;
        given[job][in] += taken;
    }
    long long wrong = 0;
    for (int k = 0; k < n; k++) for (long long g : given[k]) wrong += g != samples[k];
    printf("%llu %d %lld\n", p.items, dropped, wrong);
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(CSRC), "-o", str(d / "plan"), str(d / "plan.cpp")], check=True)
    return d / "plan"


def jobs_of(name: str):
    g = np.random.default_rng(7)
    return {
        "one": [(1, 1)], "equal": [(50, 4), (7, 4), (90, 4)], "rising": [(40, 1), (40, 2), (40, 3)], "falling": [(40, 9), (40, 5), (40, 1)],
        "heavy": [(3000, 1), (9, 1000)], "heavy first": [(1, 5000), (2000, 2)], "mixed": [(int(p), int(s)) for p, s in zip(g.integers(1, 300, 12), g.integers(1, 40, 12))],
    }[name]


@pytest.mark.parametrize("name", ["one", "equal", "rising", "falling", "heavy", "heavy first", "mixed"])
@pytest.mark.parametrize("few", [0, 1, 90, 100, 10**9])
def test_every_sample_is_drawn_once(program, name, few):
    jobs = jobs_of(name)
    text = f"{few} {len(jobs)}\n" + "\n".join(f"{p} {s}" for p, s in jobs)
    items, dropped, wrong = map(int, subprocess.run([program], input=text, capture_output=True, text=True, check=True).stdout.split())
    assert (dropped, wrong) == (0, 0)
    assert items <= sum(p * s for p, s in jobs)          # at most an item per sample
    if few == 0 or name == "equal" and few <= 100:
        assert items == sum(p * s for p, s in jobs)
    if few > 10**8:
        assert items == sum(p for p, _ in jobs)


# beside 262,144 pixels (past two per resident thread): one pixel, and a job that alone fills the threads
@pytest.mark.gpu
@pytest.mark.parametrize("width,height,samples", [(1, 1, 3000), (16, 16, 256), (600, 400, 12)])
@pytest.mark.parametrize("others", [1, 3])
def test_uneven_jobs_equal_lone_renderers(width, height, samples, others):
    a, cam_a = pt.procedural_scene(512, 512, sphere_count=4, segments=24, rings=13, seed=2, glass_fraction=0.5)
    _, cam_b = pt.procedural_scene(width, height, sphere_count=4, segments=24, rings=13, seed=2)
    jobs = [dict(scene=0, camera=cam_a, width=512, height=512, samples=others, max_depth=4, seed=1),
            dict(scene=0, camera=cam_b, width=width, height=height, samples=samples, max_depth=6, seed=2),
            dict(scene=0, camera=cam_b, width=width, height=height, samples=2, max_depth=3, seed=3)]
    b = pt.Batch([a], jobs)
    for _ in range(2):
        b.run()
    total = 0
    for k, j in enumerate(jobs):
        r = pt.CudaRenderer(a, j["camera"], j["width"], j["height"], j["seed"], max_depth=j["max_depth"])
        r.set_tail_paths(0)
        r.add_samples(j["samples"])
        total += r.rays_traced()
        assert b.sums(k).tobytes() == r.sums().tobytes(), k
    ms, rays, done = b.stats()
    assert rays == total and (done > 0).all()
