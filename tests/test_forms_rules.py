"""csrc/pt_forms.h: the sizes up to which one kernel takes an image, on either side of the pairs it was measured at."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

import ptb200 as pt

CSRC = Path(pt.__file__).resolve().parents[1] / "csrc"
PROGRAM = r"""
#include <cstdio>
#include "pt_forms.h"
int main() {
    using namespace ptb;
    char kind; double a, b, c, d;
    while (scanf(" %c %lf %lf %lf %lf", &kind, &a, &b, &c, &d) == 5) {
        if (kind == 'r') printf("%g\n", most_pixels_going_on(size_t(a)));
        if (kind == 'o') printf("%g\n", most_pixels_open(size_t(a), int64_t(b)));
        if (kind == 'c') printf("%g\n", most_pixels_cached(a != 0, size_t(b), size_t(c), int64_t(d)));
        if (kind == 'b') printf("%d\n", int(batch_in_one(a, b, c, size_t(d), 1.0)));
        if (kind == 'a') printf("%g\n", most_pixels_alone(a != 0, size_t(b), int64_t(c)));
        if (kind == 'p') printf("%d\n", int(paths_go_on(uint32_t(a))));
    }
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("forms")
    (d / "forms.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-o", str(d / "forms"), str(d / "forms.cpp")], check=True)

    def ask(kind, *values):
        text = " ".join([kind, *(str(float(v)) for v in (*values, 0, 0, 0, 0)[:4])])
        return float(subprocess.run([str(d / "forms")], input=text, capture_output=True, text=True, check=True).stdout)
    return ask


def test_rooms(rule):
    assert rule("r", 1283) < 2.4 <= rule("r", 20483) < 6.1 < rule("r", 327683) < 22      # kernel, wavefront
    assert rule("p", 1280) == 1 and rule("p", 1279) == 0 and rule("p", 0) == 0


def test_open_views(rule):
    light, heavy = 1e6, 60e6
    assert rule("o", light, 8) >= 39 and rule("o", light, 2) < 39
    assert 9.7 < rule("o", heavy, 2) < 15
    assert 22 < rule("o", heavy, 8) < 30
    assert 30 < rule("o", heavy, 32) < 39
    assert rule("o", heavy, 0) == rule("o", heavy, 7)                                    # a limit of no bounces
    assert 9.7 < rule("o", 170e6, 32) < 22 and rule("o", 170e6, 2) < 6.1
    for size in (0, light, heavy, 1e12):
        steps = [rule("o", size, b) for b in (0, 1, 4, 8, 32, 128, 1e6)]
        assert steps == sorted(steps) and steps[0] > 2 and steps[-1] <= 40


def test_cached(rule):
    heavy = 60e6
    assert rule("c", 0, 1e6, heavy, 48) == 28 and rule("c", 0, 1e6, heavy, 12) == 20
    assert rule("c", 1, 1283, heavy, 48) < 22 and 6.1 < rule("c", 1, 20483, heavy, 48) < 22 < rule("c", 1, 327683, heavy, 48)
    assert rule("c", 1, 1e9, heavy, 12) == 20
    assert 9.7 < rule("c", 0, 2.6e6, 170e6, 12) < 15 and 9.7 < rule("c", 0, 2.6e6, 170e6, 48) < 15


def test_batches(rule):
    light, heavy = 1e6, 60e6
    cornell = rule("r", 23)
    assert rule("b", 5.1, 2.4, cornell, light) == 1 and rule("b", 10.2, 4.9, cornell, light) == 0
    assert rule("b", 0, 2.3, cornell, light) == 0                                        # rooms alone
    assert rule("b", 29, 0, 0, light) == 1 and rule("b", 31, 0, 0, light) == 0
    assert rule("b", 21, 0, 0, heavy) == 1 and rule("b", 23, 0, 0, heavy) == 0
    assert rule("b", 5.2, 0, 0, 170e6) == 1 and rule("b", 10.6, 0, 0, 170e6) == 0


def test_tail_kernel_alone(rule):
    light, heavy = 6e6, 14e6
    assert 2.7 < rule("a", 0, light, 4) < 4.1 and rule("a", 0, light, 1) <= 2
    assert rule("a", 0, heavy, 16) <= 2.7 and rule("a", 1, light, 16) <= 2.7
    for size in (0, light, heavy, 1e12):                                                 # the other form takes over above it
        for samples in (1, 4, 16, 1e6):
            assert rule("a", 0, size, samples) <= rule("o", size, samples)
