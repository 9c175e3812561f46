"""The step kernel's plan (csrc/march_plan.h: staging geometry and planes per
block) on 152 SMs: on boxes where an earlier rule lost time it takes a plan
measured to be no slower than the step with a fixed two-block geometry, which
it replaced; and the boxes that the GPU tests of a geometry run take it."""
from __future__ import annotations

import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <cstdio>
#include "march_plan.h"

int main()
{
    int x, y, z;
    while (std::scanf("%d %d %d", &x, &y, &z) == 3) {
        const long long tiles = (long long)(x / 32) * (y / 8);
        const lbm::StepPlan a = lbm::step_plan_fp32(tiles, z, 152, 2, 3), b = lbm::step_plan_16bit(tiles, z, 152, 4);
        std::printf("%s %d %d\n", a.deep ? "deep" : "dense", a.tz, b.tz);
    }
}
"""

# Plans (depths of the FP32 kernel's two geometries, of the 16-bit kernel's one)
# measured within 0.4 % of the replaced rule's time or faster.
FP32 = {
    (384, 320, 40): {"deep": {8, 9, *range(12, 19), 25, 26, 27, 28}, "dense": {*range(6, 19), 27}},
    (320, 192, 22): {"deep": {5, 6, 7, 9, 10, 13, 14, 15, *range(17, 23)}, "dense": {4, 5, 6, 7, 8, 14, 15}},
    (384, 384, 32): {"deep": {26, 27, 28, 32}, "dense": {*range(10, 16), 20, 21, 22, 23}},
    (256, 256, 12): {"deep": {9, 10, 11, 12}, "dense": {8}},
    (32, 104, 72): {"deep": {4, 7}, "dense": set()},
    (160, 40, 38): {"deep": {4, 7}, "dense": {7}},
    (160, 160, 34): {"deep": {11, 12}, "dense": {8}},
    (256, 128, 48): {"deep": {7, 11, 21, 22, 23, 24}, "dense": {5, 7, 14, 15, 16, 17}},
    (160, 104, 93): {"deep": {6, 7, 8, 10, 11, *range(21, 26)}, "dense": {5, 7, 8, *range(13, 18)}},
    (256, 256, 256): {"deep": {12, 14, 15, *range(17, 24), 25, 27, 28, 29, 32, 37}, "dense": {*range(9, 28), 37}},
}
BIT16 = {
    (448, 256, 30): {6, 7, 8, 9, 12, 13, 23, 24},
    (416, 416, 44): {*range(6, 15), *range(16, 21)},
    (416, 400, 42): {*range(5, 21), 25, 26, 27, 28},
    (352, 480, 14): set(range(4, 12)),
    (160, 488, 19): {4, 5, 6, 7, 8, 11},
    (512, 384, 18): set(range(5, 16)),
    (640, 280, 38): {*range(6, 19), *range(24, 29)},
    (160, 104, 93): {4, 5, 6, 7, 8, 10, 11},
    (256, 256, 256): {*range(7, 30), 37},
    (192, 192, 192): {*range(5, 29), 48},
}


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "p.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "lbm_bench_gpu_gb300" / "csrc"), str(d / "p.cpp"),
                    "-o", str(d / "p")], check=True)

    def of(*box):
        r = subprocess.run([str(d / "p")], input="%d %d %d" % box, capture_output=True, text=True, check=True)
        geometry, tz, tz16 = r.stdout.split()
        return geometry, int(tz), int(tz16)

    return of


def test_plans_are_no_slower_than_the_replaced_rule(plan):
    for box, good in FP32.items():
        geometry, tz, _ = plan(*box)
        assert tz in good[geometry], (box, geometry, tz)
    for box, good in BIT16.items():
        assert plan(*box)[2] in good, (box, plan(*box))


def test_boxes_of_the_geometry_tests_take_their_geometry(plan):
    for box in ((32, 96, 110), (96, 64, 95), (160, 104, 93), (256, 256, 256)):
        assert plan(*box)[0] == "dense", box
    for box in ((32, 8, 12), (64, 32, 48), (128, 32, 16), (64, 64, 64), (32, 96, 2)):
        assert plan(*box)[0] == "deep", box


@pytest.mark.parametrize("planes", [1, 2, 3, 5, 17, 64, 255])
def test_depths_stay_within_the_box(plan, planes):
    for x, y in ((32, 8), (32, 96), (160, 104), (256, 256), (512, 512)):
        _, tz, tz16 = plan(x, y, planes)
        assert 1 <= tz <= planes and 1 <= tz16 <= planes
