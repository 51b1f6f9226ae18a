"""How the batched form for few vectors cuts a product, and where it is taken, on the CPU."""
import itertools
import math
import os
import subprocess

import pytest

import test_gpu_few as gpu
from orome_b200 import synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SMEM_OPTIN, SMS = 232448, 148      # of a B200
NAMES = {synth.Q4_K: "q4_k", synth.Q5_K: "q5_k", synth.Q6_K: "q6_k", synth.Q8_0: "q8_0"}
FMT = {v: k for k, v in NAMES.items()}
PITCH = {synth.Q4_K: 160, synth.Q5_K: 224, synth.Q6_K: 224, synth.Q8_0: 288}      # bytes between the rows of a stage's chunk

PROGRAM = r"""
#include "few_plan.h"
#include <cstdio>
using namespace orome;
int main()
{
    int fmt, fused;
    unsigned rows, cols, batch;
    while (scanf("%d %u %u %u %d", &fmt, &rows, &cols, &batch, &fused) == 5) {
        FewShape in{fmt, rows, cols, batch, fused != 0, SMS, SMEM};
        FewPlan p = {};
        const bool fits = few_plan(in, p);
        printf("%d %d %u %u %u %u %u %u %u %u %u %u\n", (int)few_faster(in), (int)fits, p.grid, p.tiles, p.passes, p.rt, p.kp, p.steps, p.nstages, p.stage_base, p.stage_bytes, p.bytes);
    }
}
"""


class Plan:
    def __init__(self, shape, values):
        self.fmt, self.rows, self.cols, self.batch, self.fused = shape
        (self.faster, self.fits, self.grid, self.tiles, self.passes, self.rt, self.kp, self.steps, self.nstages, self.base, self.stage, self.bytes) = values
        self.chunks, self.fills = self.cols // 256, self.passes * self.steps


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    d = tmp_path_factory.mktemp("few")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", f"-DSMS={SMS}", f"-DSMEM={SMEM_OPTIN}", "-I", os.path.join(ROOT, "orome_b200", "csrc"), "-o", str(d / "plan"), str(d / "plan.cpp")])

    def run(shapes):
        text = "\n".join(" ".join(str(int(v)) for v in s) for s in shapes)
        out = subprocess.run([str(d / "plan")], input=text, capture_output=True, text=True, check=True).stdout
        return [Plan(s, tuple(int(v) for v in line.split())) for s, line in zip(shapes, out.splitlines(), strict=True)]
    return run


def test_every_plan_covers_its_rows_and_chunks_and_fits(plans):
    shapes = [(f, r, c * 256, b, fu) for f, r, c, b, fu in itertools.product(NAMES, (1, 8, 15, 17, 300, 1184, 2369, 9999, 18945, 65536, 151936), range(1, 77, 3), (1, 8, 9, 24, 32), (0, 1))
              if not (fu and b > 8)]
    for p in plans(shapes):
        t = 8 if p.fused else 16
        assert p.fits and 1 <= p.grid <= SMS and p.rt <= 8 and 1 <= p.rt * p.kp <= 16
        assert p.rt * p.passes * t >= -(-p.rows // p.grid) and (p.passes - 1) * p.rt < p.tiles
        assert p.kp * p.steps >= p.chunks > p.kp * (p.steps - 1)
        assert 1 <= p.nstages <= min(8, p.fills) and p.base % 128 == 0 and p.stage % 16 == 0
        groups = (p.batch + 7) // 8
        assert p.stage == p.rt * 16 * p.kp * PITCH[p.fmt] + p.kp * groups * 4096
        assert p.base == (p.rt * p.kp * groups * 512 if p.kp > 1 else 0) and p.bytes == p.base + p.nstages * p.stage <= SMEM_OPTIN - 1024


def test_the_gpu_tests_reach_what_they_are_for(plans):
    """Every product of test_gpu_few takes this form, and between them its rings go round, rows take two passes with chunks shared by
    warps, and chunks are shared unevenly, for every number of groups."""
    got = plans([(f, r, c, b, 0) for f in NAMES for (r, c), b in itertools.product(gpu.SHAPES, gpu.BATCHES)] + [(f, *case) for f in NAMES for case in gpu.PASSES])
    assert all(p.faster for p in got)
    for groups in (1, 2, 3, 4):
        mine = [p for p in got if (p.batch + 7) // 8 == groups and not p.fused]
        for f in NAMES:
            assert any(p.fmt == f and p.chunks % p.kp and p.kp > 1 for p in mine)
        assert any(p.fills > 2 * p.nstages for p in mine) if groups == 1 else any(p.fills > p.nstages and p.kp > 1 for p in mine)
    for f, fused in itertools.product(NAMES, (0, 1)):
        assert any(p.fmt == f and p.fused == fused and p.passes > 1 and p.kp > 1 and p.fills > p.nstages for p in got)


# us of this form and of the tensor-memory form: random products at which the two are near each other
MEASURED = [
    ("q4_k", 1024, 2304, 24, 4.94, 6.51), ("q4_k", 2304, 5376, 13, 7.01, 8.82), ("q4_k", 2560, 5632, 21, 9.86, 10.75), ("q4_k", 2816, 7936, 23, 13.3, 12.47),
    ("q4_k", 3072, 3072, 10, 6.04, 8.28), ("q4_k", 7424, 3328, 15, 11.02, 11.82), ("q4_k", 10240, 3584, 14, 12.99, 13.82), ("q4_k", 13056, 4096, 26, 20.19, 18.67),
    ("q4_k", 15616, 4608, 22, 24.32, 20.64), ("q4_k", 44035, 1024, 29, 19.42, 18.84), ("q5_k", 68, 256, 10, 2.86, 3.68), ("q5_k", 68, 256, 27, 3.4, 3.87),
    ("q5_k", 306, 2560, 17, 5.06, 6.64), ("q5_k", 2048, 4608, 24, 8.02, 8.49), ("q5_k", 2560, 2560, 27, 7.61, 7.84), ("q5_k", 3328, 10496, 19, 20.08, 16.51),
    ("q5_k", 4864, 13056, 22, 31.05, 23.81), ("q5_k", 6150, 2816, 14, 8.5, 11.07), ("q5_k", 7168, 3328, 31, 13.7, 12.8), ("q5_k", 17664, 5120, 18, 30.88, 26.3),
    ("q6_k", 125, 256, 17, 3.3, 3.87), ("q6_k", 275, 9984, 7, 10.08, 9.41), ("q6_k", 512, 3328, 18, 6.15, 7.5), ("q6_k", 2402, 8704, 25, 19.17, 17.51),
    ("q6_k", 2560, 6400, 27, 15.67, 13.08), ("q6_k", 3328, 11520, 7, 21.1, 17.61), ("q6_k", 3584, 1280, 24, 5.29, 6.64), ("q6_k", 4864, 4864, 10, 12.71, 13.35),
    ("q6_k", 6912, 2816, 21, 10.7, 13.06), ("q6_k", 14685, 1280, 16, 9.58, 11.79), ("q8_0", 718, 5888, 19, 8.63, 9.5), ("q8_0", 1024, 4608, 28, 8.31, 8.63),
    ("q8_0", 1792, 4864, 10, 6.95, 8.57), ("q8_0", 2228, 6656, 10, 8.82, 11.37), ("q8_0", 2304, 6144, 31, 10.77, 10.7), ("q8_0", 3072, 3072, 11, 6.9, 8.85),
    ("q8_0", 7680, 3840, 9, 14.19, 13.96), ("q8_0", 10165, 2816, 15, 12.53, 13.55), ("q8_0", 11520, 5120, 31, 25.72, 23.54), ("q8_0", 12032, 4608, 21, 23.71, 22.16)]


def test_the_rule_picks_the_faster_form(plans):
    """1 % slower than the better form on average and nowhere 10 %."""
    lost = [math.log((few if p.faster else other) / min(few, other)) for p, (*_, few, other) in zip(plans([(FMT[f], r, c, b, 0) for f, r, c, b, *_ in MEASURED]), MEASURED)]
    assert sum(lost) / len(lost) <= 0.01 and max(lost) <= math.log(1.1)
