"""The stage ring of the K-quant mma kernel, on the CPU: every plan the host arithmetic makes is run through a model of the
kernel's barriers in which one participant at a time is slower than all others."""
import itertools
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
UNIT = {"q4_k": 144, "q5_k": 176, "q6_k": 210}
SMEM_OPTIN, SMS = 232448, 148      # of a B200

PROGRAM = r"""
#include "mma_plan.h"
#include <cstdio>
using namespace orome;
int main()
{
    unsigned q6, unit, units, nvec, share, swiglu, two, kb;
    size_t xq;
    while (scanf("%u %u %u %u %u %u %u %zu %u", &q6, &unit, &units, &nvec, &share, &swiglu, &two, &xq, &kb) == 9) {
        MmaRingShape in{q6 != 0, unit, units, nvec, share, swiglu != 0, two != 0, xq, %d, kb};
        MmaRing r = {};
        const int fit = mma_plan_ring(in, r);
        printf("%%d %%u %%u %%u %%u %%u %%u\n", fit, r.nstages, r.ngroups, r.nwarps, r.nchunks, r.kc, r.stage_base + r.nstages * r.stage_stride);
    }
}
""".replace("%d, kb}", f"{SMEM_OPTIN}, kb}}").replace("%%", "%")


@pytest.fixture(scope="module")
def plans(tmp_path_factory):
    """plan(list of shapes) -> list of (fit, nstages, ngroups, nwarps, nchunks, kc, bytes)"""
    d = tmp_path_factory.mktemp("ring")
    (d / "plan.cpp").write_text(PROGRAM)
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "orome_b200", "csrc"), "-o", str(d / "plan"), str(d / "plan.cpp")])

    def run(shapes):
        text = "\n".join(" ".join(str(v) for v in s) for s in shapes)
        out = subprocess.run([str(d / "plan")], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(int(v) for v in line.split()) for line in out.splitlines()]
    return run


def shape(fmt, in_dim, rows, kb=0, swiglu=False, fused=False, nvec=0):
    share = -(-rows // min(SMS, -(-rows // 16)))
    return (int(fmt == "q6_k"), UNIT[fmt], in_dim // 256, nvec, share, int(swiglu), 0, 1152 if fused else 864, kb)


def stale_read(nslots, ngroups, nwarps, nprod, stages=40):
    """True if some schedule of the model lets a warp read a slot that does not hold the stage it is due.  Barriers as the kernel
    uses them: a wait for parity p passes when the barrier's current phase has the other parity; `full` completes when a copy
    lands, `empty` when the warps of the group that used the slot have arrived."""
    guarded = ngroups == 2 and nslots % 2 == 1
    for slow in [("p", p) for p in range(nprod)] + [("c", s) for s in range(nslots)] + [("w", g, w) for g in range(ngroups) for w in range(nwarps)]:
        full, empty, arrived, content, flying = [0] * nslots, [0] * nslots, [0] * nslots, [None] * nslots, [None] * nslots
        todo = {("p", p): [i for i in range(stages) if i % nslots % nprod == p] for p in range(nprod)}
        todo.update({("w", g, w): list(range(g, stages, ngroups)) for g in range(ngroups) for w in range(nwarps)})
        actors = [a for a in list(todo) + [("c", s) for s in range(nslots)] if a != slow] + [slow]

        def step(a):
            if a[0] == "c":
                s = a[1]
                if flying[s] is None:
                    return False
                content[s], flying[s] = flying[s], None
                full[s] += 1
                return True
            if not todo[a]:
                return False
            i = todo[a][0]
            s, k = i % nslots, i // nslots
            if a[0] == "p":
                if k and empty[s] & 1 == (k - 1) & 1:
                    return False
                if flying[s] is not None:
                    return None
                flying[s] = i
            else:
                if guarded and k and empty[s] & 1 == (k - 1) & 1:
                    return False
                if full[s] & 1 == k & 1:
                    return False
                if content[s] != i or flying[s] is not None:
                    return None
                arrived[s] += 1
                if arrived[s] == nwarps:
                    arrived[s] = 0
                    empty[s] += 1
            todo[a].pop(0)
            return True
        while True:
            for a in actors:               # the slow one only moves when nobody else can
                moved = step(a)
                if moved is None:
                    return True
                if moved:
                    break
            else:
                break
        assert not any(todo.values()), "the model is stuck"
    return False


def test_the_model_tells_rings_apart():
    assert stale_read(9, 2, 2, 2) and stale_read(3, 2, 2, 2)       # two producers on an odd ring
    assert not stale_read(9, 2, 2, 1) and not stale_read(8, 2, 2, 2) and not stale_read(3, 1, 2, 2)
    assert stale_read(4, 3, 2, 1)                                   # slots that change hands between three groups


def test_every_plan_keeps_its_slots_apart(plans):
    shapes = []
    for fmt, swiglu, fused, kb in itertools.product(UNIT, (False, True), (False, True), (0, 8, 12, 16, 20, 24, 30, 40, 64, 100)):
        if fmt == "q6_k" and swiglu:
            continue
        for in_dim, rows in itertools.product(range(256, 25601, 256), (16, 1000, 4096, 17408, 151936)):
            shapes.append(shape(fmt, in_dim, rows, kb, swiglu, fused))
    shapes += [shape(fmt, u * 256, 2048, 0, False, False, nvec) for fmt in ("q4_k", "q5_k") for u in range(1, 9) for nvec in range(1, 9)]
    got = plans(shapes)
    assert len(got) == len(shapes)
    rings, odd_q6, odd = set(), 0, 0
    for s, (fit, nstages, ngroups, nwarps, nchunks, kc, used) in zip(shapes, got):
        if fit == 2:
            continue
        assert nstages >= 1 and ngroups >= 1 and nwarps * ngroups <= 16 and used <= SMEM_OPTIN and kc * nchunks >= s[2]
        if nstages % ngroups:
            odd += 1
            odd_q6 += s[0]
        rings.add((nstages, ngroups, min(nwarps, 2), 2 if s[0] else 1))
    assert odd > 0 and odd_q6 == 0                                  # the guarded ring is used, but not by Q6_K
    assert (3, 2, 2, 1) in rings or (5, 2, 2, 1) in rings
    for r in sorted(rings):
        assert not stale_read(*r), r


def test_plans_the_gpu_tests_rely_on(plans):
    """4096 x 17408 Q6_K in 20-KiB stages fills nine slots, of which two groups take eight; the fused Q6_K product of that width in
    40-KiB stages three, of which they take two."""
    wide, fused = plans([shape("q6_k", 17408, 4096, 20), shape("q6_k", 17408, 5120, 40, False, True)])
    assert wide[1:3] == (8, 2) and fused[1:3] == (2, 2)
