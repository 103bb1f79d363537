"""Which domains are swept (csrc/sweep.h): the measured sides of the rule for
long rows and 2-byte storage, and on the GPU a domain of few long rows, whose
steps in one call may not be slower than one step a call."""
import subprocess
import time
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent

PLAIN, SMAG, PARTIAL, FORCED, PARTIAL_FORCED = (0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1), (0, 1, 1)
# (dim, element bytes, tiled, options, nodes of a plane, planes), swept
RULE = [
    ((2, 4, 1, PLAIN, 4096, 4096), True), ((2, 4, 1, PLAIN, 299968, 69), True), ((2, 4, 1, PLAIN, 600000, 34), False),
    ((2, 4, 0, PLAIN, 100000, 209), True), ((2, 4, 0, PLAIN, 150000, 139), False),
    ((2, 4, 0, SMAG, 150000, 139), False), ((2, 4, 0, PARTIAL_FORCED, 300000, 70), True),
    ((2, 4, 0, PLAIN, 600000, 34), False), ((2, 4, 0, PARTIAL_FORCED, 600000, 34), False),
    ((2, 8, 0, PLAIN, 300000, 69), True), ((2, 8, 1, PLAIN, 150016, 139), True),
    ((2, 2, 1, PLAIN, 4096, 4096), True), ((2, 2, 1, PLAIN, 200000, 105), True), ((2, 2, 1, PLAIN, 299968, 69), False),
    ((2, 2, 0, PLAIN, 4096, 4096), False), ((2, 2, 0, PLAIN, 6000, 3495), False), ((2, 2, 0, FORCED, 100000, 180), False),
    ((2, 2, 0, PARTIAL, 100000, 180), False), ((2, 2, 0, SMAG, 4000, 4000), True), ((2, 2, 0, SMAG, 150000, 140), False),
    ((2, 2, 0, PARTIAL_FORCED, 100000, 180), True),
    ((3, 4, 1, PLAIN, 256 * 256, 256), True), ((3, 2, 0, PLAIN, 250 * 250, 160), True),
    ((3, 4, 0, PLAIN, 640 * 640, 40), True), ((3, 8, 0, PLAIN, 640 * 640, 40), False),
]


def test_rule(tmp_path):
    exe = tmp_path / "sweep_rule"
    subprocess.run(["g++", "-std=c++17", "-O2", str(HERE / "sweep_rule.cpp"), "-o", str(exe)], check=True)
    lines = [" ".join(map(str, (dim, elem, tiled, *opt, row, planes, 9 if dim == 2 else 15)))
             for (dim, elem, tiled, opt, row, planes), _ in RULE]
    run = subprocess.run([str(exe)], input="\n".join(lines), capture_output=True, text=True, check=True)
    depths = [int(v) for v in run.stdout.split()]
    assert [d > 1 for d in depths] == [swept for _, swept in RULE], depths


# 34 rows of 600000 nodes: a call of 40 steps took 1.41 (tiled) and 1.22 times
# as long as 40 calls of one step; the limit leaves an eighth for noise.
@pytest.mark.gpu
@pytest.mark.parametrize("streaming", ["aa", "shift"])
def test_long_rows(lbmc, streaming):
    lx, ly, steps = 600000, 34, 40
    cfg = lbmc.make_config("d2q9", (lx, ly, 1), tau=0.7,
                           streaming=lbmc.STREAM_AA if streaming == "aa" else lbmc.STREAM_SHIFT)
    dom, keep = lbmc.make_domain(lx * ly, 2, 9)

    def best(call):
        call()
        times = []
        for _ in range(5):
            t = time.perf_counter()
            call()
            times.append(time.perf_counter() - t)
        return min(times)

    with lbmc.Engine(cfg, dom) as e:
        def singles():
            for _ in range(steps):
                e.iterate(1)
            e.synchronize()
        assert best(lambda: e.iterate(steps, lbmc.SYNC)) <= 1.125 * best(singles)
