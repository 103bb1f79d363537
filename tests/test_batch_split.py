"""Which batched domains stay in shared memory (csrc/batch_split.h): the
measured sides on the CPU, and on the GPU a batch of as many equal domains as
the chip has SMs, which may not be slower than with every one of them kept in
shared memory."""
import subprocess
import time
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent

# (nodes of the domains that do not fit, groups of (count, nodes)), how many go wide on 148 SMs
SPLITS = [
    ((0, [(148, 10000)]), 0), ((0, [(100, 2304)]), 0), ((0, [(1000, 1024)]), 0), ((0, [(3000, 256)]), 0),
    ((0, [(1000, 8100)]), 0), ((0, [(1, 256)]), 0), ((0, []), 0),
    ((0, [(1, 10000)]), 1), ((0, [(8, 4096)]), 8), ((0, [(1, 10000), (200, 1024)]), 1),
    # one more round for a few: these go
    ((0, [(160, 10000)]), 12), ((0, [(300, 10000)]), 4),
    # beside work that outlasts them they stay
    ((10 ** 7, [(20, 12000)]), 0),
    # beside a few larger domains: the share's line, unless it costs the SMs their domains
    ((10 ** 6, [(5, 12000), (10, 6500), (10, 3000)]), 15), ((40000, [(148, 10000)]), 0),
]


def test_split(tmp_path):
    exe = tmp_path / "batch_split"
    subprocess.run(["g++", "-std=c++17", "-O2", str(HERE / "batch_split.cpp"), "-o", str(exe)], check=True)
    lines = []
    for (rest, groups), _ in SPLITS:
        share = max(2048, 3 * (rest + sum(count * nodes for count, nodes in groups)) // (4 * 148))
        lines.append(" ".join(map(str, [rest, share, 148, *(v for g in groups for v in g)])))
    run = subprocess.run([str(exe)], input="\n".join(lines), capture_output=True, text=True, check=True)
    assert [int(v) for v in run.stdout.split()] == [n for _, n in SPLITS]


# All of them over every SM: 1.75 (100x100) and 1.54 times as long.
@pytest.mark.gpu
@pytest.mark.parametrize("count,side", [(148, 100), (100, 48)])
def test_equal_domains(lbmc, count, side):
    geometry = np.zeros((side, side))

    def run(**kw):
        best = np.inf
        for _ in range(6):
            with lbmc.Batch([geometry] * count, tau=0.9, storage="f16", block_threads=512, steps_per_launch=100, **kw) as b:
                t = time.perf_counter()
                b.run(1000, 0.0, 100)
                best = min(best, time.perf_counter() - t)
        return best

    assert run() <= 1.25 * run(wide_min_nodes=1 << 30, wide_below=-1)
