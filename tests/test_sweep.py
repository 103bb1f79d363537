"""Sweeps of several steps through L2 (csrc/sweep.h): the order of the
launches on the CPU, and on the GPU domains larger than the sweep's limit
against the same handle stepped one step per call, which never sweeps."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from cases import make_case

HERE = Path(__file__).resolve().parent


def test_order_of_a_sweep(tmp_path):
    exe = tmp_path / "sweep_check"
    subprocess.run(["g++", "-std=c++17", "-O2", str(HERE / "sweep_check.cpp"), "-o", str(exe)], check=True)
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0 and run.stdout.startswith("OK"), run.stdout


# Odd sizes, the last slab a remainder; the steps are one sweep of eight, one
# of five and the step that stores.  Nothing may differ in a bit.
@pytest.mark.gpu
@pytest.mark.parametrize("lattice,length,storage,streaming,kw", [
    ("d3q15", (121, 127, 123), "f64", "shift", dict(collision_type=2, micro="zh", solids=0.2)),
    ("d3q15", (128, 113, 119), "f64", "aa", dict(collision_type=0, forcing=True, c_smag=0.1)),
    ("d3q15", (150, 143, 141), "f32", "aa", dict(collision_type=2, micro="zh", solids=0.2)),
    ("d3q15", (192, 131, 113), "f32", "aa", dict(collision_type=3, forcing=True, solids=0.2)),
    ("d3q15", (215, 205, 203), "f16sr", "shift", dict(collision_type=0, forcing=True)),
    ("d2q9", (2311, 2011, 1), "f32", "aa", dict(collision_type=1, forcing=True, solids=0.2, partial=0.2)),
    ("d2q9", (1601, 1503, 1), "f64", "shift", dict(collision_type=0, macro="random")),
    # two planes a block: odd planes, a slab and a launch that end on half a block
    ("d3q15", (256, 193, 181), "bf16", "aa", dict(collision_type=2, micro="zh", solids=0.2)),
    ("d3q15", (192, 219, 217), "f16", "aa", dict(collision_type=0, c_smag=0.1)),
    ("d2q9", (2304, 2051, 1), "f32", "aa", dict(collision_type=1, forcing=True, partial=0.2)),
])
def test_sweep_equals_single_steps(lbmc, lattice, length, storage, streaming, kw):
    case = make_case(lattice, length, seed=4, **kw)
    st = lbmc.STREAM_AA if streaming == "aa" else lbmc.STREAM_SHIFT
    flags = lbmc.STORE_MACROS | lbmc.REDUCE_DIAG | lbmc.SYNC
    ends = []
    for whole in (True, False):
        with lbmc.Engine.from_case(case, storage=lbmc.STORAGE_IDS[storage], streaming=st) as e:
            if whole:
                e.iterate(14, flags)
            else:
                for _ in range(13):
                    e.iterate(1)
                e.iterate(1, flags)
            d = e.diag()
            ends.append((e.rho(), e.u(), e.f()[-3:], d.mass, d.kinetic_energy))
    for a, b in zip(*ends):
        np.testing.assert_array_equal(a, b)
