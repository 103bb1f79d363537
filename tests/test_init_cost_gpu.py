"""lbmc_init and lbmc_destroy of a small domain cost what their own device
allocation and stream cost, not more: a program that makes a handle per
parameter set makes and drops them one after the other, with none alive in
between.  Measured in a process of its own, against the same CUDA calls made
there through the runtime."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

PROGRAM = """
import ctypes, sys, time
sys.path.insert(0, sys.argv[1])
import lbmc
import torch  # loads the runtime
rt = ctypes.CDLL("libcudart.so.12")

def best(call, n=25):
    times = []
    for _ in range(n):
        t = time.perf_counter()
        call()
        times.append(time.perf_counter() - t)
    return min(times)

def resources():
    p, s = ctypes.c_void_p(), ctypes.c_void_p()
    assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(1 << 20)) == 0
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(s), 1) == 0
    rt.cudaStreamDestroy(s)
    rt.cudaFree(p)

def handle():
    cfg = lbmc.make_config("d2q9", (128, 64, 1), tau=0.8)
    dom, keep = lbmc.make_domain(128 * 64, 2, 9)
    lbmc.Engine(cfg, dom).close()

resources(), handle()
print(best(handle), best(resources))
"""


# The allocation with its release and the stream take ~0.75 ms, the uploads of
# a few KB and the launches as much again at most: three times is the limit.
# (A page-locked block mapped and unmapped with each handle took 2.3-5 ms.)
def test_init_and_destroy(lbmc):
    run = subprocess.run([sys.executable, "-c", PROGRAM, str(ROOT / "lbm-c_b200")], capture_output=True, text=True,
                         timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]
    handle, resources = (float(v) for v in run.stdout.split())
    assert handle <= 3 * resources, f"{handle * 1e3:.2f} ms against {resources * 1e3:.2f} ms"
