"""The sweep's other routes: on a caller's stream and captured in a graph
(the sweep forks to a stream of its own and joins), and the kernels that take
two planes a block, one-plane launches beside them, all bit for bit."""
import ctypes

import numpy as np
import pytest

from cases import make_case

pytestmark = pytest.mark.gpu


def large_case():
    # 150 x 143 x 141 FP32 is above the line: sweeps of eight, the last slab a remainder
    return make_case("d3q15", (150, 143, 141), collision_type=2, micro="zh", solids=0.2, seed=4)


@pytest.mark.parametrize("streaming", [0, 1])
def test_callers_stream_and_capture(lbmc, streaming):
    import torch
    case = large_case()
    lib = lbmc.library()
    ends = []
    for route in ("own", "stream", "graph"):
        with lbmc.Engine.from_case(case, storage=lbmc.F32, streaming=streaming) as e:
            if route == "own":
                e.iterate(11)
                e.iterate(11)
            else:
                stream = torch.cuda.Stream()
                lbmc.check(lib.lbmc_set_stream(e.h, ctypes.c_void_p(stream.cuda_stream)))
                if route == "stream":
                    e.iterate(11)
                    e.iterate(11)
                else:
                    e.iterate(11)
                    stream.synchronize()
                    graph = torch.cuda.CUDAGraph()
                    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
                        e.iterate(11)
                    graph.replay()
                    torch.cuda.synchronize()
                stream.synchronize()
            e.synchronize()
            assert e.step() == 22
            f = e.f()
            e.iterate(1, lbmc.STORE_MACROS | lbmc.SYNC)
            ends.append((f, e.rho(), e.u()))
            if route != "own":
                lbmc.check(lib.lbmc_set_stream(e.h, None))
    for other in ends[1:]:
        for a, b in zip(ends[0], other):
            np.testing.assert_array_equal(a, b)


# D2Q9 domains of 16 waves and more take two planes a block in every plain
# launch; a step that reduces diagnostics takes one.  (Odd and even row counts.)
@pytest.mark.parametrize("length,storage,kw", [
    ((2304, 2051, 1), "f32", dict(collision_type=1, forcing=True, partial=0.2)),
    ((2048, 1500, 1), "bf16", dict(collision_type=0, c_smag=0.1)),
    ((1536, 2049, 1), "f16sr", dict(collision_type=2, solids=0.2, macro="random")),
])
def test_two_planes_equal_one(lbmc, length, storage, kw):
    case = make_case("d2q9", length, seed=6, **kw)
    ends = []
    for flags in (0, lbmc.REDUCE_DIAG):
        with lbmc.Engine.from_case(case, storage=lbmc.STORAGE_IDS[storage], streaming=lbmc.STREAM_AA) as e:
            for _ in range(5):
                e.iterate(1, flags)
            ends.append(e.f())
    np.testing.assert_array_equal(*ends)
