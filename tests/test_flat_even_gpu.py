"""The plain AA layout's even step runs over the node index: sizes below, at
and past a block and a warp, rows shorter than a warp and rows that blocks
cut anywhere, with per-node inputs (boundaries, forces, porosity) that would
show a wrong node, against the shift layout bit for bit."""
import numpy as np
import pytest

from cases import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,length", [
    ("d3q15", (1, 1, 1)), ("d3q15", (63, 1, 1)), ("d3q15", (5, 7, 9)), ("d3q15", (65, 3, 2)), ("d3q15", (31, 2, 33)),
    ("d3q15", (3, 50, 4)), ("d3q15", (100, 9, 7)), ("d2q9", (101, 203, 1)), ("d2q9", (7, 2999, 1))])
@pytest.mark.parametrize("storage", ["f32", "f16sr"])
def test_even_step_over_nodes(lbmc, lattice, length, storage):
    case = make_case(lattice, length, collision_type=1, forcing=True, solids=0.15, partial=0.2, macro="random", seed=8)
    ends = []
    for streaming in (lbmc.STREAM_AA, lbmc.STREAM_SHIFT):
        with lbmc.Engine.from_case(case, storage=lbmc.STORAGE_IDS[storage], streaming=streaming,
                                   kernel=lbmc.KERNEL_DIRECT) as e:
            f = []
            for _ in range(3):
                e.iterate(1, 0)
                f.append(e.f())
            e.iterate(2, lbmc.STORE_MACROS | lbmc.SYNC)
            ends.append((f, e.rho(), e.u()))
    for a, b in zip(ends[0][0], ends[1][0]):
        np.testing.assert_array_equal(a, b)
    np.testing.assert_array_equal(ends[0][1], ends[1][1])
    np.testing.assert_array_equal(ends[0][2], ends[1][2])
