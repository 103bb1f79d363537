"""FP64 steps of a small 2-D domain do not depend on how they are grouped:
many in one launch out of shared memory and the direct kernel's single steps
end bit for bit the same, in every collision, force and porosity variant, with
boundaries and with the reference's own quirks, in both layouts."""
import numpy as np
import pytest

from cases import make_case

pytestmark = pytest.mark.gpu

OPTIONS = [dict(collision_type=0), dict(collision_type=0, forcing=True), dict(collision_type=0, macro="random"),
           dict(collision_type=0, forcing=True, uniform_force=True, solids=0.2, micro="zh"),
           dict(collision_type=1, partial=0.3), dict(collision_type=1, partial=0.3, forcing=True, macro="random"),
           dict(collision_type=0, c_smag=0.12), dict(collision_type=0, c_smag=0.12, forcing=True, macro="random"),
           dict(collision_type=1, c_smag=0.1, partial=0.3), dict(collision_type=1, c_smag=0.1, partial=0.3, forcing=True),
           dict(collision_type=2, micro="zh", solids=0.1), dict(collision_type=2, forcing=True),
           dict(collision_type=3, partial=0.3), dict(collision_type=3, partial=0.3, forcing=True),
           dict(collision_type=2, mrt_conserved=1.1), dict(collision_type=2, mrt_conserved=1.1, forcing=True, micro="zh"),
           dict(collision_type=3, mrt_conserved=1.1, partial=0.3),
           dict(collision_type=3, mrt_conserved=1.1, partial=0.3, forcing=True, macro="random"),
           dict(collision_type=2, micro="zh", compat=0xF), dict(collision_type=3, partial=0.3, forcing=True, compat=0xF)]


@pytest.mark.parametrize("streaming", [0, 1])
@pytest.mark.parametrize("opt", range(len(OPTIONS)))
@pytest.mark.parametrize("length", [(41, 23, 1), (128, 120, 1)])
def test_grouping(lbmc, length, opt, streaming):
    case = make_case("d2q9", length, seed=3 + opt, **OPTIONS[opt])
    ends = []
    for kernel, groups in ((lbmc.KERNEL_AUTO, (7, 33, 60)), (lbmc.KERNEL_AUTO, (1,) * 5 + (95,)),
                           (lbmc.KERNEL_DIRECT, (100,))):
        with lbmc.Engine.from_case(case, storage=lbmc.F64, streaming=streaming, kernel=kernel) as e:
            for n in groups:
                e.iterate(n)
            f = e.f()
            e.iterate(1, lbmc.STORE_MACROS | lbmc.SYNC)
            ends.append((f, e.rho(), e.u()))
    assert np.all(np.isfinite(ends[0][0]))
    for other in ends[1:]:
        for a, b in zip(ends[0], other):
            np.testing.assert_array_equal(a, b)
