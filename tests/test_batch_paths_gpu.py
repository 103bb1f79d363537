"""The routes of the batched sweep end bit for bit the same: launches that
are replayed and launches that are not (odd step counts, a check interval
that does not divide them, the step cap inside a launch), domains on the
edges of the default split, and domains that stop in the middle of a launch.
The base of the comparison is one block per domain, one step per launch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(16, 24), (33, 62), (64, 32), (41, 50), (75, 160), (130, 90), (31, 129), (5, 500), (1, 40), (300, 310)]


def domains():
    import workloads
    rng = np.random.default_rng(7)
    return [workloads.circle_domain(lx, ly, rng.uniform(0.2, 0.4), rng, tau=0.8) if min(lx, ly) > 12
            else np.where(rng.random((ly, lx)) < 0.1, 0.3, 0.0) for lx, ly in SIZES]


def run(lbmc, geoms, storage, cap, check, tol, **kw):
    with lbmc.Batch(geoms, tau=0.8, force=(1e-5, 2e-6), storage=storage, **kw) as b:
        res = b.run(cap, tol, check)
        return ([(r.steps, r.converged, np.float64(r.delta_u).tobytes()) for r in res],
                [b.fetch(d, lbmc.FIELD_F) for d in range(b.n)])


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("steps,check,cap,tol", [
    (7, 5, 33, 0.0), (6, 3, 31, 0.0), (10, 5, 40, 0.0), (1, 1, 3, 0.0), (4, 2, 2, 0.0), (20, 10, 205, 2e-6),
    (0, 5, 97, 0.0), (0, 10, 400, 2e-6)])
def test_routes_agree(lbmc, storage, steps, check, cap, tol):
    geoms = domains()
    base = run(lbmc, geoms, storage, cap, check, tol, block_threads=256, steps_per_launch=1, wide_min_nodes=1 << 30,
               wide_below=-1)
    assert any(s == cap for s, _, _ in base[0])
    threads = 512 if steps else 0
    for split in (dict(), dict(wide_min_nodes=1), dict(wide_min_nodes=1 << 30, wide_below=-1)):
        got = run(lbmc, geoms, storage, cap, check, tol, block_threads=threads, steps_per_launch=steps, **split)
        assert got[0] == base[0]
        for a, b in zip(got[1], base[1]):
            np.testing.assert_array_equal(a, b)
