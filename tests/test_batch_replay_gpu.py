"""Launch groups whose step count is odd or does not go into the check
interval are replayed from graphs of their own pattern: many groups of every
pattern end bit for bit as one step per group on one block per domain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(33, 62), (64, 32), (41, 50), (75, 160), (130, 90), (5, 500), (150, 150)]


def run(lbmc, geoms, storage, cap, check, tol, **kw):
    with lbmc.Batch(geoms, tau=0.8, force=(1e-5, 2e-6), storage=storage, **kw) as b:
        res = b.run(cap, tol, check)
        return ([(r.steps, r.converged, np.float64(r.delta_u).tobytes()) for r in res],
                [b.fetch(d, lbmc.FIELD_F) for d in range(b.n)])


# (steps a group, check interval, cap, tolerance): every offset of the test in
# a group of both parities (7, 5), groups longer than the interval (9, 2),
# groups mostly without a test (3, 40), more patterns than are kept (45, 46),
# domains that stop on the way.
@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("steps,check,cap,tol", [
    (7, 5, 400, 0.0), (9, 2, 300, 0.0), (3, 40, 500, 0.0), (1, 3, 200, 0.0), (45, 46, 4300, 0.0), (7, 10, 600, 3e-6),
    (2, 7, 300, 3e-6)])
def test_patterns(lbmc, storage, steps, check, cap, tol):
    rng = np.random.default_rng(3)
    geoms = [np.where(rng.random((ly, lx)) < 0.1, rng.choice([0.3, 1.0], (ly, lx)), 0.0) for lx, ly in SIZES]
    base = run(lbmc, geoms, storage, cap, check, tol, block_threads=256, steps_per_launch=1, wide_min_nodes=1 << 30,
               wide_below=-1)
    for split in (dict(), dict(wide_min_nodes=1), dict(wide_min_nodes=1 << 30, wide_below=3)):
        got = run(lbmc, geoms, storage, cap, check, tol, block_threads=512, steps_per_launch=steps, **split)
        assert got[0] == base[0]
        for a, b in zip(got[1], base[1]):
            np.testing.assert_array_equal(a, b)
