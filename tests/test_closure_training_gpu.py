"""The training kernels at the sizes where their split can go wrong: batches
below, at and past a warp's group of samples, a block's pass and the chip's
one pass per SM, against the FP64 gradient; one Adam step against its
formula; and training that is the same bits each time."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def network(lbmc, seed=3):
    rng = np.random.default_rng(seed)
    m = lbmc.Mlp(seed=seed)
    m.set_params(rng.standard_normal(mo.PARAMS) * 0.3)
    m.set_normalization(np.linspace(-0.5, 0.5, 6), np.linspace(0.7, 1.5, 6), target_scale=0.5)
    return m, rng


# FP32 sums in the kernel: about 100 terms in a row per sample (6 + 32 + 32 +
# 32 and the activations), 100 * 2^-24 = 6e-6 of the magnitudes that are
# added; the residual y - t and the sum over the samples cancel part of them,
# by less than a factor of 5 for these random targets.
TOL = 3e-5


@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 32, 33, 63, 148 * 32 - 1, 148 * 32 + 1, 20001])
def test_gradient_at_the_edges_of_the_split(lbmc, n):
    m, rng = network(lbmc)
    X = rng.standard_normal((n, 6)).astype(np.float32)
    t = (0.5 * rng.standard_normal(n)).astype(np.float32)
    g, loss = m.gradients(X, t)
    mean, std = (a.astype(np.float64) for a in m._norm[:2])
    loss_ref, g_ref = mo.loss_and_grad(m.params().astype(np.float64), (X - mean) / std, t / 0.5)
    assert abs(loss - loss_ref) <= TOL * loss_ref
    assert np.linalg.norm(g - g_ref) <= TOL * np.linalg.norm(g_ref)


def test_first_adam_step(lbmc):
    """From zero moments Adam's first step is p - lr g / (|g| + eps); the
    weights come back rounded to BF16: equal to the formula's value rounded
    the same way, wherever FP32 rounding (1e-6) cannot reach a boundary."""
    m, rng = network(lbmc)
    X = rng.standard_normal((1000, 6)).astype(np.float32)
    t = rng.standard_normal(1000).astype(np.float32)
    p0 = m.params().astype(np.float64)
    m.set_params(p0)
    g, loss = m.gradients(X, t)
    hist = m.train(X, t, epochs=1, batch=1000, lr=1e-2)
    step = 1e-2 * g / (np.abs(g) + 1e-8)
    sure = np.abs(g) > 1e-4 * np.abs(g).max()  # where the order of the sum cannot turn the sign
    expected = p0 - step
    sure &= mo.bf16(expected - 1e-6) == mo.bf16(expected + 1e-6)
    assert sure.mean() > 0.9
    np.testing.assert_array_equal(m.params().astype(np.float64)[sure], mo.bf16(expected)[sure])
    assert abs(hist[0] - loss) <= TOL * loss


@pytest.mark.parametrize("batch", [1, 7, 100, 4096])
def test_training_repeats_bit_for_bit(lbmc, batch):
    n = 40 * batch + batch // 2 if batch < 4096 else 10000
    ends = []
    for _ in range(2):
        m, rng = network(lbmc, seed=5)
        X = rng.standard_normal((n, 6)).astype(np.float32)
        t = np.tanh(X[:, 0]) * 0.5
        hist = m.train(X, t, epochs=3, batch=batch, lr=2e-3)
        ends.append((hist, m.params()))
    assert np.all(np.isfinite(ends[0][1])) and ends[0][0][-1] < 2 * ends[0][0][0]
    np.testing.assert_array_equal(ends[0][0], ends[1][0])
    np.testing.assert_array_equal(ends[0][1], ends[1][1])


def test_batch_larger_than_the_set_takes_no_step(lbmc):
    m, rng = network(lbmc)
    p0 = m.params()
    X = rng.standard_normal((10, 6)).astype(np.float32)
    hist = m.train(X, X[:, 0], epochs=2, batch=11, lr=1e-2)
    np.testing.assert_array_equal(m.params(), p0)
    np.testing.assert_array_equal(hist, 0)
