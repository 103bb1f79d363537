"""The training kernels where a group of samples is not full and over many
steps: a batch that ends inside a warp's group of four with a network that
overflows on a zero input, and several epochs against an FP64 Adam loop."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def test_lanes_past_the_batch_count_nothing(lbmc):
    """W1 x + b1 cancels for the samples and is 1e30 without inputs, which
    W2 turns into infinity: the gradient of one to three samples is finite and
    that of the formula."""
    p = np.zeros(mo.PARAMS)
    p[mo.W1:mo.B1:mo.IN] = -1e30
    p[mo.B1:mo.W2] = 1e30
    p[mo.W2:mo.B2] = 1e10
    p[mo.B2:mo.W3] = np.linspace(-1, 1, mo.H)
    p[mo.W3:mo.B3] = 0.5
    m = lbmc.Mlp()
    m.set_params(p)
    for n in (1, 2, 3, 5):
        X = np.zeros((n, 6), np.float32)
        X[:, 0] = 1
        t = np.linspace(0.1, 0.5, n).astype(np.float32)
        g, loss = m.gradients(X, t)
        loss_ref, g_ref = mo.loss_and_grad(mo.bf16(p), X.astype(np.float64), t.astype(np.float64))
        assert np.all(np.isfinite(g)) and np.isfinite(loss)
        assert abs(loss - loss_ref) <= 1e-5 * loss_ref
        assert np.linalg.norm(g - g_ref) <= 1e-5 * np.linalg.norm(g_ref)


def test_epochs_against_an_fp64_adam_loop(lbmc):
    """One batch an epoch, so that no order of samples enters.  The history is
    the loss before each step; FP32 gradients (3e-5 of their norm) move a
    weight by a whole step only where its gradient is that small, which moves
    the loss by less than 1e-3 of itself over these steps."""
    rng = np.random.default_rng(11)
    n, epochs, lr = 500, 12, 3e-3
    X = rng.standard_normal((n, 6)).astype(np.float32)
    t = (0.5 * np.tanh(X[:, 0] - 0.5 * X[:, 1])).astype(np.float32)
    p = mo.bf16(rng.standard_normal(mo.PARAMS) * 0.3)
    m = lbmc.Mlp()
    m.set_params(p)
    hist = m.train(X, t, epochs=epochs, batch=n, lr=lr)
    master, mom, var, ref = p.copy(), np.zeros(mo.PARAMS), np.zeros(mo.PARAMS), []
    for k in range(1, epochs + 1):
        loss, g = mo.loss_and_grad(mo.bf16(master), X.astype(np.float64), t.astype(np.float64))
        ref.append(loss)
        mom = 0.9 * mom + 0.1 * g
        var = 0.999 * var + 0.001 * g * g
        master -= lr * (mom / (1 - 0.9 ** k)) / (np.sqrt(var / (1 - 0.999 ** k)) + 1e-8)
    assert ref[-1] < 0.7 * ref[0]
    np.testing.assert_allclose(hist, ref, rtol=1e-3)


@pytest.mark.parametrize("batch", [100, 1000])
def test_history_of_epochs_is_that_of_single_epochs(lbmc, batch):
    """Several batches an epoch, more than sixteen of them for 100: the call
    of three epochs starts like the call of one (the shuffle starts anew with
    each call), and its later entries keep falling."""
    rng = np.random.default_rng(5)
    X = rng.standard_normal((3300, 6)).astype(np.float32)
    t = np.tanh(X[:, 0]).astype(np.float32)
    three, one = lbmc.Mlp(seed=4), lbmc.Mlp(seed=4)
    hist = three.train(X, t, epochs=3, batch=batch, lr=2e-3)
    assert hist[0] == one.train(X, t, epochs=1, batch=batch, lr=2e-3)[0]
    assert hist[2] < hist[1] < hist[0]


def test_history_longer_than_its_buffer(lbmc):
    """One sample a batch, 131 losses counted an epoch: the buffer of 4096
    holds 31 epochs.  The first entries are those of a short call; the others
    are means of 131 squared residuals under a rate that hardly moves the
    weights, within a factor of three of each other (7 standard deviations)."""
    rng = np.random.default_rng(6)
    X = rng.standard_normal((2090, 6)).astype(np.float32)
    t = np.tanh(X[:, 0]).astype(np.float32)
    m, short = lbmc.Mlp(seed=4), lbmc.Mlp(seed=4)
    hist = m.train(X, t, epochs=64, batch=1, lr=1e-7)
    np.testing.assert_array_equal(hist[:2], short.train(X, t, epochs=2, batch=1, lr=1e-7))
    assert np.all(hist > 0.33 * hist.max())
