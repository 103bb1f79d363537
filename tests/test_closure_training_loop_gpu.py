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
