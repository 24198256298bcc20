"""The closure's training kernels at the sizes where their split can go wrong: samples come
in groups of 4 per warp, 64 per CTA, at most one CTA per SM."""
import numpy as np
import pytest

from aerosim_b200 import sgs
from oracle import mlp as omlp

pytestmark = pytest.mark.gpu


def _data(n, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(0.0, 1.0, (n, 8)).astype(np.float32)
    Y = np.abs(X[:, 0] * X[:, 1] + 0.5 * X[:, 7] + 0.3 * rng.normal(size=n)).astype(np.float32)
    return X, Y


# FP32 sums of at most 32 products and of the samples' contributions: errors of some tens
# of half-ulps (6e-8) on terms whose sizes add up to a few times the largest component
@pytest.mark.parametrize("n", [1, 3, 4, 5, 63, 64, 65, 9471, 9473])
def test_gradient_at_group_and_cta_edges(n):
    X, Y = _data(n, n)
    p = sgs.init_params(3)
    g, loss = sgs.gradients(p, X, Y)
    loss_o, g_o = omlp.loss_and_grad(p.astype(np.float64), X, Y)
    assert abs(loss - loss_o) <= 1e-5 * loss_o + 1e-12
    assert np.abs(g - g_o).max() <= 1e-4 * np.abs(g_o).max()
    g2, loss2 = sgs.gradients(p, X, Y)
    assert np.array_equal(g, g2) and loss == loss2  # fixed summation order


def _rows(seed, it, batch, n):
    m = (1 << 64) - 1
    out = []
    for i in range(batch):
        z = (seed + 0x9E3779B97F4A7C15 * (it * 1000003 + i + 1)) & m
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
        out.append((z ^ (z >> 31)) % n)
    return np.array(out)


@pytest.mark.parametrize("n,batch", [(1, 1), (2, 7), (3, 64), (1000, 65), (65537, 130)])
def test_minibatch_rows_and_adam_steps(n, batch):
    """The mini-batches are the hashed rows and the parameters follow Adam: the loss of each
    iteration against float64 Adam on the same rows."""
    X, Y = _data(n, 17)
    p0, iters, lr = sgs.init_params(4), 3, 1e-3
    p, curve = sgs.train(p0, X, Y, iters=iters, batch=batch, lr=lr, seed=11)
    q = p0.astype(np.float64)
    m, v = np.zeros_like(q), np.zeros_like(q)
    for it in range(iters):
        r = _rows(11, it, batch, n)
        loss, g = omlp.loss_and_grad(q, X[r], Y[r])
        # the parameters of iteration it differ by at most it sign flips of lr on gradients
        # that are zero to rounding, which moves the loss by far less than its gradient does
        assert abs(curve[it] - loss) <= 1e-5 * loss + 1e-4 * it * loss + 1e-9, it
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        q = q - lr * (m / (1 - 0.9 ** (it + 1))) / (np.sqrt(v / (1 - 0.999 ** (it + 1))) + 1e-8)
    assert np.isfinite(p).all() and np.abs(p - p0).max() <= 1.01 * iters * lr
