"""The network's gradient and training steps at the edges of the records' tiles (32 to
a block, 296 blocks a grid) against the same network in FP64.  Each parameter's gradient
is a sum over the records in FP32: with up to n terms added in tiles of 32, blocks and
blocks of blocks, and activations rounded to FP32, the relative L2 error stays within a
few hundred roundings of 2^-24 (6e-8): 2e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def records(n, seed):
    rng = np.random.default_rng(seed)
    G = rng.uniform(0.2, 2.0, (n, 8, 4))
    T = np.einsum("nmj,nj->nm", G, rng.dirichlet(np.ones(4), n)) * (1 + 0.05 * rng.standard_normal((n, 8)))
    return np.concatenate([rng.standard_normal((n, 5)), G.reshape(n, 32), T], axis=1).astype(np.float32)


def grad64(p, r):
    p, r = p.astype(np.float64), r.astype(np.float64)
    W1, b1, W2, b2, W3, b3 = np.split(p, np.cumsum([160, 32, 1024, 32, 128]))
    W1, W2, W3 = W1.reshape(32, 5), W2.reshape(32, 32), W3.reshape(4, 32)
    x, G, T = r[:, :5], r[:, 5:37].reshape(-1, 8, 4), r[:, 37:]
    h1 = np.tanh(x @ W1.T + b1)
    h2 = np.tanh(h1 @ W2.T + b2)
    z = np.exp(h2 @ W3.T + b3)
    w = z / z.sum(1, keepdims=True)
    e = (np.einsum("nmj,nj->nm", G, w) - T) / T
    dw = np.einsum("nm,nmj->nj", e / (4 * T), G)
    dz = w * (dw - (w * dw).sum(1, keepdims=True))
    d2 = dz @ W3 * (1 - h2 * h2)
    d1 = d2 @ W2 * (1 - h1 * h1)
    return float((e * e).mean(1).sum()), np.concatenate(
        [(d1.T @ x).ravel(), d1.sum(0), (d2.T @ h1).ravel(), d2.sum(0), (dz.T @ h2).ravel(), dz.sum(0)])


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 4096, 296 * 32, 296 * 32 + 1, 20011])
def test_gradient_tiles(n):
    from hawassi_c_b200 import learned
    mlp, r = learned.MLP(seed=3), records(n, n)
    loss, g = mlp.grad(r)
    l64, g64 = grad64(mlp.params(), r)
    assert abs(loss - l64) <= 2e-5 * l64
    assert np.linalg.norm(g - g64) <= 2e-5 * np.linalg.norm(g64)


def test_training_equals_its_steps():
    """A call of several epochs over a ragged last minibatch ends where one call per
    epoch ends (the same kernels in the same order), and its losses are the epochs'."""
    from hawassi_c_b200 import learned
    r = records(1000, 5)
    a, b = learned.MLP(seed=1), learned.MLP(seed=1)
    la = a.train(r, epochs=3, batch=300, lr=1e-3)
    lb = np.concatenate([b.train(r, epochs=1, batch=300, lr=1e-3) for _ in range(3)])
    assert np.array_equal(la, lb) and np.array_equal(a.params(), b.params())
    assert la[2] < la[0]
