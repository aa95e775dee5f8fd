"""The forecaster's loss gradient and its training round every value as plain FP32 arithmetic does, sample by
sample: products before they are added, units in ascending order, 32 samples in the pairs of a butterfly, four
such sums after one another to a block sum, block sums after one another. So a hidden unit is on or off as in that
arithmetic, and the weights after a step are equal bit for bit."""
import numpy as np
import pytest

from dacti_b200.forecast import Mlp
from test_gpu_forecast_train import _order

pytestmark = pytest.mark.gpu
F, H = np.float32, 64


def _net(n_in, seed):
    rng = np.random.default_rng(seed)
    net = Mlp(n_in, seed=seed)
    net.params = (net.params + F(0.05) * rng.standard_normal(net.n_params).astype(F)).astype(F)
    return net, rng


def _unpack(w, n_in):
    cut = np.cumsum([H * n_in, H, H * H, H, H])
    w1, b1, w2, b2, w3, b3 = np.split(w, cut)
    return w1.reshape(H, n_in), b1, w2.reshape(H, H), b2, w3, b3


def _one_sample(w, x, dz):
    """The gradient of one sample from dl/dz, one rounding per operation (numpy does not contract)."""
    w1, b1, w2, b2, w3, _ = _unpack(w, x.size)
    a1, a2, d1 = b1.copy(), b2.copy(), np.zeros(H, F)
    for i in range(x.size):
        a1 += w1[:, i] * x[i]
    a1 = np.maximum(a1, F(0))
    for j in range(H):
        a2 += w2[:, j] * a1[j]
    a2 = np.maximum(a2, F(0))
    d2 = np.where(a2 > 0, dz * w3, F(0))
    for k in range(H):
        d1 += w2[k] * d2[k]
    d1 = np.where(a1 > 0, d1, F(0))
    return np.concatenate([np.outer(d1, x).ravel(), d1, np.outer(d2, a1).ravel(), d2, dz * a2, [dz]]).astype(F)


def _tile(g):
    """The sum of 32 rows: those 16 apart first, then 8, 4, 2, 1."""
    h = 16
    while h:
        g = g[:h] + g[h:2 * h]
        h //= 2
    return g[0]


def _block_sum(grads):
    """Tiles of 32 samples (missing ones zero) after one another."""
    s = np.zeros(grads.shape[1], F)
    for first in range(0, len(grads), 32):
        t = np.zeros((32, grads.shape[1]), F)
        t[:len(grads[first:first + 32])] = grads[first:first + 32]
        s = s + _tile(t)
    return s


@pytest.mark.parametrize("n_in", [1, 15, 20, 32])
def test_gradient_of_one_sample(n_in):
    net, rng = _net(n_in, 3)
    w = net.params
    for _ in range(8):
        x = rng.standard_normal(n_in).astype(F)
        _, g = net.loss_grad(x, [1.0], pos_weight=2.5)
        assert np.array_equal(g, _one_sample(w, x, g[-1]))
    net.close()


def test_logit_sums_in_the_units_order():
    """A running sum that loses the units between two large opposite ones: 7 + 1 units of 0.02 go, 54 stay."""
    net = Mlp(1)
    w = np.zeros(net.n_params, F)
    _, _, _, b2, w3, _ = _unpack(w, 1)
    b2[:], w3[:] = 1, F(0.02)
    w3[7], w3[9] = F(1e9), F(-1e9)
    net.params = w
    z = F(0)
    for k in range(H):
        z = F(z + w3[k])
    _, g = net.loss_grad([0.0], [0.0])
    net.close()
    assert abs(g[-1] - 1 / (1 + np.exp(-float(z)))) <= 1e-6  # a sum in parts is off by 0.02


@pytest.mark.parametrize("n_in,n", [(15, 32), (15, 33), (20, 100), (32, 128)])
def test_gradient_of_a_block(n_in, n):
    net, rng = _net(n_in, n)
    x = rng.standard_normal((n, n_in)).astype(F)
    y = (rng.random(n) < 0.3).astype(F)
    each = np.stack([net.loss_grad(x[k], y[k:k + 1], pos_weight=2.5)[1] for k in range(n)])
    assert np.array_equal(net.loss_grad(x, y, pos_weight=2.5)[1], _block_sum(each))
    net.close()


@pytest.mark.parametrize("n_in,n", [(15, 31), (15, 128), (20, 500), (15, 512), (15, 1024), (32, 513)])
def test_weights_after_a_step(n_in, n):
    """One minibatch, at the edges of a cluster's round of sixteen tiles: the block sums of 128 samples after one another,
    then Adam's first step (its bias corrections are 1 - 0.9f and 1 - 0.999f)."""
    net, rng = _net(n_in, n)
    w = net.params
    x = rng.standard_normal((n, n_in)).astype(F)
    y = (rng.random(n) < 0.3).astype(F)
    o = _order(n, 11)
    g = np.zeros(net.n_params, F)
    for first in range(0, n, 128):
        part = o[first:first + 128]
        g = g + net.loss_grad(x[part], y[part], pos_weight=2.5)[1]
    net.train(x, y, epochs=1, batch=n, lr=3e-3, pos_weight=2.5, seed=11)
    got = net.params
    net.close()
    g = g * (F(1) / F(n))
    b1, b2 = F(0.9), F(0.999)
    m, v = (F(1) - b1) * g, (F(1) - b2) * g * g
    want = w - F(3e-3) * (m / (F(1) - b1)) / (np.sqrt(v / (F(1) - b2)) + F(1e-8))
    assert np.array_equal(got, want)
