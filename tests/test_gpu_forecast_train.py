"""One epoch of training on the GPU against the oracle's gradients and Adam in FP64, at the edges of the
kernel's tiles (32 samples, up to sixteen tiles side by side) and of the input widths it takes."""
import os
import sys

import numpy as np
import pytest

from conftest import ROOT
from dacti_b200.forecast import Mlp

sys.path.insert(0, os.path.join(ROOT, "oracle"))
import forecast_mlp as ref  # noqa: E402

pytestmark = pytest.mark.gpu
LR, PW, SEED = 3e-3, 2.5, 11


def _order(n, state):
    """Fisher-Yates with splitmix64, as the training draws it."""
    perm, mask = list(range(n)), (1 << 64) - 1
    for k in range(n - 1, 0, -1):
        state = (state + 0x9E3779B97F4A7C15) & mask
        z = ((state ^ (state >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        j = (z ^ (z >> 31)) % (k + 1)
        perm[k], perm[j] = perm[j], perm[k]
    return np.array(perm)


@pytest.mark.parametrize("n_in,n,batch", [(1, 1, 1), (15, 31, 8), (15, 64, 32), (7, 97, 33), (32, 513, 511), (15, 1024, 512),
                                          (20, 1500, 700), (3, 300, 1000)])
def test_epoch_matches_oracle(n_in, n, batch):
    rng = np.random.default_rng(n + n_in)
    net = Mlp(n_in, seed=2)
    w = net.params.astype(np.float64)
    x = rng.normal(size=(n, n_in)).astype(np.float32)
    y = (rng.random(n) < 0.3).astype(np.float32)
    got = net.train(x, y, epochs=1, batch=batch, lr=LR, pos_weight=PW, seed=SEED)
    order, loss = _order(n, SEED), 0.0
    m, v, t = np.zeros_like(w), np.zeros_like(w), 0
    for first in range(0, n, batch):
        idx = order[first:first + batch]
        part, g = ref.loss_grad(w, x[idx], y[idx], PW)
        loss, g, t = loss + part, g / len(idx), t + 1
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        w = w - LR * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    # FP32 gradients are good to about 1e-6 of the largest; a step is lr times a ratio of gradients, so a
    # weight whose gradient is a thousandth of the largest moves by lr (1 +- 1e-3)
    off = net.params - w
    assert np.sqrt((off ** 2).mean()) <= 1e-3 * LR * t
    assert abs(got - loss / n) <= 1e-5 * abs(loss / n) + LR * 1e-3
    net.close()


def test_gradient_over_many_tiles():
    rng = np.random.default_rng(8)
    net = Mlp(15, seed=4)
    n = 148 * 2 * 32 * 2 + 17  # more tiles than blocks, the last one ragged
    x = rng.normal(size=(n, 15)).astype(np.float32)
    y = (rng.random(n) < 0.3).astype(np.float32)
    loss, g = net.loss_grad(x, y, pos_weight=PW)
    rl, rg = ref.loss_grad(net.params.astype(np.float64), x, y, PW)
    assert abs(loss - rl) <= 1e-5 * abs(rl)
    assert np.abs(g - rg).max() <= 1e-5 * np.abs(rg).max()
    net.close()


@pytest.mark.parametrize("widths", [(20, 15), (32, 1), (15, 32, 20)])
def test_networks_of_several_widths_at_once(widths):
    """A network made later, with fewer inputs, takes nothing from those that are there."""
    rng = np.random.default_rng(5)
    nets = [Mlp(w, seed=3) for w in widths]
    for _ in range(2):
        for net in nets:
            x = rng.normal(size=(100, net.n_in)).astype(np.float32)
            y = (rng.random(100) < 0.3).astype(np.float32)
            loss, g = net.loss_grad(x, y, pos_weight=PW)
            rl, rg = ref.loss_grad(net.params.astype(np.float64), x, y, PW)
            assert abs(loss - rl) <= 1e-5 * abs(rl) and np.abs(g - rg).max() <= 1e-5 * np.abs(rg).max()
            assert np.isfinite(net.train(x, y, epochs=1, batch=64, lr=LR, pos_weight=PW, seed=SEED))
            assert np.isfinite(net.predict(x)).all()
    for net in nets:
        net.close()


@pytest.mark.parametrize("n,batch,epochs", [(300, 64, 3), (1024, 512, 5)])
def test_epochs_match_oracle(n, batch, epochs):
    """Several epochs: each runs in its own order, which the host draws while the GPU runs the one before."""
    rng = np.random.default_rng(n)
    net = Mlp(15, seed=2)
    w = net.params.astype(np.float64)
    x = rng.normal(size=(n, 15)).astype(np.float32)
    y = (rng.random(n) < 0.3).astype(np.float32)
    got = net.train(x, y, epochs=epochs, batch=batch, lr=LR, pos_weight=PW, seed=SEED)
    perm, state, mask = list(range(n)), SEED, (1 << 64) - 1
    m, v, t = np.zeros_like(w), np.zeros_like(w), 0
    for _ in range(epochs):
        for k in range(n - 1, 0, -1):
            state = (state + 0x9E3779B97F4A7C15) & mask
            z = ((state ^ (state >> 30)) * 0xBF58476D1CE4E5B9) & mask
            z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
            j = (z ^ (z >> 31)) % (k + 1)
            perm[k], perm[j] = perm[j], perm[k]
        loss = 0.0
        for first in range(0, n, batch):
            idx = perm[first:first + batch]
            part, g = ref.loss_grad(w, x[idx], y[idx], PW)
            loss, g, t = loss + part, g / len(idx), t + 1
            m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
            w = w - LR * (m / (1 - 0.9 ** t)) / (np.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    off = net.params - w  # the bounds of test_epoch_matches_oracle
    assert np.sqrt((off ** 2).mean()) <= 1e-3 * LR * t
    assert abs(got - loss / n) <= 1e-5 * abs(loss / n) + LR * 1e-3
    net.close()
