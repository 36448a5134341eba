"""The network's products on either tile width against the FP64 oracle: shapes
on both sides of the rule (a 64 x 64 tile for every SM) with remainders in
every dimension, and more rows than 65535 tiles of 32 hold."""
import importlib

import numpy as np
import pytest

import mlp_oracle as mo

pytestmark = pytest.mark.gpu


def _net(hidden, layers, rows, n_out=3):
    sur = importlib.import_module("matlab-cuda-efief-vs-cpu_b200.surrogate")
    net = sur.Surrogate(n_hidden=hidden, n_layers=layers, seed=5)
    r = np.random.default_rng(rows)
    X = r.uniform(-1, 1, (rows, 5)).astype(np.float32)
    T = r.uniform(-1, 1, (rows, n_out)).astype(np.float32)
    return net, mo.layer_shapes(5, hidden, layers, n_out), X, T


# 64-wide tiles of the hidden layer's products: 147, 148, 149 x 1, 74 x 2, 37 x 4 and their remainders
@pytest.mark.parametrize("hidden,layers,rows", [(64, 1, 147 * 64), (64, 1, 147 * 64 + 1), (33, 2, 149 * 64 - 31),
                                                (65, 2, 73 * 64), (65, 2, 73 * 64 + 17), (250, 2, 36 * 64),
                                                (250, 2, 37 * 64 - 5), (1030, 2, 600)])
def test_gradients_match_oracle(hidden, layers, rows):
    net, shapes, X, T = _net(hidden, layers, rows)
    p = net.get_params()
    loss, g = net.loss_grad(X, T)
    lo, go = mo.loss_grad(p, shapes, X, T)
    # the network's bounds: FP32 sums of BF16-weighted FP32 activations
    Y, Yo = net.forward(X), mo.forward(p, shapes, X)
    assert np.linalg.norm(Y - Yo) <= 1e-5 * np.linalg.norm(Yo)
    assert abs(loss - lo) <= 1e-5 * lo
    assert np.linalg.norm(g - go) <= 1e-4 * np.linalg.norm(go)


def test_more_rows_than_narrow_tiles_reach():
    rows = 65535 * 32 + 3
    net, shapes, X, T = _net(8, 1, rows)
    loss, g = net.loss_grad(X, T)
    lo, go = mo.loss_grad(net.get_params(), shapes, X, T)
    assert abs(loss - lo) <= 1e-5 * lo
    # the bias sums run over rows / 8 terms in FP32: sqrt(262141) * 2^-24 = 3e-5 of their size, which
    # is up to |T| / |mean dY| ~ 30 times the gradient's
    assert np.linalg.norm(g - go) <= 1e-3 * np.linalg.norm(go)
