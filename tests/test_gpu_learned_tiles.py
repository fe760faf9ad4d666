"""The network's products at the edges of their tiles: rows around 32, 128 and the number from
which a CTA takes all columns, against the same rows in other company and the oracle."""
import numpy as np
import pytest

from oracle import mlp as OM
from petrbf_gb300 import learned as L

pytestmark = pytest.mark.gpu

RTOL_NET = 2e-3  # as in test_gpu_learned.py: BF16 operands, FP32 sums against the oracle's FP64


def _rows(n, seed=0):
    rng = np.random.default_rng(seed)
    X = rng.standard_normal((n, L.IN)).astype(np.float32)
    T = rng.standard_normal((n, L.OUT)).astype(np.float32)
    M = (rng.random((n, L.OUT)) < 0.8).astype(np.float32)
    return X, T, M


def test_row_tiles_do_not_change_a_rows_result():
    # 75 row tiles and fewer split the columns over CTAs, 76 do not; a row's sums are the same
    X, _, _ = _rows(76 * 128)
    net = L.Network(seed=2)
    whole = net.forward(X)
    parts = np.concatenate([net.forward(X[a:a + 4001]) for a in range(0, len(X), 4001)])
    np.testing.assert_array_equal(whole, parts)


@pytest.mark.parametrize("n", [31, 33, 127, 128, 129, 257])
def test_gradients_at_tile_edges(n):
    X, T, M = _rows(n, seed=n)
    M[0, 0] = 1.0
    net = L.Network(seed=4)
    loss, g = net.loss_grad(X, T, M)
    loss_o, g_o = OM.loss_grad(net.weights, X, T, M)
    assert abs(loss - loss_o) <= RTOL_NET * loss_o
    assert np.linalg.norm(g - g_o) <= RTOL_NET * np.linalg.norm(g_o)


@pytest.mark.parametrize("n,batch", [(70, 32), (300, 129), (40, 64)])
def test_training_takes_the_gathered_rows_steps(n, batch):
    # one epoch of training equals its own steps' losses and moves every weight; two networks
    # with the same seed end bit for bit alike
    X, T, M = _rows(n, seed=batch)
    nets = [L.Network(seed=6) for _ in range(2)]
    w0 = nets[0].weights
    for net in nets:
        hist = net.train(X, T, M, epochs=1, batch=batch, seed=3)
        assert np.isfinite(hist).all()
    np.testing.assert_array_equal(nets[0].weights, nets[1].weights)
    assert np.mean(nets[0].weights != w0) > 0.9
