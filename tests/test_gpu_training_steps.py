"""An epoch of training replayed step by step: the library's permutation, the oracle's gradients of
each step's rows and Adam on the host, against the network's loss and weights; and the network's
BF16 copies of the weights after it."""
import numpy as np
import pytest

from oracle import mlp as OM
from petrbf_gb300 import learned as L

pytestmark = pytest.mark.gpu

RTOL_NET = 2e-3  # as in test_gpu_learned.py


def _permutation(n, seed):
    """learned.cu: Fisher-Yates from the end, splitmix64."""
    mask = (1 << 64) - 1
    state, perm = seed, list(range(n))

    def mix():
        nonlocal state
        state = (state + 0x9E3779B97F4A7C15) & mask
        z = state
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        return z ^ (z >> 31)

    for i in range(n - 1, 0, -1):
        j = mix() % (i + 1)
        perm[i], perm[j] = perm[j], perm[i]
    return np.array(perm)


@pytest.mark.parametrize("n,batch", [(300, 129), (200, 64)])
def test_an_epoch_takes_the_permutations_steps(n, batch):
    rng = np.random.default_rng(batch)
    X = rng.standard_normal((n, L.IN)).astype(np.float32)
    T = rng.standard_normal((n, L.OUT)).astype(np.float32)
    # rows differ in their number of targets, so that a step with another step's rows shows
    M = (rng.random((n, L.OUT)) < rng.uniform(0.2, 1.0, (n, 1))).astype(np.float32)
    M[:, 0] = 1.0
    lr, b1, b2, eps = 1e-3, 0.9, 0.999, 1e-8
    net = L.Network(seed=6)
    w = net.weights.astype(np.float64)
    w0 = w.copy()
    m1, m2 = np.zeros_like(w), np.zeros_like(w)
    perm = _permutation(n, 3)
    losses, steps = [], 0
    for b in range(0, n, batch):
        r = perm[b:b + batch]
        loss, g = OM.loss_grad(w.astype(np.float32), X[r], T[r], M[r])
        losses.append(loss)
        steps += 1
        m1 = b1 * m1 + (1 - b1) * g
        m2 = b2 * m2 + (1 - b2) * g * g
        w = w - lr * (m1 / (1 - b1 ** steps)) / (np.sqrt(m2 / (1 - b2 ** steps)) + eps)
    hist = net.train(X, T, M, epochs=1, batch=batch, lr=lr, seed=3)
    assert abs(hist[-1] - np.mean(losses)) <= RTOL_NET * np.mean(losses)
    # Adam's first steps have the size of lr whatever the gradient's, so a weight whose gradient
    # is within the network's tolerance (2e-3 of the mean square) of zero may move the other way, two
    # in a thousand, 0.06 of the norm; all others move alike
    moved, want = net.weights - w0, w - w0
    assert np.linalg.norm(moved - want) <= 0.1 * np.linalg.norm(want)
    # another permutation's rows do not: the test can tell
    other = L.Network(seed=6)
    other.train(X, T, M, epochs=1, batch=batch, lr=lr, seed=4)
    assert np.linalg.norm(other.weights - w0 - want) > 0.2 * np.linalg.norm(want)
    # the BF16 copies that the products read follow the weights: the loss (row-major) and the
    # gradients of the inner layers (transposed), against the oracle at the trained weights
    loss, g = net.loss_grad(X, T, M)
    loss_o, g_o = OM.loss_grad(net.weights, X, T, M)
    assert abs(loss - loss_o) <= RTOL_NET * loss_o
    assert np.linalg.norm(g - g_o) <= RTOL_NET * np.linalg.norm(g_o)
