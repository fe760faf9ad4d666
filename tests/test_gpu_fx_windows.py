"""The FP64 sums about the widest 3D windows of the fixed-point form, and with infinite weights."""
import numpy as np
import pytest

from petrbf_gb300.api import Context
from test_gpu_fx_sums import _check

pytestmark = pytest.mark.gpu


# from 12.4 sigma per axis (half a cell included; between sigma_trunc 21 and 22 with cells of 3
# sigma) the wide form, from 15.2 (27 and 28) the FP64 pipe's kernels
@pytest.mark.parametrize("nt", [20, 21, 22, 23, 25, 27, 28])
def test_3d_windows_at_the_rules_limit(nt):
    rng = np.random.default_rng(nt)
    k = rng.uniform(0.0, 0.9, (1500, 3))
    _check(k[:, 0].copy(), k[:, 1].copy(), k[:, 2].copy(), 0.04, 3, nt)


@pytest.mark.parametrize("dim", [2, 3])
def test_infinite_weights_reach_their_targets(dim):
    rng = np.random.default_rng(dim)
    k = rng.uniform(0.0, 1.0, (3000, dim))
    g = rng.uniform(0.5, 1.5, 3000)
    box = 3 * 0.02 + 1e-6
    col = lambda d: k[:, d].copy() if d < dim else None  # noqa: E731
    with Context(dim=dim, sigma=0.02, nsigma_box=3, sigma_buffer=7, sigma_trunc=17) as c:
        c.matvec_setup(col(0), col(1), col(2))
        plain = c.matvec(g)
        h = g.copy()
        h[5], h[6] = np.inf, -np.inf
        got = c.matvec(h)
        h[6] = g[6]
        one = c.matvec(h)
    lo = k.min(0) - 1e-6
    centre = lo + (np.floor((k - lo) / box) + 0.5) * box
    reach = [np.all(np.abs(k[j] - centre) < 17 * 0.02 / 2 + 1e-6, axis=1) for j in (5, 6)]
    assert reach[0].any() and not reach[0].all()
    assert np.all(one[reach[0]] == np.inf)
    both = reach[0] & reach[1]
    assert np.all(np.isnan(got[both])) if both.any() else True
    assert np.all(got[reach[1] & ~reach[0]] == -np.inf)
    far = ~reach[0] & ~reach[1]
    np.testing.assert_array_equal(got[far], plain[far])
