"""How exact the FP64 sums are when all terms have one sign: 3D targets with some nine thousand
sources, against long double."""
import numpy as np
import pytest

from petrbf_gb300 import workloads as W
from petrbf_gb300.api import Context

pytestmark = pytest.mark.gpu

WIDTHS = (3, 7, 17)


@pytest.mark.parametrize("m,overlap", [(26, 0.8), (28, 0.9), (30, 1.0)])
def test_one_signed_3d_sums(m, overlap):
    x, y, z, h = W.lattice_3d(m, jitter=0.25, seed=m)
    sigma = h / overlap
    rng = np.random.default_rng(m)
    g = rng.uniform(0.5, 1.5, x.size)
    with Context(dim=3, sigma=sigma, nsigma_box=WIDTHS[0], sigma_buffer=WIDTHS[1], sigma_trunc=WIDTHS[2]) as c:
        c.matvec_setup(x, y, z)
        product = c.matvec(g)
        evaluated = c.evaluate(x, y, z, x, y, z, g)
    p = [x, y, z]
    box, length = WIDTHS[0] * sigma + 1e-6, WIDTHS[2] * sigma / 2 + 1e-6
    lo = [a.min() - 1e-6 for a in p]
    ld = np.longdouble
    norm = 1 / ((ld(np.pi) + ld(1.2246467991473532e-16)) * 2 * ld(sigma) * ld(sigma))
    err = []
    for i in rng.permutation(x.size)[:150]:
        keep, own = np.ones(x.size, bool), np.ones(x.size, bool)
        for a, b in zip(p, lo):
            k = np.floor((a[i] - b) / box)
            keep &= np.abs(a - (b + (k + 0.5) * box)) < length
            own &= np.floor((a - b) / box) == k
        j = np.flatnonzero(keep | own)
        d2 = sum((ld(a[i]) - a[j].astype(ld)) ** 2 for a in p)
        want = (np.exp(-d2 / (2 * ld(sigma) ** 2)) * g[j]).sum() * norm
        err.append([float((ld(w[i]) - want) / want) for w in (product, evaluated)])
    err = np.array(err)
    # in units of the result's last place: five halvings of the lanes' sums 0.40, their chains of
    # up to 48 terms 0.25, the last addition and the norm's product 0.29 each: 0.63, 0.74 of it as
    # the mantissas lie, 0.46 x 2^-52; a third on top for 150 samples. The mean: the rounding of
    # the norm, half a unit, and an eighth of the terms
    assert np.all(err.std(axis=0) <= 0.6 * 2.0 ** -52)
    assert np.all(np.abs(err.mean(axis=0)) <= 0.625 * 2.0 ** -52)
