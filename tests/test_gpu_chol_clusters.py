"""The FP64 block Cholesky with one to eight CTAs per block: the number of blocks picks the
cluster, so point sets of few and many cells with blocks of ragged sizes (tiles' edges at 64,
row shares of 8; the apply's CTAs of one to eight warps), each compared bit for bit with the restated block arithmetic through the
Schwarz apply."""
import numpy as np
import pytest

import oracle as O
from petrbf_gb300.api import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pc", ["rasm", "asm"])
@pytest.mark.parametrize("cells,most", [(1, 1), (1, 63), (1, 64), (1, 65), (1, 129), (2, 200), (13, 150), (30, 260),
                                        (60, 90), (100, 140), (152, 60), (220, 70), (310, 66),
                                        (700, 20), (2700, 9)])
def test_applies_equal_the_restatement(cells, most, pc):
    rng = np.random.default_rng(cells * 1000 + most)
    prm = (0.0175, 22, 30, 24)  # lattice steps of 1.3 sigma and more: no shifted blocks
    box = prm[1] * prm[0] + 1e-6
    x, y = [], []
    for c in range(cells):  # a row of cells, up to `most` jittered lattice points each
        k = most if c == 0 else int(rng.integers(1, most + 1))
        m = int(np.ceil(np.sqrt(k)))
        i = np.arange(m * m)
        pick = np.sort(rng.permutation(m * m)[:k])
        jit = rng.uniform(-0.2, 0.2, (m * m, 2))
        x.append((c + 0.02 + 0.96 * ((i // m + 0.5 + jit[:, 0]) / m)[pick]) * box)
        y.append((0.02 + 0.96 * ((i % m + 0.5 + jit[:, 1]) / m)[pick]) * box)
    x, y = np.concatenate(x), np.concatenate(y)
    r = rng.standard_normal(x.size)
    with Context(dim=2, sigma=prm[0], nsigma_box=prm[1], sigma_buffer=prm[2], sigma_trunc=prm[3], pc=pc) as c:
        c.matvec_setup(x, y)
        c.pc_setup("fp64")
        z = c.pc_apply(r)
    g = O.grid_for(x, y, None, *prm)
    perm, cs = O.cell_sort(g, x, y)
    zo = np.empty(x.size)
    zo[perm] = O.Rasm(g, x[perm], y[perm], None, cs, basic=pc == "asm", factor="chol").apply(r[perm])
    np.testing.assert_array_equal(z, zo)
