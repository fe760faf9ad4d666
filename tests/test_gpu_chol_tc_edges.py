"""The FP32 tensor-core block Cholesky at the edges of its layout: blocks of one to four cells
whose neighbour and centre counts run over the remainders of a 16-byte unit (empty columns
between the two), of a 64-row tile, of a 128-row panel and of a 128-byte row pitch, and more
than 128 centre points (two passes of S_c). Each apply against the FP64 blocks of the oracle.

Tolerance: points at steps of 1.29 sigma and more (jittered by a fifth of a step) give blocks of
condition number up to about 300; the FP32 entries and factors carry about 2^-22 each, summed
over a block (a factor of 20 at 260 points): 300 * 20 * 2^-22 = 1.4e-3 of the result's norm, taken
as 2e-3. A lost or misplaced row changes it by 1 / sqrt(n), at least 0.06."""
import numpy as np
import pytest

import oracle as O
from petrbf_gb300.api import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pc", ["rasm", "asm"])
@pytest.mark.parametrize("counts", [(1,), (3,), (31,), (64,), (65,), (129,), (260,), (5, 1), (1, 5), (33, 62), (62, 33),
                                    (64, 64), (130, 63), (63, 130), (128, 129), (7, 66), (31, 97, 2, 128)])
def test_apply_tracks_fp64_blocks(counts, pc):
    rng = np.random.default_rng(sum(counts) * 10 + len(counts))
    prm = (0.0175, 22, 30, 24)
    box = prm[1] * prm[0] + 1e-6
    x, y = [], []
    for c, k in enumerate(counts):  # a row of cells
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
        c.pc_setup("mixed")
        z = c.pc_apply(r)
    g = O.grid_for(x, y, None, *prm)
    perm, cs = O.cell_sort(g, x, y)
    zo = np.empty(x.size)
    zo[perm] = O.Rasm(g, x[perm], y[perm], None, cs, basic=pc == "asm", factor="chol").apply(r[perm])
    assert np.linalg.norm(z - zo) <= 2e-3 * np.linalg.norm(zo)
