"""The point data of the FP64 and FP32 sums (csrc/gauss.cu, k_point_forms) with few and many lanes
per cell: sparse cells with empty ones between, cells on both sides of 16 points on average, the
widest windows of 15 cells; single products against the oracle, FP32 ones to FP32's rounding."""
import numpy as np
import pytest

import oracle as O
from petrbf_gb300.api import Context, batch_interpolate
from test_gpu_fx_sums import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,nb,nt", [(2, 1, 15), (2, 4, 20), (3, 1, 9), (3, 2, 16)])
@pytest.mark.parametrize("per_cell", [0.3, 1.0, 4.0, 15.0, 17.0, 33.0])
def test_products(dim, nb, nt, per_cell):
    sigma = 0.02
    cells = 12 if dim == 2 else 5
    rng = np.random.default_rng(int(10 * per_cell) + nb)
    n = max(3, int(per_cell * cells ** dim))
    k = rng.uniform(0.0, cells * nb * sigma, (n, dim))
    z = k[:, 2].copy() if dim == 3 else None
    _check(k[:, 0].copy(), k[:, 1].copy(), z, sigma, nb, nt)
    # the FP32 data of the same words
    torch = pytest.importorskip("torch")
    v = rng.standard_normal(n)
    with Context(dim=dim, sigma=sigma, nsigma_box=nb, sigma_buffer=nb, sigma_trunc=nt) as c:
        c.matvec_setup(k[:, 0].copy(), k[:, 1].copy(), z)
        ref = c.matvec(v)
        size = c.matvec(np.abs(v))
        d = torch.from_numpy(v).cuda()
        out = torch.empty_like(d)
        torch.cuda.synchronize()
        c.matvec_dev(d.data_ptr(), out.data_ptr(), fp32=True)
        c.synchronize()
    # terms to 64 units of FP32 (coordinates to 2^-24 of half a cell's width, reach up to 10 sigma)
    assert np.max(np.abs(out.cpu().numpy() - ref) / size) <= 64 * 2.0 ** -24


def test_batches_of_sparse_and_dense_problems():
    # one problem of two points a cell among denser ones: the words are each problem's own
    probs = []
    for m, ov in ((9, 1.6), (30, 0.9), (45, 0.8)):
        h = 2.0 / m
        rng = np.random.default_rng(m)
        a = np.meshgrid(*([-1 + h * np.arange(m)] * 2), indexing="ij")
        x, y = (q.ravel() + rng.uniform(-0.2 * h, 0.2 * h, q.size) for q in a)
        probs.append(dict(x=x, y=y, f=np.cos(2 * x) * y, sigma=h * 0.5 / ov if m == 9 else h / ov, nsigma_box=4,
                          sigma_buffer=12, sigma_trunc=20))
    for order in (probs, probs[:1]):
        g, _, reason, _ = batch_interpolate(order, pc="asm")
        for q, w, r in zip(order, g, reason):
            gr = O.grid_for(q["x"], q["y"], None, q["sigma"], 4, 12, 20)
            perm, cs = O.cell_sort(gr, q["x"], q["y"])
            res = O.matvec(gr, q["x"][perm], q["y"][perm], None, cs, w[perm]) - q["f"][perm]
            assert r > 0 and np.linalg.norm(res) <= 1e-10 * np.linalg.norm(q["f"])
