"""The FP64 sums with fixed-point exponents (csrc/gauss_fx.cu) where they can go wrong: cells
at the edges of a warp's, a pass's and a tile's targets, windows at the rule's limits, shifted
coordinates, targets without sources, several vectors."""
import numpy as np
import pytest

import oracle as O
from petrbf_gb300.api import Context

pytestmark = pytest.mark.gpu

# every term within a few 2^-53 of the oracle's, and sums of at most some thousand terms in
# another order: 1e-14 of the sum of the terms' sizes
TOL = 1e-14


def _check(x, y, z, sigma, nb, nt, seed=0):
    rng = np.random.default_rng(seed)
    v = rng.standard_normal(x.size)
    with Context(dim=3 if z is not None else 2, sigma=sigma, nsigma_box=nb, sigma_buffer=nb, sigma_trunc=nt) as c:
        c.matvec_setup(x, y, z)
        got = c.matvec(v)
        again = c.matvec(v)
    g = O.grid_for(x, y, z, sigma, nb, nb, nt)
    perm, cs = O.cell_sort(g, x, y, z)
    pz = z[perm] if z is not None else None
    want, size = np.empty(x.size), np.empty(x.size)
    want[perm] = O.matvec(g, x[perm], y[perm], pz, cs, v[perm])
    size[perm] = O.matvec(g, x[perm], y[perm], pz, cs, np.abs(v[perm]))
    assert np.max(np.abs(got - want) / size) <= TOL
    np.testing.assert_array_equal(got, again)


@pytest.mark.parametrize("n", [1, 7, 8, 31, 32, 33, 44, 63, 64, 65, 88, 89, 127, 128, 129, 300])
@pytest.mark.parametrize("dim", [2, 3])
def test_cell_sizes(dim, n):
    # a cell of n points, its neighbour of 40, and one point five cells away
    sigma, nb = 0.01, 4
    box = nb * sigma + 1e-6
    rng = np.random.default_rng(n)
    k = rng.uniform(0.02, 0.98, (n + 41, dim)) * box
    k[n:n + 40, 0] += box
    k[n + 40:] += 5 * box
    k[0] = 0.0  # the grid starts here
    z = k[:, 2].copy() if dim == 3 else None
    _check(k[:, 0].copy(), k[:, 1].copy(), z, sigma, nb, 20)


# widths inside and just outside of what the fixed-point coordinates reach (18.65 sigma per
# axis in 2D, 15.2 in 3D, half a cell included), small and large windows
@pytest.mark.parametrize("dim,nb,nt", [(2, 8, 29), (2, 8, 30), (2, 2, 20), (2, 1, 16), (2, 6, 6), (2, 8, 0),
                                       (3, 3, 27), (3, 3, 28), (3, 2, 16), (3, 8, 8)])
@pytest.mark.parametrize("shift", [0.0, 1e4])
def test_windows_and_shifts(dim, nb, nt, shift):
    rng = np.random.default_rng(nb * 100 + nt)
    n = 1500
    k = rng.uniform(0.0, 0.5, (n, dim)) + shift
    k[3] = k[2]  # coincident points
    z = k[:, 2].copy() if dim == 3 else None
    _check(k[:, 0].copy(), k[:, 1].copy(), z, 0.02 if dim == 2 else 0.04, nb, nt)


def _long_double_sum(t, s, g, sigma, nb, nt):
    """The truncated sum and the sum of its terms' sizes in long double. (The oracle rounds the
    exponent, so its terms of e^-75 are off by 75 2^-53 relative: too far for TOL.)"""
    box, length = nb * sigma + 1e-6, nt * sigma / 2 + 1e-6
    lo = np.minimum(t.min(0), s.min(0)) - 1e-6
    ct, cs = np.floor((t - lo) / box), np.floor((s - lo) / box)
    keep = np.ones((len(t), len(s)), bool)
    same = np.ones_like(keep)
    d2 = np.zeros(keep.shape, np.longdouble)
    for k in range(t.shape[1]):
        keep &= np.abs(s[None, :, k] - (lo[k] + (ct[:, k, None] + 0.5) * box)) < length
        same &= ct[:, k, None] == cs[None, :, k]
        d2 += (t[:, k, None].astype(np.longdouble) - s[None, :, k]) ** 2
    e = np.where(keep | same, np.exp(-d2 / (2 * np.longdouble(sigma) ** 2)), 0) / (2 * np.pi * sigma * sigma)
    return (e * g).sum(1), (e * np.abs(g)).sum(1)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("nt", [1, 5, 1000])
def test_evaluation_off_the_sources(dim, nt):
    rng = np.random.default_rng(nt)
    s = rng.uniform(0.0, 0.4, (700, dim))
    t = rng.uniform(-0.3, 1.0, (nt, dim))  # many cells without any source in reach
    g = rng.standard_normal(700)
    prm = (0.02, 4, 4, 20)
    col = lambda a, k: a[:, k].copy() if k < dim else None  # noqa: E731
    with Context(dim=dim, sigma=prm[0], nsigma_box=prm[1], sigma_buffer=prm[2], sigma_trunc=prm[3]) as c:
        got = c.evaluate(col(t, 0), col(t, 1), col(t, 2), col(s, 0), col(s, 1), col(s, 2), g)
    want, size = _long_double_sum(t, s, g, prm[0], prm[1], prm[3])
    assert np.all(np.abs(got - want) <= TOL * size)


@pytest.mark.parametrize("dim,nrhs", [(2, 2), (2, 4), (2, 5), (3, 2), (3, 4)])
def test_several_vectors(dim, nrhs):
    # the residual of the weights by the oracle's operator: GMRES stops at 1e-13 of the
    # preconditioned residual, the condition of the blocks far below 1e2
    m = 40 if dim == 2 else 12
    h = 2.0 / m
    rng = np.random.default_rng(nrhs)
    ax = np.meshgrid(*([-1 + h * np.arange(m)] * dim), indexing="ij")
    p = [a.ravel() + rng.uniform(-0.2 * h, 0.2 * h, a.size) for a in ax]
    z = p[2] if dim == 3 else None
    prm = (h, 4, 12, 20) if dim == 2 else (h, 3, 7, 17)
    f = np.stack([np.cos((k + 1) * p[0]) * p[1] for k in range(nrhs)], axis=1)
    with Context(dim=dim, sigma=prm[0], nsigma_box=prm[1], sigma_buffer=prm[2], sigma_trunc=prm[3], pc="asm") as c:
        g, _ = c.interpolate(p[0], p[1], z, f)
    gr = O.grid_for(p[0], p[1], z, *prm)
    perm, cs = O.cell_sort(gr, p[0], p[1], z)
    pz = z[perm] if dim == 3 else None
    for k in range(nrhs):
        r = O.matvec(gr, p[0][perm], p[1][perm], pz, cs, g[perm, k]) - f[perm, k]
        assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(f[:, k])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("stopped", [0, 1, 2])
def test_stopped_right_hand_sides_are_left_out(precision, stopped):
    # a zero right-hand side among three stops at once, the others go on without it (from 4096
    # points); weights against the oracle's residual, as above
    m = 18
    h = 2.0 / m
    rng = np.random.default_rng(stopped)
    ax = np.meshgrid(*([-1 + h * np.arange(m)] * 3), indexing="ij")
    x, y, z = (a.ravel() + rng.uniform(-0.2 * h, 0.2 * h, a.size) for a in ax)
    prm = (h, 3, 7, 17)
    f = np.stack([np.cos((k + 1) * x) * y for k in range(3)], axis=1)
    f[:, stopped] = 0.0
    with Context(dim=3, sigma=prm[0], nsigma_box=prm[1], sigma_buffer=prm[2], sigma_trunc=prm[3], pc="asm",
                 precision=precision) as c:
        g, _ = c.interpolate(x, y, z, f)
    assert not g[:, stopped].any()
    gr = O.grid_for(x, y, z, *prm)
    perm, cs = O.cell_sort(gr, x, y, z)
    for k in range(3):
        if k != stopped:
            r = O.matvec(gr, x[perm], y[perm], z[perm], cs, g[perm, k]) - f[perm, k]
            assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(f[:, k])
