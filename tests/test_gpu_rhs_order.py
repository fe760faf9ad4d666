"""Right-hand sides that stop one by one, in every order of the columns: each count of vectors
left runs kernels of its own on whichever columns are left (from 4096 points), so the weights are
the same bits wherever a column stands, and the mixed form needs no FP64 solve."""
import itertools

import numpy as np
import pytest

from petrbf_gb300.api import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,precision,pc", [(3, "mixed", "asm"), (3, "fp64", "asm"), (2, "mixed", "asm"),
                                              (2, "mixed", "rasm"), (2, "fp64", "rasm"), (2, "fp64", "asm")])
def test_weights_do_not_depend_on_the_order_of_the_columns(dim, precision, pc):
    m = 17 if dim == 3 else 66
    h = 2.0 / m
    rng = np.random.default_rng(dim)
    ax = np.meshgrid(*([-1 + h * np.arange(m)] * dim), indexing="ij")
    p = [a.ravel() + rng.uniform(-0.2 * h, 0.2 * h, a.size) for a in ax]
    z = p[2] if dim == 3 else None
    prm = (h, 3, 7, 17) if dim == 3 else (h, 4, 12, 20)
    # nothing, a smooth field, noise: they stop after different numbers of iterations
    cols = [np.zeros(p[0].size), np.cos(p[0]) * p[1], rng.standard_normal(p[0].size)]
    want = None
    with Context(dim=dim, sigma=prm[0], nsigma_box=prm[1], sigma_buffer=prm[2], sigma_trunc=prm[3], pc=pc,
                 precision=precision) as c:
        for order in itertools.permutations(range(3)):
            g, st = c.interpolate(p[0], p[1], z, np.stack([cols[k] for k in order], axis=1))
            assert st.fp64_fallback == 0 and st.true_rel_resid <= 1e-10
            got = np.stack([g[:, order.index(k)] for k in range(3)])
            assert not got[0].any()
            want = got if want is None else want
            np.testing.assert_array_equal(got, want)
