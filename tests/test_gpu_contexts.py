"""Several contexts of one process: what one of them sets up takes nothing away from another,
one after the other and on threads of their own."""
import threading

import numpy as np
import pytest

from petrbf_gb300 import _native as N
from petrbf_gb300 import workloads as W
from petrbf_gb300.api import Context, PrbfError, rbf_interpolation

pytestmark = pytest.mark.gpu


def _lattice(dim, m, seed=0):
    if dim == 2:
        x, y, h = W.lattice_2d(m, jitter=0.25, seed=seed)
        return x, y, None, dict(dim=2, sigma=h / 0.8, nsigma_box=8, sigma_buffer=24, sigma_trunc=24)
    x, y, z, h = W.lattice_3d(m, jitter=0.25, seed=seed)
    return x, y, z, dict(dim=3, sigma=h / 0.8, nsigma_box=3, sigma_buffer=7, sigma_trunc=17)


@pytest.mark.parametrize("dim,precision,pc", [(2, "fp64", "rasm"), (2, "fp64", "asm"), (2, "mixed", "rasm"),
                                              (3, "fp64", "asm"), (3, "mixed", "asm")])
def test_applies_after_a_context_with_smaller_blocks(dim, precision, pc):
    big, small = _lattice(dim, 40 if dim == 2 else 12), _lattice(dim, 6 if dim == 2 else 3)
    r = np.random.default_rng(1).standard_normal(big[0].size)
    with Context(pc=pc, **big[3]) as a, Context(pc=pc, **small[3]) as b:
        a.matvec_setup(*big[:3])
        a.pc_setup(precision)
        before = a.pc_apply(r)
        b.matvec_setup(*small[:3])
        b.pc_setup(precision)
        np.testing.assert_array_equal(a.pc_apply(r), before)


def _blob(n, seed):
    # points so close that the Cholesky of their block meets a pivot that is not positive, and
    # no two alike: LU factors it
    rng = np.random.default_rng(seed)
    x, y = rng.uniform(0.0, 0.2, (2, n))
    return x, y, dict(dim=2, sigma=1.0, nsigma_box=8, sigma_buffer=24, sigma_trunc=24, block_fallback="lu")


def test_lu_applies_after_a_context_with_smaller_blocks():
    big, small = _blob(200, 1), _blob(40, 2)
    r = np.random.default_rng(3).standard_normal(200)
    with Context(**big[2]) as a, Context(**small[2]) as b:
        out = []
        for c, p in ((a, big), (b, small)):
            c.matvec_setup(p[0], p[1])
            c.pc_setup("fp64")
            with pytest.raises(PrbfError) as e:  # no Cholesky factor to read back: it is LU's
                c.pc_block(0, block=False)
            assert e.value.status == N.ERR_STATE
            out.append(a.pc_apply(r))
    np.testing.assert_array_equal(out[0], out[1])


def test_threads_with_blocks_of_different_sizes():
    def job(k):
        m, precision, nrhs = [(12, "fp64", 1), (33, "fp64", 2), (24, "mixed", 1), (50, "fp64", 1), (40, "mixed", 3),
                              (16, "fp64", 3)][k]
        x, y, _, prm = _lattice(2, m, seed=k)
        f = W.lamb_oseen(x, y)
        if nrhs > 1:
            f = np.stack([f * (1 + v) + x * v for v in range(nrhs)], axis=1)
        prm = dict(prm)
        prm.pop("dim")
        return rbf_interpolation(x, y, f, *prm.values(), precision=precision)[0]

    alone = [job(k) for k in range(6)]
    wrong = []

    def run(t):
        for k in [(i + t) % 6 for i in range(6)] * 3:
            try:
                if not np.array_equal(job(k), alone[k]):
                    wrong.append((t, k, "another result"))
            except Exception as e:  # noqa: BLE001 (a call that fails is a failure of the test)
                wrong.append((t, k, repr(e)))

    threads = [threading.Thread(target=run, args=(t,)) for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
