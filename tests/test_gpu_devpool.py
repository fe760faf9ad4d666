"""Device memory kept between calls: contexts of several threads and of different sizes reuse
one another's blocks and still compute what a lone context computes; what is kept is bounded."""
import threading

import numpy as np
import pytest

from petrbf_gb300 import workloads as W
from petrbf_gb300.api import Context, rbf_interpolation, vorticity_evaluation

pytestmark = pytest.mark.gpu


def _work(m, seed):
    rng = np.random.default_rng(seed)
    x, y, h = W.lattice_2d(m, jitter=0.25, seed=seed)
    t = rng.uniform(-1, 1, (2, 500 + 37 * m))
    prm = (h / 0.8, 8, 24, 24)
    f = W.lamb_oseen(x, y)
    with Context(sigma=prm[0], nsigma_box=8, sigma_buffer=24, sigma_trunc=24) as c:
        c.matvec_setup(x, y)
        a = c.matvec(f)
        c.matvec_setup(x[: x.size // 2], y[: x.size // 2])  # a smaller set in the same buffers
        b = c.matvec(f[: x.size // 2])
    w = vorticity_evaluation(t[0], t[1], x, y, f * h * h, *prm)
    g, its = rbf_interpolation(x, y, f, *prm) if m < 40 else (f, 0)
    return a, b, w, g


def test_threads_and_sizes_get_the_lone_contexts_results():
    jobs = [(m, s) for s, m in enumerate((12, 90, 33, 61, 24, 140))]
    alone = [_work(*j) for j in jobs]
    bad = []

    def run(order):
        for k in order:
            for p, q in zip(_work(*jobs[k]), alone[k]):
                if not np.array_equal(p, q):
                    bad.append(k)

    threads = [threading.Thread(target=run, args=([(k + t) % len(jobs) for k in range(len(jobs))] * 2,))
               for t in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_what_is_kept_is_bounded():
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    for s, m in enumerate((700, 650, 600, 550, 500, 450, 400, 350)):
        x, y, h = W.lattice_2d(m, jitter=0.25, seed=s)
        vorticity_evaluation(x[::7].copy(), y[::7].copy(), x, y, np.ones_like(x), h / 0.8, 8, 24, 24)
    assert before - torch.cuda.mem_get_info()[0] < (2 << 30) + (256 << 20)
