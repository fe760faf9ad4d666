"""Device memory kept between calls on the GPU: the bound after more work than it holds, no growth
on repeated calls, and the release call."""
import numpy as np
import pytest

from petrbf_gb300 import workloads as W
from petrbf_gb300.api import Context, memory_kept, release_memory, vorticity_evaluation

pytestmark = pytest.mark.gpu


def _evaluate(m):
    x, y, h = W.lattice_2d(m, jitter=0.25, seed=m)
    w = vorticity_evaluation(x[::50].copy(), y[::50].copy(), x, y, np.ones_like(x), h / 0.8, 8, 24, 24)
    return w


def test_bound_reuse_and_release():
    torch = pytest.importorskip("torch")
    torch.cuda.synchronize()
    release_memory()
    assert memory_kept() == 0
    first = _evaluate(1000)
    # (some fifteen arrays of 10^6 points, four to eight bytes each, are kept)
    assert memory_kept() > 50 << 20
    kept = memory_kept()
    np.testing.assert_array_equal(_evaluate(1000), first)
    assert memory_kept() == kept
    for m in (3200, 3000, 2800, 2600):  # 0.7 to 1.3 GB each, in size classes of their own
        _evaluate(m)
        assert memory_kept() <= 2 << 30
    assert memory_kept() > 1 << 30
    kept, free = memory_kept(), torch.cuda.mem_get_info()[0]
    release_memory()
    assert memory_kept() == 0
    assert torch.cuda.mem_get_info()[0] >= free + kept - (64 << 20)
    np.testing.assert_array_equal(_evaluate(1000), first)


def test_release_beside_a_live_context():
    x, y, h = W.lattice_2d(200, jitter=0.25, seed=1)
    v = np.random.default_rng(0).standard_normal(x.size)
    with Context(sigma=h / 0.8) as c:
        c.matvec_setup(x, y)
        a = c.matvec(v)
        release_memory()
        np.testing.assert_array_equal(c.matvec(v), a)
        c.matvec_setup(x, y)
        np.testing.assert_array_equal(c.matvec(v), a)
