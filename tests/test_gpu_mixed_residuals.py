"""The FP64 residuals of 3D mixed-precision refinement: a batch takes the same sums as a single
solve, over wide and narrow truncation windows."""
import numpy as np
import pytest

from petrbf_gb300 import workloads as W
from petrbf_gb300.api import Context, batch_interpolate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths", [(3, 7, 17), (4, 8, 12)])
@pytest.mark.parametrize("m", [10, 17])
def test_batch_of_one_is_the_single_solve(widths, m):
    # one problem: the same reduction blocks, sums and block solves, hence the same bits
    x, y, z, h = W.lattice_3d(m, jitter=0.2, seed=m)
    f = np.cos(2 * x) * np.exp(-y * y) + z
    q = dict(x=x, y=y, z=z, f=f, sigma=h / 0.9, nsigma_box=widths[0], sigma_buffer=widths[1], sigma_trunc=widths[2])
    with Context(dim=3, sigma=q["sigma"], nsigma_box=widths[0], sigma_buffer=widths[1], sigma_trunc=widths[2],
                 precision="mixed", pc="asm") as c:
        g, st = c.interpolate(x, y, z, f)
    gb, its, reason, sb = batch_interpolate([q], dim=3, pc="asm", precision="mixed")
    assert st.fp64_fallback == 0 and sb.nprob_fp64 == 0
    assert st.reason == 2 and reason[0] == 2 and its[0] == st.its and sb.outer_its == st.outer_its
    np.testing.assert_array_equal(gb[0], g)
