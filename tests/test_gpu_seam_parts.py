"""The packed FP32 product in parts: calls large enough to be cut against calls of few blocks."""
import numpy as np
import pytest

from petrbf_gb300.api import gpumatmult

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("total,dim", [(2 * 2**21 - 1, 2), (2 * 2**21, 2), (3 * 2**21 + 5, 2), (2 * 2**21 + 3, 3)])
def test_gpumatmult_in_parts_equals_single_parts(total, dim):
    # From 2 x 2^21 sources on a call copies and sums in parts of whole blocks. Blocks of ragged
    # sizes (empty ones too, starts at every remainder of four): each block's sum runs over its
    # own sources in order, so calls of few blocks give the same bits.
    rng = np.random.default_rng(total % 1000 + dim)
    cnt = rng.integers(0, 8000, 2 * total // 8000)
    cnt[rng.integers(0, len(cnt), 40)] = 0
    off = np.concatenate([[0], np.cumsum(cnt)])
    off = off[off <= total]
    off[-1] = total
    off = off.astype(np.int32)
    nb = len(off) - 1
    t = [rng.uniform(0, 1, 128 * nb).astype(np.float32) for _ in range(dim)] + [None] * (3 - dim)
    s = [rng.uniform(0, 1, total).astype(np.float32) for _ in range(dim)] + [None] * (3 - dim)
    g = rng.standard_normal(total).astype(np.float32)
    whole = gpumatmult(*t, *s, g, off, 0.05)
    step = 100
    for b in range(0, nb, step):
        e = min(nb, b + step)
        cut = lambda a, lo, hi: a[lo:hi] if a is not None else None
        part = gpumatmult(*(cut(a, 128 * b, 128 * e) for a in t), *(cut(a, off[b], off[e]) for a in s),
                          g[off[b]:off[e]], off[b:e + 1] - off[b], 0.05)
        np.testing.assert_array_equal(whole[128 * b:128 * e], part)
