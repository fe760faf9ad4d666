"""Batched sums with items of 32, 64 and 128 targets (tests/native/batch_tiles.cu)."""
import subprocess

import pytest

from native_build import compile_native

pytestmark = pytest.mark.gpu


def test_items_compute_their_own_targets(tmp_path):
    exe = compile_native("batch_tiles", tmp_path)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout[-1000:], r.stderr[-1000:])
