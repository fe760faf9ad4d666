"""The LU fallback's applies to several vectors at once (tests/native/lu_vectors.cu)."""
import subprocess

import pytest

from native_build import compile_native

pytestmark = pytest.mark.gpu


def test_several_vectors_at_once(tmp_path):
    exe = compile_native("lu_vectors", tmp_path)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout[-1000:], r.stderr[-1000:])
