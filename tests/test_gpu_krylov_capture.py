"""The iteration's capture into a graph when an operator fails inside it (a host exception, a
launch that the runtime refuses): tests/native/krylov_capture.cu, in a process of its own."""
import subprocess

import pytest

from native_build import compile_native

pytestmark = pytest.mark.gpu


def test_a_failure_inside_the_capture_leaves_a_usable_state(tmp_path):
    exe = compile_native("krylov_capture", tmp_path)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout[-1000:], r.stderr[-1000:])
