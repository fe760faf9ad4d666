"""Slots of basic Schwarz with several right-hand sides (tests/native/slot_budget.cu)."""
import subprocess

import pytest

from native_build import compile_native

pytestmark = pytest.mark.gpu


def test_slots_of_several_vectors_stay_within_the_budget(tmp_path):
    exe = compile_native("slot_budget", tmp_path)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout[-1000:], r.stderr[-1000:])
