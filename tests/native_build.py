"""Programs of tests/native, compiled against the library's own headers and linked to it."""
import os
import subprocess

from conftest import ROOT


def compile_native(name, out_dir):
    from petrbf_gb300 import build
    lib = build.build()
    exe = os.path.join(str(out_dir), name)
    cmd = [build.NVCC] + build.ARCH + ["-O2", "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC, "-I",
                                       os.path.join(ROOT, "include"),
                                       os.path.join(ROOT, "tests", "native", name + ".cu"), "-o", exe, lib,
                                       "-Xlinker", "-rpath=" + os.path.dirname(lib)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe
