"""Memory the library takes for itself, when it runs out, on a fake of the CUDA
calls that hand it out (tests/host_memory_check.cpp; no GPU)."""
import os
import shutil
import subprocess

import pytest

from harness import PKG, ROOT


def test_out_of_memory_and_what_is_kept():
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = os.path.join(ROOT, "_build", "host_memory_check")
    os.makedirs(out, exist_ok=True)
    exe = os.path.join(out, "host_memory_check")
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "include"), "-I", os.path.join(PKG, "csrc"),
                    "-I", "/usr/local/cuda/include", os.path.join(ROOT, "tests", "host_memory_check.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip().endswith("ok")
