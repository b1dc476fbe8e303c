"""Giving host arrays their pages before a download leaves what they hold, checked by tests/host_pages_check.cpp
against the library's own object."""
import os
import shutil
import subprocess

import pytest

from pachydermacoustic_universal_gb300 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_touching_pages_keeps_their_contents(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    build.build()
    obj = os.path.join(build.OUT_DIR, "host_pages.cpp.o")
    exe = str(tmp_path / "host_pages_check")
    inc = build._cuda_include(build._nvcc())
    r = subprocess.run([gxx, "-O2", "-std=c++17", "-I" + inc, os.path.join(HERE, "host_pages_check.cpp"), obj, "-o", exe,
                        "-lpthread"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
