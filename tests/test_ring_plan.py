"""The rings a run asks for, and those it falls back to when their memory cannot be had, checked on the host by
tests/ring_plan_check.cpp."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_each_fallback_asks_for_less(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "ring_plan_check")
    r = subprocess.run([gxx, "-O2", "-std=c++17", "-Wall", os.path.join(HERE, "ring_plan_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
