"""The proposal network's weight-gradient row ranges fit the buffer of a larger network, checked on the host by
tests/mlp_ranges_check.cpp for every padded row count up to 65536."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_ranges_of_every_row_count_fit_the_partial_products(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "mlp_ranges_check")
    r = subprocess.run([gxx, "-O2", "-std=c++17", "-Wall", os.path.join(HERE, "mlp_ranges_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
