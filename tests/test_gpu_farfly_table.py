"""The logarithm of the double-FP32 far field says so when a distance lies outside its table (fly_table.cpp)."""
import os
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.gpu
def test_distances_outside_the_log_table_are_reported(gpu, tmp_path):
    from h2weak_gb300 import buildlib
    lib = buildlib.build()
    exe = str(tmp_path / "fly_table")
    r = subprocess.run([buildlib.nvcc(), "-std=c++17", "--cudart", "shared", "-I", os.path.join(ROOT, "include"),
                        os.path.join(ROOT, "tests", "fly_table.cpp"), lib, "-o", exe,
                        "-Xlinker", "-rpath=" + os.path.dirname(lib)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
