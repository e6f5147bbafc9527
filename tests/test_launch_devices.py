"""Handles of several devices in one process: every launcher sets what a launch needs on the device it launches on.
The launchers run against a runtime that only keeps books (launch_devices.cpp); no GPU is used."""
import os
import subprocess

from conftest import ROOT


def test_launch_attributes_belong_to_the_device(tmp_path):
    from h2weak_gb300 import buildlib
    lib = buildlib.build()
    exe = str(tmp_path / "launch_devices")
    r = subprocess.run([buildlib.nvcc(), "-std=c++17", "--cudart", "shared", "-I", os.path.join(ROOT, "include"),
                        os.path.join(ROOT, "tests", "launch_devices.cpp"), lib, "-o", exe,
                        "-Xlinker", "--export-dynamic", "-Xlinker", "-rpath=" + os.path.dirname(lib)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
