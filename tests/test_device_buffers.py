"""Growth of the device buffers where memory runs out, and the arrays too far apart
for one two-dimensional copy (tests/cpp/device_buffers.cpp, on the CPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ladds_b200", "csrc")


def test_buffer_in_hand_outlives_a_failed_growth(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "device_buffers")
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-I", CSRC,
                        os.path.join(HERE, "cpp", "device_buffers.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "device_buffers: ok" in r.stdout, r.stdout + r.stderr
