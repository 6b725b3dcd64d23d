"""Kernel limits are kept per device by CUDA, so they are set once for each
device a process uses, not once a process (the header compiles as plain C++)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ekman_bl_gb300", "csrc")


def test_once_per_device(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = tmp_path / "device_once_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-pthread", "-I", CSRC,
                    os.path.join(ROOT, "tests", "native", "device_once_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
