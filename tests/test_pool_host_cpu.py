"""Device memory pool (emg_pool.cpp): builds tests/pool_check.cpp against the
library source, with the CUDA calls it makes replaced, and runs it."""

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_pool(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("needs g++")
    exe = tmp_path / "pool_check"
    src = os.path.join(ROOT, "emfem_b200", "csrc")
    subprocess.run([cxx, "-O2", "-std=c++17", "-pthread", "-I", src, "-I/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "pool_check.cpp"), os.path.join(src, "emg_pool.cpp"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
