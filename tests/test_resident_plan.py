"""Layouts of the resident kernel (csrc/resident_launch.h) checked on the host:
over 60,000 grids, HABC widths, orders and block counts, every region holds
the columns and rows its boundary rules read, fits the shared memory it is
given, and the exchange's sender and receiver agree on every message."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_INCLUDE = "/usr/local/cuda/include"


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INCLUDE), reason="needs g++ and the CUDA headers")
def test_resident_layouts(tmp_path):
    exe = tmp_path / "plan_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CUDA_INCLUDE, os.path.join(HERE, "resident_plan_check.cpp"),
                    "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
