"""Column ranges of the voxelizer (csrc/column_range.h) on the CPU, grid sizes beyond 2^24 included."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pv2013_gb300", "csrc")


def test_last_column(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + CSRC,
                    os.path.join(HERE, "columnrange", "column_range_check.cpp"), "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0 and "column range ok" in run.stdout, run.stdout[-2000:]
