"""Launch plans shared by handles of different block sizes (csrc/launch_plan.h) against a fake attribute, from threads,
under ThreadSanitizer where the compiler has it."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pv2013_gb300", "csrc")


@pytest.mark.parametrize("flags", [[], ["-fsanitize=thread"]])
def test_launch_plans(tmp_path, flags):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "check")
    cmd = ["g++", "-std=c++17", "-O1", "-g", "-pthread", *flags, "-I" + CSRC,
           os.path.join(HERE, "launchplan", "launch_plan_check.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    if flags and r.returncode != 0:
        pytest.skip("ThreadSanitizer not available")
    assert r.returncode == 0, r.stderr[-3000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    if flags and "unexpected memory mapping" in run.stderr:
        pytest.skip("ThreadSanitizer cannot run here")
    assert run.returncode == 0 and "launch plans ok" in run.stdout, (run.stdout[-2000:], run.stderr[-3000:])
