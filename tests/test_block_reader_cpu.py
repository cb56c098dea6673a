"""The threaded block reader of the device STL reader (csrc/block_reader.h) against a destination that refuses pinned
memory, a reader or a copy; with AddressSanitizer where the compiler has it."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "pv2013_gb300", "csrc")


@pytest.mark.parametrize("flags", [[], ["-fsanitize=address,undefined", "-fno-sanitize-recover=all"]])
def test_block_reader(tmp_path, flags):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", *flags, "-I" + CSRC,
                        os.path.join(HERE, "blockreader", "block_reader_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    if flags and r.returncode != 0:
        pytest.skip("AddressSanitizer not available")
    assert r.returncode == 0, r.stderr[-3000:]
    run = subprocess.run([exe, str(tmp_path)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and "block reader ok" in run.stdout, (run.stdout[-2000:], run.stderr[-3000:])
