"""The pixel range of a gridding row (bsoft_b200/csrc/row_range.h), compiled here
with g++ and checked against the FP64 bounds over random views and views a hair
off an axis, whose bounds lie beyond any integer (tests/row_range_check.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_sure_ranges_are_the_fp64_ones(tmp_path):
    exe = str(tmp_path / "row_range_check")
    subprocess.run(["g++", "-O1", "-fwrapv", "-std=c++17", "-o", exe, os.path.join(HERE, "row_range_check.cpp")],
                   check=True)
    r = subprocess.run([exe, "2000000"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    rows, sure, empty, wrong = (int(v) for v in r.stdout.split()[1::2])
    assert wrong == 0 and sure > 0.9 * rows and 0.1 * rows < empty < 0.9 * rows
