"""The search's division of tiles over the SMs (bsoft_b200/csrc/search_runs.h),
compiled here with g++ (tests/search_runs_check.cpp): every tile once, every
slot of partial results filled once, and on short panels no CTA with more tiles
than when they are dealt out in groups of ten M tiles by 15 ranges."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_divisions_cover_every_tile(tmp_path):
    exe = str(tmp_path / "search_runs_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "search_runs_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.endswith(" wrong 0 more 0\n"), r.stdout
