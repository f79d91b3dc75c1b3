"""The order in which the device tries the phase lattices
(bsoft_b200/csrc/lattice.cu, lattice.h) gives the choice of the plain loops:
compiled here with g++ (tests/lattice_order_check.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="g++ not available")
def test_candidates_give_the_loops_choice(tmp_path):
    exe = str(tmp_path / "lattice_order_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-o", exe, os.path.join(HERE, "lattice_order_check.cpp")], check=True)
    r = subprocess.run([exe, "300"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("out_of_order 0 ") and r.stdout.endswith(" differ 0\n"), r.stdout
