"""The plan of a case's passes of several steps (lbc_gb300/csrc/near_plan.h): built
from the special nodes' runs, it is the one that the distance of every node gives,
on random walls, columns and blocks, with and without periodic axes, for odd and
even widths, compiled here for the CPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "lbc_gb300", "csrc")


def test_plan_matches_distances(tmp_path):
    from lbc_gb300.build import nvcc
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    include = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc()))), "include")
    exe = str(tmp_path / "near_plan")
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", CSRC, "-I", include, os.path.join(HERE, "near_plan_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe, "3000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
