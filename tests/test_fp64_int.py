"""The integer form of the FP64 step (lbc_gb300/csrc/fp64_int.cuh) against the
plain FP64 operation sequence of lbc's moments and collision
(src/core/compute_macroscopic_fields.c:23-46, src/core/collision.c:24-38),
compiled here for the CPU: equal bit for bit on every node it accepts. The
nodes reach from quiescent flow to the ends of its ranges, with zero and tied
velocities, short mantissas (ties in every rounding), densities whose mantissa
is all ones, and body forces."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "lbc_gb300", "csrc")


@pytest.mark.parametrize("force", [0, 1, 2])
def test_integer_form_matches_fp64(tmp_path, force):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "fp64_int")
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-Wno-unknown-pragmas", "-I", CSRC,
                    os.path.join(HERE, "fp64_int_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe, "400000", str(force)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    nodes, wrong, refused = (int(x) for x in r.stdout.split()[-3:])
    assert wrong == 0, r.stdout
    # most of the sampled nodes are ordinary ones, which it must accept
    assert refused < nodes // 10, r.stdout
