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


def _other_weights():
    """A periodic flow with weights that keep lbc's pair symmetry but are not
    lbc's: outside the integer form."""
    from lbc_gb300 import cases
    case, st = cases.taylor_green(48, 40, 0.04, 0.56)
    w = case.w.copy()
    w[0] += 4e-3
    w[1:5] -= 1e-3
    case.w = w
    f = cases.equilibrium(st.rho, st.u, st.v, w)
    return case, cases.State(f, f.copy(), st.rho, st.u, st.v)


@pytest.mark.gpu
@pytest.mark.parametrize("storage", ["f64", "f64fma"])
def test_other_weights_take_the_fp64_pipe(oracle, storage):
    """Weights the integer form does not serve, alone and in a batch with a
    case it does: F64 equals the oracle bit for bit, F64_FMA to 1e-12, and each
    case of the batch equals itself alone."""
    import numpy as np
    import casezoo
    from lbc_gb300 import GpuBatch, GpuSolver, STORAGE
    built = [_other_weights(), casezoo.build("cylinder_wake_small")[0], _other_weights()]
    alone, solvers = [], []
    for case, st in built:
        s = GpuSolver(case, STORAGE[storage])
        s.set_state(st)
        s.run(20)
        alone.append(s.get_state())
        s = GpuSolver(case, STORAGE[storage])
        s.set_state(st)
        solvers.append(s)
    GpuBatch(solvers).run(20)
    for s, a in zip(solvers, alone):
        got = s.get_state()
        for fld in ("f", "f_new", "rho", "u", "v"):
            assert np.array_equal(getattr(got, fld), getattr(a, fld), equal_nan=True), fld
    case, st = built[0]
    oracle.run(case, st, 20)
    for fld in ("f", "f_new", "rho", "u", "v"):
        a, b = getattr(alone[0], fld), getattr(st, fld)
        if storage == "f64":
            assert np.array_equal(a, b), fld
        else:
            assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b)), fld
