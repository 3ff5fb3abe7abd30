"""Kernels of a step that run side by side (pdl.cuh): the edges or special nodes
of a step go first and its bulk kernel beside them, and the next step may start
only when both are done. On small grids the edges are the longer of the two, so
a step that started early would read a node before its edge was written. Runs
of many steps (captured graphs) against the same steps taken one by one, each
waited for, and in FP64 against the oracle, bit for bit, repeated."""
import numpy as np
import pytest

import casezoo
from conftest import same
from lbc_gb300 import cases

pytestmark = pytest.mark.gpu
FIELDS = ("f", "f_new", "rho", "u", "v")


def _case(name):
    if name == "zou_he_convective":
        return casezoo.build("cylinder_golden_res2")[0]
    if name == "regularized":
        return casezoo.build("cylinder_wake_small")[0]
    if name == "lid":
        return casezoo.build("cavity_zouhe")[0]
    return cases.all_regularized_box(40, 24)


@pytest.mark.parametrize("storage", ["f64", "f32"])
@pytest.mark.parametrize("name", ["zou_he_convective", "regularized", "lid", "box"])
@pytest.mark.parametrize("hist", [False, True])
def test_steps_wait_for_their_edges(oracle, name, storage, hist):
    from lbc_gb300 import GpuSolver, STORAGE
    case, st = _case(name)
    if hist and not case.solid_mask.any():
        pytest.skip("no walls: no force history")
    steps = 401
    states, forces = [], []
    for chunk in (steps, steps, 1):
        s = GpuSolver(case, STORAGE[storage])
        if hist:
            s.enable_force_history(steps)
        s.set_state(st)
        for _ in range(steps // chunk):
            s.run(chunk)
            s.forces()  # waits for the run
        states.append(s.get_state())
        forces.append(s.force_history(steps) if hist else s.forces())
        s.close()
    for got, f in zip(states[:2], forces[:2]):
        for fld in FIELDS:
            assert same(getattr(got, fld), getattr(states[2], fld)), fld
        assert np.array_equal(f, forces[2])
    if storage == "f64":
        oracle.run(case, st, steps)
        for fld in FIELDS:
            assert same(getattr(states[0], fld), getattr(st, fld)), fld


@pytest.mark.parametrize("storage", ["f32", "f16"])
def test_chained_steps_of_a_pass_see_each_other(storage):
    """The lists beside a pass follow each other while the one before still
    runs: buffer 2 is read by step 2 of a pass, written by step 3 and read
    again by step 4. Many passes against steps taken one by one."""
    from lbc_gb300 import GpuSolver, STORAGE
    case, _ = cases.cylinder_wake(3400, 620, D=90.0, xc=500.0, yc=310.0, u_max=0.05, Re=80.0)
    st = cases.random_state(case, 4)
    a, b = (GpuSolver(case, STORAGE[storage]) for _ in range(2))
    for s in (a, b):
        s.set_state(st)
    for n in (513, 1, 1286):
        a.run(n)
    for _ in range(1800):
        b.run(1)
    x, y = a.get_state(), b.get_state()
    for fld in FIELDS:
        assert same(getattr(x, fld), getattr(y, fld)), fld
    assert a.forces() == b.forces()
    a.close()
    b.close()
