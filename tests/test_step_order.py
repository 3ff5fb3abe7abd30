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
