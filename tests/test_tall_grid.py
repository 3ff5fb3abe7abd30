"""Grids of more rows than a launch of 64 x 2 blocks has (2 x 65535): the FP64
step takes taller blocks there, and the tuner leaves out the shapes that do not
reach the last row."""
import pytest

from conftest import same
from lbc_gb300 import cases

pytestmark = pytest.mark.gpu
FIELDS = ("f", "f_new", "rho", "u", "v")


@pytest.mark.parametrize("ny", [131070, 131071, 140003])
def test_tall_fp64_grid_matches_oracle(oracle, ny):
    from lbc_gb300 import F64, GpuSolver
    case, _ = cases.taylor_green(6, ny)
    st = cases.random_state(case, 2)
    s = GpuSolver(case, F64)
    s.set_state(st)
    s.run(4)
    got = s.get_state()
    s.close()
    oracle.run(case, st, 4)
    for fld in FIELDS:
        assert same(getattr(got, fld), getattr(st, fld)), fld


@pytest.mark.parametrize("storage", ["f64", "f32"])
def test_tuner_on_a_tall_grid(storage):
    from lbc_gb300 import GpuSolver, STORAGE
    case, _ = cases.taylor_green(6, 140003)
    st = cases.random_state(case, 2)
    out = []
    for tune in (0, 1):
        s = GpuSolver(case, STORAGE[storage])
        s.set_autotune(tune)
        s.set_state(st)
        s.run(40)
        out.append(s.get_state())
        s.close()
    for fld in FIELDS:
        assert same(getattr(out[0], fld), getattr(out[1], fld)), fld
