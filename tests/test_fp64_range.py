"""FP64 flows past the ranges of the integer form (fp64_int.cuh), alone in a warp,
in part of it and everywhere: speeds above 1/4 along the axes and the
diagonals, densities above 2 and below 9/16, populations below 2^-8 and
non-equilibrium parts above 2^-6, with walls, links, edges and a body force.
The same bits as the oracle. Six steps: with an outlet held at density 1 the
thin flow has left the numbers at twelve."""
import numpy as np
import pytest

import casezoo
from conftest import same
from lbc_gb300 import cases

pytestmark = pytest.mark.gpu
FIELDS = ("f", "f_new", "rho", "u", "v")


def _state(case, name):
    Ny, Nx = case.Ny, case.Nx
    rng = np.random.default_rng(6)
    rho = 1 + 0.01 * rng.uniform(-1, 1, (Ny, Nx))
    u, v = (0.05 * rng.uniform(-1, 1, (Ny, Nx)) for _ in range(2))
    x, y = np.arange(Nx)[None, :], np.arange(Ny)[:, None]
    if name == "fast":
        u = u + 0.3
    elif name == "fast_patch":
        u = np.where((x % 37 < 5) & (y % 11 < 3), 0.2, u)
        v = np.where((x % 37 < 5) & (y % 11 < 3), -0.2, v)
    elif name == "dense":
        rho = rho * 2.5
    elif name == "thin":
        rho = rho * 0.1
    elif name == "thin_patch":
        rho = np.where(x % 41 == 3, 0.4, rho)
    st = cases.equilibrium_state(rho, u, v)
    if name == "far":  # non-equilibrium parts up to 0.05
        st.f *= 1 + 0.2 * rng.uniform(-1, 1, st.f.shape)
        st.f_new = st.f.copy()
    return st


@pytest.mark.parametrize("name", ["fast", "fast_patch", "dense", "thin", "thin_patch", "far"])
@pytest.mark.parametrize("case_name", ["taylor_green", "poiseuille", "cylinder_golden_res2", "cylinder_wake_small"])
@pytest.mark.parametrize("batch", [False, True])
def test_out_of_range_nodes_match_oracle(oracle, case_name, name, batch):
    from lbc_gb300 import F64, GpuBatch, GpuSolver
    case, _ = casezoo.build(case_name)[0]
    st = _state(case, name)
    s = GpuSolver(case, F64)
    s.set_state(st)
    if batch:
        b = GpuBatch([s])
        b.run(6)
        b.close()
    else:
        s.run(6)
    got = s.get_state()
    s.close()
    oracle.run(case, st, 6)
    for fld in FIELDS:
        assert same(getattr(got, fld), getattr(st, fld)), fld
