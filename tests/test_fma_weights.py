"""The fused multiply-add step (moments_fma, collide_fma) is what F64_FMA storage
takes with weights of lbc's pair symmetry that are not lbc's own (those take the
integer form). With such weights: walls, cut links, every Boundary kind, body
forces, open edges and odd widths within 1e-12 of the oracle, as
tests/test_fma64.py measures it; and cases of every arithmetic in one batch,
each as it is alone, bit for bit."""
import numpy as np
import pytest

import casezoo
from conftest import force_close, gross_force, same
from lbc_gb300 import cases
from test_fma64 import RTOL, _check, _run_fma

pytestmark = pytest.mark.gpu
FIELDS = ("f", "f_new", "rho", "u", "v")


def _other_weights(built):
    """The case with w0 a little above lbc's and w1..w4 below, from the
    equilibrium of those weights."""
    case, st = built
    case.w = case.w.copy()
    case.w[0] += 4e-3
    case.w[1:5] -= 1e-3
    f = cases.equilibrium(st.rho, st.u, st.v, case.w)
    return case, cases.State(f, f.copy(), st.rho, st.u, st.v)


def _omega(built):
    """The case with an omega of its own at every node."""
    case, st = built
    case.omega_eff = case.omega_eff * np.random.default_rng(8).uniform(0.9, 1.0, case.omega_eff.shape)
    return case, st


@pytest.mark.parametrize("omega", [False, True])
@pytest.mark.parametrize("name", [n for n, _, _ in casezoo.standard_cases()])
def test_every_edge_case(oracle, name, omega):
    built, steps = casezoo.build(name)
    case, st = _other_weights(_omega(built) if omega else built)
    hist = bool(case.solid_mask.any())
    got, h = _run_fma(case, st, steps, hist)
    fo = oracle.run(case, st, steps, record_forces=True)
    _check(case, got, st, name)
    if hist:
        mag = gross_force(case)
        assert force_close(h[:, 0], fo[:, 1], rtol=RTOL, scale=mag), name
        assert force_close(h[:, 1], fo[:, 0], rtol=RTOL, scale=mag), name


@pytest.mark.parametrize("storage", ["f64", "f64fma"])
@pytest.mark.parametrize("mixed", [False, True])
def test_batch_equals_alone(storage, mixed):
    """Alone in a batch (one arithmetic) and beside cases of lbc's weights."""
    from lbc_gb300 import GpuBatch, GpuSolver, STORAGE
    names = ["zoo_ibb", "taylor_green", "poiseuille", "cylinder_wake_small", "zoo_convective_chain"]

    def build():
        out = [_other_weights(casezoo.build(n)[0]) for n in names]
        return out + ([casezoo.build(n)[0] for n in names] if mixed else [])

    def solvers():
        out = []
        for case, st in build():
            s = GpuSolver(case, STORAGE[storage])
            if case.solid_mask.any():
                s.enable_force_history(50)
            s.set_state(st)
            out.append(s)
        return out

    together, alone = solvers(), solvers()
    b = GpuBatch(together)
    b.run(20)
    b.run(25)
    for n, (x, y) in enumerate(zip(together, alone)):
        y.run(45)
        got, want = x.get_state(), y.get_state()
        for fld in FIELDS:
            assert same(getattr(got, fld), getattr(want, fld)), (n, fld)
        assert x.forces() == y.forces(), n
    b.close()
