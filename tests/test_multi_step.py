"""Several time steps per pass over memory (kernels_multi.cu) against the
one-step kernels. A run takes the passes when it is long enough and one-step
launches otherwise, so the same steps taken one by one give the reference: the
populations, the other buffer and the fields must be the same bits. Sizes:
strips that wrap around odd and even widths, last strips of one pair or one
column, few rows, on both sides of the sizes from which passes take two and
four steps, with body forces, FP32 and FP16 storage."""
import numpy as np
import pytest

from lbc_gb300 import cases

pytestmark = pytest.mark.gpu
FIELDS = ("f", "f_new", "rho", "u", "v")


def _solver(storage, nx, ny, force):
    from lbc_gb300 import GpuSolver, STORAGE
    case, _ = cases.taylor_green(nx, ny)
    case.Fx, case.Fy = (1e-5, -2e-5) if force else (0.0, 0.0)
    s = GpuSolver(case, STORAGE[storage])
    s.set_state(cases.random_state(case, 5))
    return s


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("nx,ny", [(8, 8), (300, 201), (760, 360), (601, 450), (91, 3000), (32768, 8), (90, 6000),
                                   (1031, 1023), (57, 9300), (168, 18600), (2049, 1030), (65536, 33)])
def test_passes_match_single_steps(storage, nx, ny):
    for force in (False, True):
        a, b = _solver(storage, nx, ny, force), _solver(storage, nx, ny, force)
        for n in (41, 8, 18):
            a.run(n)
        for _ in range(67):
            b.run(1)
        x, y = a.get_state(), b.get_state()
        for fld in FIELDS:
            assert np.array_equal(getattr(x, fld), getattr(y, fld)), (force, fld)
        a.close()
        b.close()


def test_probes_see_every_step():
    """A case with per-step records is stepped one at a time."""
    a, b = _solver("f32", 300, 64, False), _solver("f32", 300, 64, False)
    a.set_probes([(3, 5), (299, 63)], 40)
    a.run(40)
    h = a.probe_history(40)
    b.run(40)
    assert h.shape == (40, 2, 3) and len(np.unique(h[:, 0, 1])) > 30
    for fld in FIELDS:
        assert np.array_equal(getattr(a.get_state(), fld), getattr(b.get_state(), fld)), fld


def _walls(name):
    from lbc_gb300 import impedance as imp
    if name == "wake":
        return cases.cylinder_wake(1029, 257, D=20.0, xc=270.0, yc=127.0, u_max=0.05, Re=60.0, seed=3), None
    if name == "wake4":
        return cases.cylinder_wake(2051, 1544, D=64.0, xc=520.0, yc=500.0, u_max=0.05, Re=60.0, seed=3), None
    if name == "cavity":
        return cases.cavity_moving_wall(513, 0.1, 300.0), None
    if name == "cavity4":
        return cases.cavity_moving_wall(1450, 0.1, 300.0), None
    if name == "box":
        return cases.all_regularized_box(600, 450), None
    if name == "open":  # inlet and outlet between open rows: neighbours with slots of their own
        case, st = cases.cylinder_wake(900, 400, D=40.0, xc=300.0, yc=200.0, u_max=0.05, Re=60.0)
        case.solid_mask[0] = case.solid_mask[-1] = 0
        return (case, st), None
    if name == "boxblock":  # several groups of edges around a body
        case, st = cases.all_regularized_box(610, 450)
        case.solid_mask[200:240, 300:360] = 1
        return (case, st), None
    if name == "golden":
        return cases.cylinder_golden(17)[:2], None
    if name == "blocks":  # obstacles across both periodic edges, body force
        case, st = cases.taylor_green(641, 450)
        for i, j in ((0, 0), (300, 449), (640, 200), (100, 100), (101, 109)):
            case.solid_mask[j:j + 6, i:i + 8] = 1
        case.Fx, case.Fy = 1e-6, -2e-6
        return (case, st), None
    p = imp.LinerParams(2100, 130, 0.2, 1.0 * imp.CS, 5e-3, 0.05)
    return imp.liner_duct(p), p


@pytest.mark.parametrize("storage", ["f32", "f16"])
@pytest.mark.parametrize("name", ["wake", "wake4", "cavity", "cavity4", "box", "boxblock", "open", "golden", "blocks",
                                  "duct"])
def test_walls_and_edges_match_single_steps(storage, name):
    """Cases with a flag word: cut links, moving walls, Zou-He, convective,
    regularized and impedance edges, slots off open edges, odd sizes, with and
    without a force history; runs that enter and leave the passes twice."""
    from lbc_gb300 import GpuSolver, STORAGE, impedance as imp
    (case, st), duct = _walls(name)
    if duct is None:
        st = cases.random_state(case, 7)
    for hist in (False, True):
        pair = []
        for _ in range(2):
            s = GpuSolver(case, STORAGE[storage])
            if duct is not None:
                s.set_impedance_wall(imp.LINER_ENTRY, *imp.liner_arrays(duct), imp.TRACKED_OMEGAS, 1.0, imp.MEAN_RATE, 500)
            if hist and case.solid_mask.any():
                s.enable_force_history(100)
            s.set_state(st)
            pair.append(s)
        a, b = pair
        for n in (41, 2, 44):
            a.run(n)
        for _ in range(87):
            b.run(1)
        x, y = a.get_state(), b.get_state()
        for fld in FIELDS:
            assert np.array_equal(getattr(x, fld), getattr(y, fld), equal_nan=True), (hist, fld)
        assert a.forces() == b.forces()
        if hist and case.solid_mask.any():
            assert np.array_equal(a.force_history(100), b.force_history(100))
        if duct is not None:
            for p, q in zip(a.impedance_readback(imp.LINER_ENTRY), b.impedance_readback(imp.LINER_ENTRY)):
                assert np.array_equal(p, q)
        a.close()
        b.close()


def _batch_cases(name):
    from lbc_gb300 import impedance as imp
    if name == "ducts":
        return [(imp.liner_duct(p), p) for p in imp.sample_liners(24, 11)]
    built = [cases.cylinder_wake(2501, 701, D=40.0, xc=400.0, yc=200.0, u_max=0.05, Re=60.0), cases.taylor_green(1401, 850),
             cases.cavity_moving_wall(900, 0.1, 300.0), cases.poiseuille(1500, 633, 0.8, 1e-5),
             cases.cylinder_golden(12)[:2], cases.taylor_green(640, 33)]
    return [((c, cases.random_state(c, n)), None) for n, (c, _) in enumerate(built)]


@pytest.mark.parametrize("name", ["ducts", "mix"])
def test_batch_passes_match_cases_alone(name):
    """A batch large enough for passes of several steps (with walls, links,
    edges, impedance walls, periodic cases of odd width, with and without body
    forces) leaves every case as single steps alone do, over two runs."""
    from lbc_gb300 import F32_SHIFTED, GpuBatch, GpuSolver, impedance as imp
    built = _batch_cases(name)
    assert sum(c.nodes for (c, _), _ in built) >= 1 << 22

    def solvers():
        out = []
        for (case, st), duct in built:
            s = GpuSolver(case, F32_SHIFTED)
            if duct is not None:
                s.set_impedance_wall(imp.LINER_ENTRY, *imp.liner_arrays(duct), imp.TRACKED_OMEGAS, 1.0, imp.MEAN_RATE, 500)
            s.set_state(st)
            out.append(s)
        return out

    mixed, alone = solvers(), solvers()
    b = GpuBatch(mixed)
    b.run(47)
    b.run(38)
    for n, (x, y, (_, duct)) in enumerate(zip(mixed, alone, built)):
        for _ in range(85):
            y.run(1)
        got, want = x.get_state(), y.get_state()
        for fld in FIELDS:
            assert np.array_equal(getattr(got, fld), getattr(want, fld), equal_nan=True), (n, fld)
        assert x.forces() == y.forces()
        if duct is not None:
            for p, q in zip(x.impedance_readback(imp.LINER_ENTRY), y.impedance_readback(imp.LINER_ENTRY)):
                assert np.array_equal(p, q)
    b.close()
