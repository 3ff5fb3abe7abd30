"""When a case with walls is set up for passes of several steps: not for the first
few steps asked of it, which would not pay for its plan, buffers and graph, but
after them, in one run or in several; what lbm_gpu_launch_stats says of it; and
every kind of wall and edge in runs long enough to take the passes."""
import pytest

from conftest import same
from lbc_gb300 import cases

pytestmark = pytest.mark.gpu
FIELDS = ("f", "f_new", "rho", "u", "v")


def _cavity():
    from lbc_gb300 import F32_SHIFTED, GpuSolver
    case, st = cases.cavity_moving_wall(1500, 0.1, 300.0)
    s = GpuSolver(case, F32_SHIFTED)
    s.set_state(st)
    return s


def _launches(s, n):
    before = s.launch_stats()[0]
    s.run(n)
    return s.launch_stats()[0] - before


def test_first_steps_are_taken_one_at_a_time():
    # special nodes and clean pairs: two kernels a step, five for four steps in passes
    s = _cavity()
    assert _launches(s, 50) >= 2 * 49
    assert _launches(s, 400) <= 1.4 * 400
    s.close()
    s = _cavity()
    assert _launches(s, 400) <= 1.4 * 400
    s.close()
    s = _cavity()
    assert _launches(s, 34) >= 2 * 33
    for _ in range(5):
        s.run(34)
    assert _launches(s, 34) <= 1.6 * 34
    s.close()


def test_same_bits_before_and_after():
    a, b = _cavity(), _cavity()
    for n in (50, 90, 300, 41):
        a.run(n)
    for _ in range(481):
        b.run(1)
    x, y = a.get_state(), b.get_state()
    for fld in FIELDS:
        assert same(getattr(x, fld), getattr(y, fld)), fld
    a.close()
    b.close()


def test_batch_first_steps_are_taken_one_at_a_time():
    """Two batches of the same cases, the second built when they have their plans."""
    from lbc_gb300 import F32_SHIFTED, GpuBatch, GpuSolver
    built = [cases.cylinder_wake(1500, 1000, D=60.0, xc=300.0, yc=500.0), cases.cavity_moving_wall(1700, 0.1, 300.0)]

    def solvers():
        out = []
        for case, st in built:
            s = GpuSolver(case, F32_SHIFTED)
            s.set_state(st)
            out.append(s)
        return out

    together, alone = solvers(), solvers()
    for runs in ((40, 90, 200), (80,)):
        b = GpuBatch(together)
        for n in runs:
            b.run(n)
        b.close()
    for x, y in zip(together, alone):
        for _ in range(410):
            y.run(1)
        got, want = x.get_state(), y.get_state()
        for fld in FIELDS:
            assert same(getattr(got, fld), getattr(want, fld)), fld


def _stage_periodic():
    # a periodic entry behind another: it reads the opposite edge after the collision
    case, st = cases.cylinder_golden(33)[:2]
    case.bcs = [b for b in case.bcs if not b.name.startswith("periodic")] + [cases.BC("periodic_y", 0, None, None)]
    return case, st


def _porous():
    import numpy as np
    case, st = cases.taylor_green(1200, 1000)
    case.solid_mask[::6, ::6] = 1  # more than an eighth of the nodes beside a solid one
    return case, st


@pytest.mark.parametrize("name,storage,want", [
    ("cavity", "f32", 4), ("periodic", "f32", 4), ("cavity", "f64", 1), ("edge_periodic", "f32", 1), ("porous", "f32", 1)])
def test_launch_stats_reports_the_passes_taken(name, storage, want):
    from lbc_gb300 import GpuSolver, STORAGE
    case, st = {"cavity": lambda: cases.cavity_moving_wall(1500, 0.1, 300.0), "periodic": lambda: cases.taylor_green(1200, 1000),
                "edge_periodic": _stage_periodic, "porous": _porous}[name]()
    s = GpuSolver(case, STORAGE[storage])
    s.set_state(st)
    assert case.nodes >= 1 << 20 and s.launch_stats()[1] == want
    s.run(200)
    assert s.launch_stats()[1] == want
    s.close()


# (with 1024 steps asked for below 1.3 M nodes, with 192 above)
LONG = [(n, "f32", 1060) for n in ("wake", "cavity", "golden", "open", "blocks", "box_large", "boxblock_large", "duct_large",
                                   "open_large", "golden_large")]
LONG += [("wake4", "f32", 230), ("wake4", "f16", 230), ("cavity4", "f32", 230), ("cavity_f16", "f16", 230)]


@pytest.mark.parametrize("hist", [False, True])
@pytest.mark.parametrize("name,storage,first", LONG)
def test_walls_and_edges_in_long_runs(name, storage, first, hist):
    """As test_multi_step's cases: passes entered and left twice, against single steps."""
    import numpy as np
    from lbc_gb300 import GpuSolver, STORAGE, impedance as imp
    from test_multi_step import _walls
    duct = None
    if name.startswith("open"):
        case, st = cases.cylinder_wake(*((1500, 760) if name == "open_large" else (900, 400)), D=40.0, xc=300.0, yc=200.0,
                                       u_max=0.05, Re=60.0)
        case.solid_mask[0] = case.solid_mask[-1] = 0
    elif name in ("box_large", "boxblock_large"):  # several groups of edges
        case, st = cases.all_regularized_box(1210, 900)
        case.omega_eff[:] = 1 / 0.8
        if name == "boxblock_large":
            case.solid_mask[200:240, 300:360] = 1
    elif name == "duct_large":
        duct = imp.LinerParams(2100, 520, 0.2, 1.0 * imp.CS, 5e-3, 0.05)
        case, st = imp.liner_duct(duct)
    elif name == "golden_large":
        case, st = cases.cylinder_golden(33)[:2]
        st = cases.random_state(case, 7)
    elif name == "cavity_f16":
        case, st = cases.cavity_moving_wall(1690, 0.1, 300.0)
    else:
        (case, st), _ = _walls(name)
        st = cases.random_state(case, 7)
    if hist and (duct is not None or not case.solid_mask.any()):
        pytest.skip("no force to record")
    pair = []
    for _ in range(2):
        s = GpuSolver(case, STORAGE[storage])
        if duct is not None:
            s.set_impedance_wall(imp.LINER_ENTRY, *imp.liner_arrays(duct), imp.TRACKED_OMEGAS, 1.0, imp.MEAN_RATE, 500)
        if hist:
            s.enable_force_history(1200)
        s.set_state(st)
        pair.append(s)
    a, b = pair
    assert a.launch_stats()[1] > 1
    for n in (first, 2, 91):
        a.run(n)
    for _ in range(first + 93):
        b.run(1)
    assert a.launch_stats()[0] < 0.8 * b.launch_stats()[0]
    x, y = a.get_state(), b.get_state()
    assert np.isfinite(x.rho[case.solid_mask == 0]).all()
    for fld in FIELDS:
        assert same(getattr(x, fld), getattr(y, fld)), fld
    assert a.forces() == b.forces()
    if hist:
        assert np.array_equal(a.force_history(1200), b.force_history(1200))
    if duct is not None:
        for p, q in zip(a.impedance_readback(imp.LINER_ENTRY), b.impedance_readback(imp.LINER_ENTRY)):
            assert np.array_equal(p, q)
    a.close()
    b.close()


@pytest.mark.parametrize("name", ["ducts", "mix"])
def test_batch_passes_in_long_runs(name):
    """As test_multi_step's batches: passes taken in the first and the second run."""
    import numpy as np
    from lbc_gb300 import F32_SHIFTED, GpuBatch, GpuSolver, impedance as imp
    from test_multi_step import _batch_cases
    built = _batch_cases(name)

    def solvers():
        out = []
        for (case, st), duct in built:
            s = GpuSolver(case, F32_SHIFTED)
            if duct is not None:
                s.set_impedance_wall(imp.LINER_ENTRY, *imp.liner_arrays(duct), imp.TRACKED_OMEGAS, 1.0, imp.MEAN_RATE, 500)
            s.set_state(st)
            out.append(s)
        return out

    together, alone = solvers(), solvers()
    held = sum(s.info().device_bytes for s in together)
    b = GpuBatch(together)
    b.run(170)
    assert sum(s.info().device_bytes for s in together) > 1.2 * held  # the buffers of passes
    b.run(38)
    for n, (x, y, (_, duct)) in enumerate(zip(together, alone, built)):
        for _ in range(208):
            y.run(1)
        got, want = x.get_state(), y.get_state()
        for fld in FIELDS:
            assert same(getattr(got, fld), getattr(want, fld)), (n, fld)
        assert same(np.array(x.forces()), np.array(y.forces()))
        if duct is not None:
            for p, q in zip(x.impedance_readback(imp.LINER_ENTRY), y.impedance_readback(imp.LINER_ENTRY)):
                assert np.array_equal(p, q)
    b.close()


@pytest.mark.parametrize("storage,kind,nx,ny,want", [
    ("f32", "vortex", 128, 4505, 1), ("f32", "vortex", 512, 1126, 1), ("f32", "vortex", 2048, 281, 4), ("f32", "vortex", 256, 1638, 2),
    ("f32", "vortex", 128, 3276, 1), ("f32", "vortex", 256, 6144, 4), ("f32", "vortex", 100, 5767, 4), ("f32", "channel", 256, 2252, 2),
    ("f32", "channel", 512, 2150, 1), ("f32", "cavity", 724, 724, 1), ("f32", "cavity", 533, 533, 2), ("f32", "lid", 533, 533, 1),
    ("f32", "lid", 1050, 1050, 4), ("f32", "cylinder", 1068, 267, 2), ("f32", "cylinder", 1492, 373, 1), ("f16", "vortex", 256, 8601, 1), ("f16", "vortex", 1024, 2150, 1),
    ("f16", "vortex", 4096, 1024, 4), ("f16", "cavity", 1450, 1450, 1)])
def test_shapes_that_leave_lanes_idle(storage, kind, nx, ny, want):
    """Passes only where their strips fill about as many lanes as the one-step
    kernel's blocks, or the grid is large enough not to mind."""
    from lbc_gb300 import GpuSolver, STORAGE
    case = {"vortex": lambda: cases.taylor_green(nx, ny), "channel": lambda: cases.poiseuille(nx, ny, 0.8, 1e-6),
            "cavity": lambda: cases.cavity_moving_wall(nx, 0.1, 300.0), "lid": lambda: cases.cavity_zouhe(nx, 0.1, 300.0),
            "cylinder": lambda: cases.cylinder_wake(nx, ny, D=ny / 8, xc=nx / 4, yc=ny / 2)}[kind]()[0]
    s = GpuSolver(case, STORAGE[storage])
    assert s.launch_stats()[1] == want
    s.close()
