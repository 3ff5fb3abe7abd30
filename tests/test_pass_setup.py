"""When a case with walls is set up for passes of several steps: not in the first
few steps asked of it, which would not pay for its plan, buffers and graph, but
after them, in one run or in several; and what lbm_gpu_launch_stats says of it."""
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
    for _ in range(4):
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
    for runs in ((40, 90, 200), (60,)):
        b = GpuBatch(together)
        for n in runs:
            b.run(n)
        b.close()
    for x, y in zip(together, alone):
        for _ in range(390):
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
