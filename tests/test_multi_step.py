"""Several time steps per pass over memory (kernels_multi.cu) against the
one-step kernels. A run takes the passes when it is long enough and one-step
launches otherwise, so the same steps taken one by one give the reference: the
populations, the other buffer and the fields must be the same bits. Sizes:
below one strip of 64 columns, strips that wrap around odd and even widths,
last strips of one pair or one column, grids of fewer rows than warps, with
body forces, FP32 and FP16 storage."""
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
@pytest.mark.parametrize("nx,ny", [(8, 8), (57, 9), (64, 8), (112, 31), (113, 30), (300, 201), (255, 129),
                                   (760, 200), (1031, 1023), (2048, 1030)])
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
