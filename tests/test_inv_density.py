"""The reciprocal of the density in the FP32 collision (shifted_math.cuh) for
every float: as the intrinsic rounds it, 0 for an infinite density, and right to
the last subnormal bit above 2^126."""
import os
import subprocess

import numpy as np
import pytest

from lbc_gb300 import cases

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_every_density(tmp_path):
    from lbc_gb300.build import ARCH, CSRC, nvcc
    exe = str(tmp_path / "inv")
    subprocess.run([nvcc(), "-std=c++17", "-O3", "--fmad=false", "-I", CSRC] + ARCH +
                   [os.path.join(HERE, "inv_density_device.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
    assert r.stdout.split() == ["0", str((1 << 24) - 1)]


@pytest.mark.parametrize("exponent", [120, 125.5, 126.5])
def test_velocity_at_huge_densities(exponent):
    """A uniform stream at a density near the top of FP32: u = j / rho."""
    from lbc_gb300 import F32_SHIFTED, GpuSolver
    case, st = cases.taylor_green(64, 32)
    rho = np.full((32, 64), 2.0 ** exponent)
    u, v = np.full_like(rho, 0.01), np.full_like(rho, -0.02)
    st = cases.equilibrium_state(rho, u, v)
    s = GpuSolver(case, F32_SHIFTED)
    s.set_state(st)
    s.run(1)
    got = s.get_state()
    s.close()
    # the momentum is a sum of terms up to rho / 9, each right to 2^-24, and the
    # subnormal reciprocal adds 2^-22 of u: a few 1e-7
    assert np.max(np.abs(got.u - 0.01)) <= 3e-6 and np.max(np.abs(got.v + 0.02)) <= 3e-6
