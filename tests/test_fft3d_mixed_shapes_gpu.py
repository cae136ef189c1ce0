"""FFTSolver3D's mixed-radix line passes at the launch shapes of large grids (128
and 256 threads a line, with and without a prime above 13, both precisions), two
steps through a z-invariant medium, against the same split step with numpy's
transforms: FP64 <= 1e-10 relative L2, FP32 <= 1e-4 of the intensity."""
import numpy as np
import pytest

from paxpro_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,precision", [(701 + 1, 0), (713, 0), (1265, 1), (1364, 1), (2700, 0), (2697, 0),
                                         (2697, 1), (2704, 0), (2728, 1)])
def test_large_line_shapes(n, precision):
    import paxpro_b200 as pxp
    half, dz, steps = 500.0, 2000.0, 2
    dx = wl.step_for_nodes(-half, half, n)
    x = wl.coords(-half, dx, n)
    gx = np.exp(-((x - 30.0) / 350.0) ** 2) * np.exp(1j * 1e-3 * x)
    gy = np.exp(-((x + 60.0) / 300.0) ** 2)
    u0 = gy[:, None] * gx[None, :]  # [row: y][column: x]
    inside = ((x + 60.0)[:, None] ** 2 + (x - 40.0)[None, :] ** 2) < 200.0 ** 2
    delta, beta = np.where(inside, 4.5e-5, 0.0), np.where(inside, 3.6e-6, 0.0)
    with pxp.Solver(pxp.ProblemSpec(kind=pxp.FFT_SOLVER_3D, x=pxp.Disc(-half, half, dx),
                                    y=pxp.Disc(-half, half, dx), z=pxp.Disc(0.0, steps * dz, dz),
                                    wavenumber=wl.K, precision=precision)) as s:
        s.set_material_table(delta, beta)
        s.set_initial_conditions(u0)
        s.step(steps)
        got = s.get_last_solution()
    i = np.arange(n)
    f2 = (2.0 * np.pi * np.where(i > n // 2, n - i, i) / (dx * n)) ** 2
    prop = np.exp(-0.5j * dz / wl.K * (f2[:, None] + f2[None, :]))
    t = np.exp(-wl.K * dz * (beta + 1j * delta))
    u = u0
    for _ in range(steps):
        u = np.fft.ifft2(np.fft.fft2(u) * prop) * t
    if precision:
        got, u = np.abs(got) ** 2, np.abs(u) ** 2
    assert np.linalg.norm(got - u) <= (1e-4 if precision else 1e-10) * np.linalg.norm(u)
