"""The register-resident radix-8 FFTSolver2D kernel at every size it takes
(less than a warp to 512 threads), with a medium sampled per step, fused flux
sums, saves and chunked calls, against the oracle: FP64 <= 1e-10, FP32 <= 1e-4 of
the intensity."""
import math

import numpy as np
import pytest

from oracle import pyoracle as po
from paxpro_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 128, 256, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("precision", [0, 1])
def test_radix8_sizes(n, precision):
    import paxpro_b200 as pxp
    xmin, xmax, dz, nsteps = -250.0, 250.0, 1000.0, 30
    dx = wl.step_for_nodes(xmin, xmax, n)
    x = wl.coords(xmin, dx, n)
    u0 = np.exp(-((x - 7.0) / 60.0) ** 2) * np.exp(1j * 4e-3 * x)
    d, b = wl.Waveguide(core_half_width=60.0, ramp_points=min(25, n // 8)).tables(x)
    g = po.grid(xmin, xmax, dx, 0.0, nsteps * dz, dz, wl.K)
    _, ref = po.fft2d_run(g, po.MaterialSpec(po.MAT_XTABLE, delta_table=d, beta_table=b), u0, nsteps, 10)
    a, e = n // 5, n - n // 4
    with pxp.Solver(pxp.ProblemSpec(kind=pxp.FFT_SOLVER_2D, x=pxp.Disc(xmin, xmax, dx),
                                    z=pxp.Disc(0.0, nsteps * dz, dz), wavenumber=wl.K,
                                    precision=precision, save_every=10)) as s:
        s.set_material_planes(np.tile(d, (nsteps, 1)), np.tile(b, (nsteps, 1)), 1, nsteps)
        s.set_initial_conditions(u0)
        s.step(11)
        s.set_flux_windows(12, np.full(nsteps - 11, a), np.full(nsteps - 11, e))
        s.step(nsteps - 11)
        saves = [s.get_saved(i) for i in range(s.num_saved())]
        flux = s.get_flux(12, nsteps - 11)
    assert len(saves) == len(ref) == 3
    for v, r in zip(saves, ref):
        if precision:
            iv, ir = np.abs(v) ** 2, np.abs(r) ** 2
            assert np.linalg.norm(iv - ir) <= 1e-4 * np.linalg.norm(ir)
        else:
            assert np.linalg.norm(v - r) <= 1e-10 * np.linalg.norm(r)
    w = np.abs(saves[-1][a:e + 1]) ** 2
    want = math.fsum(2.0 * w) - w[0] - w[-1]
    assert abs(flux[-1] - want) <= 1e-13 * want
