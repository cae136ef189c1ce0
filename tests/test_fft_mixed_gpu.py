"""FFTSolver2D and FFTSolver3D on lengths that are not powers of two, against
the oracle: every radix of the mixed-radix transform (primes to 31, 9, 8, 4, 2),
repeated radices, the thread counts' edges, and lengths with a prime above 31,
which the chirp-z kernels take.  FP64 <= 1e-10 relative L2; FP32 <= 1e-4 of the
intensity."""
import numpy as np
import pytest

from oracle import pyoracle as po
from paxpro_b200 import workloads as wl

pytestmark = pytest.mark.gpu

FP64_TOL = 1e-10
FP32_INT_TOL = 1e-4


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _int_rel(a, b):
    return _rel(np.abs(a) ** 2, np.abs(b) ** 2)


@pytest.mark.parametrize("n,precision", [
    (9, 0), (12, 0), (17 * 2, 0), (19 * 27, 0), (23 * 8, 0), (29 * 4, 0), (31 * 31, 0),
    (7 * 11 * 13, 0), (400, 0), (401, 0), (405, 0), (13 * 13 * 5, 0), (4095, 0), (37 * 4, 0),
    (19 * 27, 1), (1000, 1), (31 * 29, 1), (401, 1), (4095, 1)])
def test_fft2d_lengths(n, precision):
    import paxpro_b200 as pxp
    xmin, xmax, nsteps = -250.0, 250.0, 20
    dx = wl.step_for_nodes(xmin, xmax, n)
    x = wl.coords(xmin, dx, n)
    u0 = np.exp(-((x - 7.0) / 90.0) ** 2) * np.exp(1j * 4e-3 * x)
    d, b = wl.Waveguide(core_half_width=60.0, ramp_points=min(25, n // 8)).tables(x)
    g = po.grid(xmin, xmax, dx, 0.0, nsteps * 1000.0, 1000.0, wl.K)
    _, ref = po.fft2d_run(g, po.MaterialSpec(po.MAT_XTABLE, delta_table=d, beta_table=b), u0, nsteps, 5)
    with pxp.Solver(pxp.ProblemSpec(kind=pxp.FFT_SOLVER_2D, x=pxp.Disc(xmin, xmax, dx),
                                    z=pxp.Disc(0.0, nsteps * 1000.0, 1000.0), wavenumber=wl.K,
                                    precision=precision, save_every=5)) as s:
        s.set_material_table(d, b)
        s.set_initial_conditions(u0)
        s.step(7)
        s.step(nsteps - 7)
        saves = [s.get_saved(i) for i in range(s.num_saved())]
    assert len(saves) == len(ref) == 4
    for a, r in zip(saves, ref):
        assert (_int_rel(a, r) <= FP32_INT_TOL) if precision else (_rel(a, r) <= FP64_TOL)


@pytest.mark.parametrize("n,precision,absorber", [
    (12, 0, False), (93, 0, False), (155, 0, True), (391, 0, False), (403, 0, False), (700, 0, False),
    (702, 0, False), (74, 0, False), (95, 1, True), (406, 1, False), (704, 1, False), (74, 1, False)])
def test_fft3d_lengths(n, precision, absorber):
    import paxpro_b200 as pxp
    L, nsteps = 1000.0, 4
    dx = wl.step_for_nodes(-L / 2, L / 2, n)
    x = wl.coords(-L / 2, dx, n)
    gx = np.exp(-((x - 30.0) / 350.0) ** 2) * np.exp(1j * 1e-3 * x)
    u0 = np.asfortranarray(gx[:, None] * gx[None, :])
    sph = [(20.0, -30.0, 4000.0, 180.0, 4.5e-5, 3.6e-6), (-60.0, 40.0, 3000.0, 1500.0, 2e-6, 1e-7)]
    aw, ad = (0.1 * L, 0.05 * L) if absorber else (0.0, 0.0)
    g = po.grid(-L / 2, L / 2, dx, 0.0, nsteps * 2000.0, 2000.0, wl.K)
    _, ref = po.fft3d_run(g, po.MaterialSpec(po.MAT_SPHERES, spheres=sph), u0, nsteps, 1, aw, ad)
    with pxp.Solver(pxp.ProblemSpec(kind=pxp.FFT_SOLVER_3D, x=pxp.Disc(-L / 2, L / 2, dx),
                                    y=pxp.Disc(-L / 2, L / 2, dx),
                                    z=pxp.Disc(0.0, nsteps * 2000.0, 2000.0), wavenumber=wl.K,
                                    precision=precision, save_every=1, absorber_width=aw,
                                    absorber_damping=ad)) as s:
        s.set_material_spheres([pxp.Sphere(*sp) for sp in sph])
        s.set_initial_conditions(u0)
        s.step(nsteps)
        saves = [s.get_saved(i) for i in range(s.num_saved())]
    assert len(saves) == len(ref) == nsteps
    for a, r in zip(saves, ref):
        assert (_int_rel(a, r) <= FP32_INT_TOL) if precision else (_rel(a, r) <= FP64_TOL)
