"""CrankNicholson's two-sided solve (z-invariant media, Dirichlet ends) at every
launch shape, with fused flux sums and saves, against the oracle; and the wide
and narrow cluster forms of a launch (few or many problems) bit for bit."""
import math

import numpy as np
import pytest

from oracle import pyoracle as po
from paxpro_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _problem(n, nsteps, seed=0):
    xmin, xmax, dz = -250.0, 250.0, 500.0
    dx = wl.step_for_nodes(xmin, xmax, n)
    x = wl.coords(xmin, dx, n)
    rng = np.random.default_rng(seed)
    u0 = np.exp(-((x - rng.uniform(-9, 9)) / 60.0) ** 2) * np.exp(1j * 4e-3 * x)
    d, b = wl.Waveguide(core_half_width=rng.uniform(20, 60), ramp_points=min(25, n // 8)).tables(x)
    return xmin, xmax, dx, dz, u0, d, b


def _solver(pxp, n, nsteps, precision, save_every, seed=0):
    xmin, xmax, dx, dz, u0, d, b = _problem(n, nsteps, seed)
    s = pxp.Solver(pxp.ProblemSpec(kind=pxp.CRANK_NICHOLSON, x=pxp.Disc(xmin, xmax, dx),
                                   z=pxp.Disc(0.0, nsteps * dz, dz), wavenumber=wl.K,
                                   precision=precision, save_every=save_every))
    s.set_material_table(d, b)
    s.set_initial_conditions(u0)
    return s


@pytest.mark.parametrize("n,precision", [
    (64, 0), (65, 0), (128, 0), (255, 0), (512, 0), (513, 0), (1024, 0), (2048, 0), (2049, 0),
    (4096, 0), (4097, 0), (16000, 0), (64, 1), (1000, 1), (4096, 1), (8192, 1), (16384, 1)])
def test_two_sided_sizes(n, precision):
    import paxpro_b200 as pxp
    nsteps = 24
    xmin, xmax, dx, dz, u0, d, b = _problem(n, nsteps)
    g = po.grid(xmin, xmax, dx, 0.0, nsteps * dz, dz, wl.K)
    _, ref = po.cn2d_run(g, po.MaterialSpec(po.MAT_XTABLE, delta_table=d, beta_table=b), u0, nsteps, 8)
    a, e = n // 5, n - n // 4
    with _solver(pxp, n, nsteps, precision, 8) as s:
        s.step(9)
        s.set_flux_windows(10, np.full(nsteps - 9, a), np.full(nsteps - 9, e))
        s.step(nsteps - 9)
        saves = [s.get_saved(i) for i in range(s.num_saved())]
        flux = s.get_flux(10, nsteps - 9)
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


@pytest.mark.parametrize("n,count", [(4096, 38), (8192, 38), (16384, 19)])
def test_many_problems_take_the_narrow_form_with_the_same_bits(n, count):
    import paxpro_b200 as pxp
    nsteps = 10
    solvers = [_solver(pxp, n, nsteps, 0, 0, seed=i % 3) for i in range(count)]
    batch = pxp.Batch()
    for s in solvers:
        assert batch.admit(s, nsteps)
    batch.round(nsteps)
    assert len(batch.collect()) == count
    for i in range(3):
        with _solver(pxp, n, nsteps, 0, 0, seed=i) as alone:
            alone.step(nsteps)
            assert np.array_equal(alone.get_last_solution(), solvers[i].get_last_solution())
    for s in solvers:
        s.close()
    batch.close()


@pytest.mark.parametrize("n", [500, 4096, 16384])
def test_one_step_between_two_planes(n):
    """A single sampled step whose planes at z and z - dz differ."""
    import paxpro_b200 as pxp
    xmin, xmax, dx, dz, u0, d, b = _problem(n, 2)
    d2, b2 = np.roll(d, 7) * 1.5, np.roll(b, -5) * 0.5
    with _solver(pxp, n, 2, 0, 0) as s:
        s.set_material_planes(np.stack([d2, d]), np.stack([b2, b]), 1, 1)
        s.step(1)
        got = s.get_last_solution()
    rho, r = dz / (wl.K * dx * dx), wl.K * dz
    m, m0 = 0.5 * r * (b2 + 1j * d2), 0.5 * r * (b + 1j * d)
    nb = np.zeros(n, complex)
    nb[1:] += u0[:-1]
    nb[:-1] += u0[1:]
    diag = 1.0 + 0.5j * rho + m
    left = diag * got
    left[1:] -= 0.25j * rho * got[:-1]
    left[:-1] -= 0.25j * rho * got[1:]
    right = (1.0 - 0.5j * rho - m0) * u0 + 0.25j * rho * nb
    # a backward-stable solve leaves a residual of some eps |A| |u|, |A| about 1 + rho
    assert np.linalg.norm(left - right) <= 1e-13 * (1.0 + rho) * np.linalg.norm(u0)
