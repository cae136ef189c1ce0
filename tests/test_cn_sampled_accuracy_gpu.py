"""CrankNicholson with a medium sampled per step, against a Thomas sweep in
extended precision on the same matrix entries: the rounding of a table entry that
is the same at every row of a uniform stretch and at every step would add up."""
import numpy as np
import pytest

from paxpro_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 128])
@pytest.mark.parametrize("seed", [1, 2, 3])
def test_error_of_a_long_pass(n, seed):
    import paxpro_b200 as pxp
    dz, steps, dx = 500.0, 300, wl.step_for_nodes(-250.0, 250.0, n)
    x = wl.coords(-250.0, dx, n)
    rng = np.random.default_rng(seed)
    guide = wl.Waveguide(core_half_width=rng.uniform(20, 60), ramp_points=n // 8)
    radius = rng.uniform(1e8, 1e9)
    u0 = np.exp(-((x - rng.uniform(-5, 5)) / 25.0) ** 2) * np.exp(1j * 1e-3 * x)
    d, b = np.empty((steps, 2, n)), np.empty((steps, 2, n))
    for s in range(steps):
        for q, z in enumerate(((s + 1) * dz, s * dz)):
            d[s, q], b[s, q] = guide.tables(x - z * z / radius)
    with pxp.Solver(pxp.ProblemSpec(kind=pxp.CRANK_NICHOLSON, x=pxp.Disc(-250.0, 250.0, dx),
                                    z=pxp.Disc(0.0, steps * dz, dz), wavenumber=wl.K)) as s:
        s.set_material_planes(d, b, 1, steps)
        s.set_initial_conditions(u0)
        s.step(steps)
        got = s.get_last_solution()
    L, C = np.longdouble, np.clongdouble
    rho, r = dz / (wl.K * dx * dx), wl.K * dz
    iq, u = C(1j) * (L(0.25) * L(rho)), u0.astype(C)
    for s in range(steps):
        # the entries as they are rounded in double
        diag = ((1.0 + 0.5 * (b[s, 0] * r)).astype(L) + 1j * (0.5 * rho + 0.5 * (d[s, 0] * r)).astype(L)).astype(C)
        old = (0.5 * (b[s, 1] * r)).astype(L) + 1j * (0.5 * (d[s, 1] * r)).astype(L)
        nb = np.zeros(n, C)
        nb[1:] += u[:-1]
        nb[:-1] += u[1:]
        rhs = iq * nb + (C(1) - 2 * iq - old) * u
        g, y, pg, py = [None] * n, [None] * n, C(0), C(0)
        for i in range(n):
            pg = C(1) / (diag[i] - iq * iq * pg)
            py = (rhs[i] + iq * py) * pg
            g[i], y[i] = pg, py
        v = C(0)
        for i in range(n - 1, -1, -1):
            v = y[i] + iq * g[i] * v
            u[i] = v
    err = float(np.linalg.norm(got.astype(C) - u) / np.linalg.norm(u))
    # a step: one rounding of w, the same at every step, on x of up to 2 |u| (2^-53 a
    # component of w) adds up over the steps in the worst case to 300 * 2^-52 =
    # 6.7e-14; its phase turns with the field, and a quarter of that is allowed
    assert err <= 1.67e-14, err
