"""CrankNicholson with a medium sampled per step, Dirichlet ends: the path that
factors a block of steps ahead, at its launch shapes' edges and across blocks of
steps, and the short calls that solve step by step, against a Thomas sweep on
the host.  FP64 <= 1e-10 relative L2, FP32 <= 1e-4 of the intensity."""
import numpy as np
import pytest

from paxpro_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _thomas(diag, off, rhs):
    n = len(rhs)
    g, y = [0j] * n, [0j] * n
    prev_g, prev_y = 0j, 0j
    for i in range(n):
        prev_g = 1.0 / (diag[i] - off * off * prev_g)
        prev_y = (rhs[i] - off * prev_y) * prev_g
        g[i], y[i] = prev_g, prev_y
    x = 0j
    for i in range(n - 1, -1, -1):
        x = y[i] - off * g[i] * x
        y[i] = x
    return np.array(y)


@pytest.mark.parametrize("n,calls,precision", [
    (17, [30], 0), (64, [24, 23, 30], 0), (65, [40], 0), (256, [40], 0), (300, [24, 5, 31], 0),
    (512, [30], 0), (1024, [30], 0), (1025, [30], 0), (2048, [26], 0), (2049, [26], 0),
    (3000, [190], 0), (4096, [24], 0), (100, [40], 1), (1501, [30, 3], 1), (3000, [30], 1)])
def test_sampled_planes(n, calls, precision):
    import paxpro_b200 as pxp
    xmin, xmax, dz, nsteps = -250.0, 250.0, 500.0, sum(calls)
    dx = wl.step_for_nodes(xmin, xmax, n)
    x = wl.coords(xmin, dx, n)
    rng = np.random.default_rng(n)
    u = np.exp(-((x - 7.0) / 60.0) ** 2) * np.exp(1j * 4e-3 * x)
    guide = wl.Waveguide(core_half_width=50.0, ramp_points=min(25, n // 8))

    def plane(z):
        return guide.tables(x - z * z / 4e6)

    d, b = np.empty((nsteps, 2, n)), np.empty((nsteps, 2, n))
    for s in range(nsteps):
        for q, z in enumerate(((s + 1) * dz, s * dz)):
            d[s, q], b[s, q] = plane(z)
    d[nsteps // 2, 1] *= 1.0 + 0.1 * rng.random(n)  # planes that do not continue each other
    with pxp.Solver(pxp.ProblemSpec(kind=pxp.CRANK_NICHOLSON, x=pxp.Disc(xmin, xmax, dx),
                                    z=pxp.Disc(0.0, nsteps * dz, dz), wavenumber=wl.K,
                                    precision=precision, save_every=10)) as s:
        s.set_material_planes(d, b, 1, nsteps)
        s.set_initial_conditions(u)
        for c in calls:
            s.step(c)
        got = s.get_last_solution()
        saves = [s.get_saved(i) for i in range(s.num_saved())]
    rho, r = dz / (wl.K * dx * dx), wl.K * dz
    ref = []
    for s in range(nsteps):
        m, m0 = (0.5 * r * (b[s, q] + 1j * d[s, q]) for q in (0, 1))
        nb = np.zeros(n, complex)
        nb[1:] += u[:-1]
        nb[:-1] += u[1:]
        u = _thomas(list(1.0 + 0.5j * rho + m), -0.25j * rho,
                    list((1.0 - 0.5j * rho - m0) * u + 0.25j * rho * nb))
        if (s + 1) % 10 == 0:
            ref.append(u)
    assert len(saves) == len(ref)
    for v, w in list(zip(saves, ref)) + [(got, u)]:
        if precision:
            v, w = np.abs(v) ** 2, np.abs(w) ** 2
            assert np.linalg.norm(v - w) <= 1e-4 * np.linalg.norm(w)
        else:
            assert np.linalg.norm(v - w) <= 1e-10 * np.linalg.norm(w)
