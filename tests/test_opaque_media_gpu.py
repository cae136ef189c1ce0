"""Media so opaque that the square of a matrix entry would overflow: the field is
finite, zero in them, and the same however opaque they are (ADI from every kind
of material; CrankNicholson in the step that enters such a medium)."""
import numpy as np
import pytest

from paxpro_b200 import csg
from paxpro_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,medium", [(40, "sphere"), (200, "sphere"), (513, "sphere"), (100, "spheres"),
                                      (100, "planes"), (100, "csg")])
def test_adi_through_an_opaque_sphere(n, medium):
    import paxpro_b200 as pxp
    dx = wl.step_for_nodes(-500.0, 500.0, n)
    x = pxp.Disc(-500.0, 500.0, dx)
    out = []
    for beta in (1e140, 1e160, 1e300):
        with pxp.Solver(pxp.ProblemSpec(kind=pxp.ADI, x=x, y=x, z=pxp.Disc(0.0, 8e3, 1000.0),
                                        wavenumber=wl.K)) as s:
            if medium == "planes":
                c = wl.coords(-500.0, dx, n)
                inside = ((c - 40.0)[:, None] ** 2 + (c + 10.0)[None, :] ** 2) < 200.0 ** 2
                b = np.zeros((16, n, n))
                b[4:6] = np.where(inside, beta, 0.0)
                s.set_material_planes(np.zeros((16, n, n)), b, 1, 8)
            elif medium == "csg":
                m = csg.Module()
                m.add(csg.Part(beta=beta).add(csg.Sphere(200.0).translate(40.0, -10.0, 3000.0)))
                s.set_material_csg([m])
            else:  # one, or more than travel in a launch's parameters
                s.set_material_spheres([pxp.Sphere(40.0 + i, -10.0, 3000.0, 200.0, 0.0, beta)
                                        for i in range(1 if medium == "sphere" else 40)])
            s.set_initial_conditions(np.ones((n, n), dtype=np.complex128, order="F"))
            s.step(6)
            out.append(s.get_last_solution())
    assert np.all(np.isfinite(out[1])) and np.linalg.norm(out[0]) > 0.1 * n
    # nothing passes through such a point: one more or less opaque makes no difference
    for u in out[1:]:
        assert np.linalg.norm(u - out[0]) <= 1e-12 * np.linalg.norm(out[0])


@pytest.mark.parametrize("n", [50, 300, 1501])
def test_cn_into_an_opaque_plane(n):
    import paxpro_b200 as pxp
    steps, dz, dx = 40, 500.0, wl.step_for_nodes(-250.0, 250.0, n)
    x = wl.coords(-250.0, dx, n)
    out = []
    for beta in (1e140, 1e160, 1e300):
        d, b = np.zeros((steps, 2, n)), np.zeros((steps, 2, n))
        b[20:, 0, n // 2:] = beta  # from the 21st step's new plane on
        b[21:, 1, n // 2:] = beta
        with pxp.Solver(pxp.ProblemSpec(kind=pxp.CRANK_NICHOLSON, x=pxp.Disc(-250.0, 250.0, dx),
                                        z=pxp.Disc(0.0, steps * dz, dz), wavenumber=wl.K)) as s:
            s.set_material_planes(d, b, 1, steps)
            s.set_initial_conditions(np.exp(-(x / 60.0) ** 2).astype(np.complex128))
            s.step(21)
            out.append(s.get_last_solution())
    for u in out:
        assert np.all(np.isfinite(u))
        # the step into the medium leaves rounding errors of the field there
        assert np.max(np.abs(u[n // 2 + 1:])) <= 1e-14
    for u in out[1:]:
        assert np.linalg.norm(u - out[0]) <= 1e-12 * np.linalg.norm(out[0])
