"""Batch groups that the batch tests reach no other way, bit for bit against the
solver alone: FFTSolver2D lengths with a prime above 31 (the chirp-z kernel) and
CrankNicholson solvers that no material was set on; and flux sums of sampled
media on clusters against the field's own."""
import math

import numpy as np
import pytest

from paxpro_b200 import workloads as wl
from test_cn_sampled_paths_gpu import _read, _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_chirp_z_groups_equal_alone(precision):
    from paxpro_b200 import serving as sv
    rng = np.random.default_rng(13)
    jobs = []
    for i, n in enumerate([401, 1009, 401, 2 * 1009, 401]):
        j = sv.draw_2d(rng, "fft2d", i)
        j.n, j.nsteps = n, int(rng.integers(20, 60))
        jobs.append(j)
    alone = sv.run_plain(jobs, precision=precision)
    mixed = sv.run_batched(jobs, precision=precision, max_steps=17)
    for i in range(len(jobs)):
        assert np.array_equal(alone.intensities[i], mixed.intensities[i]), jobs[i].n


@pytest.mark.parametrize("n,precision", [(40, 0), (300, 0), (1000, 1), (4096, 0), (8192, 0)])
def test_cn_without_a_material_is_vacuum(n, precision):
    """Alone, in a batch, and with a table of zeros set: the same bits; and a
    material set after steps in vacuum counts from there."""
    import paxpro_b200 as pxp
    dz, steps, dx = 500.0, 20, wl.step_for_nodes(-250.0, 250.0, n)
    x = wl.coords(-250.0, dx, n)
    u0 = np.exp(-((x - 7.0) / 60.0) ** 2) * np.exp(1j * 4e-3 * x)
    d, b = wl.Waveguide(ramp_points=min(25, n // 8)).tables(x)

    def make(zeros):
        s = pxp.Solver(pxp.ProblemSpec(kind=pxp.CRANK_NICHOLSON, x=pxp.Disc(-250.0, 250.0, dx),
                                       z=pxp.Disc(0.0, 2 * steps * dz, dz), wavenumber=wl.K,
                                       precision=precision))
        if zeros:
            s.set_material_table(np.zeros(n), np.zeros(n))
        s.set_initial_conditions(u0)
        return s

    out = []
    for zeros, batched in ((True, False), (False, False), (False, True)):
        with make(zeros) as s:
            if batched:
                batch = pxp.Batch()
                assert batch.admit(s, steps)
                batch.round(steps)
                assert len(batch.collect()) == 1
                batch.close()
            else:
                s.step(steps)
            vacuum = s.get_last_solution()
            s.set_material_table(d, b)
            s.step(steps)
            out.append((vacuum, s.get_last_solution()))
    for o in out[1:]:
        assert np.array_equal(o[0], out[0][0]) and np.array_equal(o[1], out[0][1])
    assert not np.array_equal(out[0][0], out[0][1])
    # vacuum with Dirichlet ends keeps the norm: the step matrix is unitary
    want = np.linalg.norm(u0)
    assert abs(np.linalg.norm(out[0][0]) - want) <= (1e-4 if precision else 1e-11) * want


@pytest.mark.parametrize("n,precision", [(1025, 0), (2048, 0), (2048, 1), (3000, 0), (4096, 0)])
def test_flux_of_sampled_media_on_clusters(n, precision):
    nsteps = 30
    with _solver(n, nsteps, precision) as s:
        s.step(nsteps)
        u, flux = _read(s, nsteps)[0], s.get_flux(1, nsteps)
    w = np.abs(u[n // 5:n - n // 4 + 1]) ** 2
    want = math.fsum(2.0 * w) - w[0] - w[-1]
    # some 30 roundings: 8 terms a thread, two trees, and the squares here
    assert abs(flux[-1] - want) <= 1e-14 * want
