"""CrankNicholson's step-invariant path at 4096 rows on one, two and four SMs
(beside a 3-D solver; among problems that need the SMs; alone): field, saves and
flux sums bit for bit."""
import numpy as np
import pytest

from paxpro_b200 import workloads as wl
from test_cn_two_sided_gpu import _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("n", [4096, 2500])
def test_forms_agree(n, precision):
    import paxpro_b200 as pxp
    nsteps = 24

    def result(s):
        s.set_flux_windows(1, np.full(nsteps, n // 5), np.full(nsteps, n - n // 4))
        return s

    def read(s):
        return [s.get_last_solution(), s.get_flux(1, nsteps)] + [s.get_saved(i) for i in range(s.num_saved())]

    with result(_solver(pxp, n, nsteps, precision, 8)) as s:
        s.step(nsteps)
        alone = read(s)
    assert len(alone) == 5 and np.all(np.isfinite(alone[0]))
    x = pxp.Disc(-500.0, 500.0, wl.step_for_nodes(-500.0, 500.0, 16))
    third = pxp.Solver(pxp.ProblemSpec(kind=pxp.ADI, x=x, y=x, z=pxp.Disc(0.0, 1e4, 1000.0), wavenumber=wl.K))
    third.set_initial_conditions(np.ones((16, 16), dtype=np.complex128))  # at work until waited for
    with result(_solver(pxp, n, nsteps, precision, 8)) as s:
        s.step(nsteps)
        beside = read(s)
    third.close()
    batch, many = pxp.Batch(), [result(_solver(pxp, n, nsteps, precision, 8)) for _ in range(40)]
    for s in many:
        assert batch.admit(s, nsteps)
    batch.round(nsteps)
    batch.collect()
    for other in [beside] + [read(s) for s in many]:
        assert len(other) == len(alone)
        for a, b in zip(other, alone):
            assert np.array_equal(a, b)
    for s in many:
        s.close()
    batch.close()
