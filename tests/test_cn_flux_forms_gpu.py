"""The flux sums of CrankNicholson's step-invariant path do not depend on how a
launch spreads its problems over the SMs: alone and among many, bit for bit, and
against the field's own sum."""
import math

import numpy as np
import pytest

from test_cn_two_sided_gpu import _solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count,precision", [(4096, 38, 0), (4096, 38, 1), (8192, 38, 0), (16384, 19, 0)])
def test_flux_is_the_same_alone_and_among_many(n, count, precision):
    import paxpro_b200 as pxp
    nsteps, a, e = 12, n // 5, n - n // 4

    def windows(s):
        s.set_flux_windows(2, np.full(nsteps - 1, a), np.full(nsteps - 1, e))

    solvers = [_solver(pxp, n, nsteps, precision, 0, seed=i % 3) for i in range(count)]
    batch = pxp.Batch()
    for s in solvers:
        windows(s)
        assert batch.admit(s, nsteps)
    batch.round(nsteps)
    assert len(batch.collect()) == count
    for i in range(3):
        with _solver(pxp, n, nsteps, precision, 0, seed=i) as alone:
            windows(alone)
            alone.step(nsteps)
            flux, u = alone.get_flux(2, nsteps - 1), alone.get_last_solution()
            for s in solvers[i::3]:
                assert np.array_equal(s.get_flux(2, nsteps - 1), flux)
        w = np.abs(u[a:e + 1]) ** 2
        want = math.fsum(2.0 * w) - w[0] - w[-1]
        # trees of at most 32 x 16 terms over sums of at most 16: some 30 roundings
        assert abs(flux[-1] - want) <= 1e-14 * want
    for s in solvers:
        s.close()
    batch.close()
