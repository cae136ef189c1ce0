"""CrankNicholson with a medium sampled per step gives the same bits however its
steps are split into calls, alone and in a batch (jobs of different media,
steps and first steps side by side, rounds of any length), and beside a 3-D
solver; fields, saves and flux sums."""
import numpy as np
import pytest

from paxpro_b200 import workloads as wl

pytestmark = pytest.mark.gpu

DZ = 500.0


def _solver(n, nsteps, precision, seed=0, flux=True, first=1):
    import paxpro_b200 as pxp
    dx = wl.step_for_nodes(-250.0, 250.0, n)
    x = wl.coords(-250.0, dx, n)
    rng = np.random.default_rng(seed)
    guide = wl.Waveguide(core_half_width=rng.uniform(20, 60), ramp_points=min(25, n // 8))
    radius = rng.uniform(1e6, 4e6)
    d, b = np.empty((nsteps, 2, n)), np.empty((nsteps, 2, n))
    for s in range(nsteps):
        for q, z in enumerate(((s + 1) * DZ, s * DZ)):
            d[s, q], b[s, q] = guide.tables(x - z * z / radius)
    s = pxp.Solver(pxp.ProblemSpec(kind=pxp.CRANK_NICHOLSON, x=pxp.Disc(-250.0, 250.0, dx),
                                   z=pxp.Disc(0.0, nsteps * DZ, DZ), wavenumber=wl.K, precision=precision,
                                   save_every=10))
    s.set_material_planes(d, b, 1, nsteps)
    if flux:
        s.set_flux_windows(1, np.full(nsteps, n // 5), np.full(nsteps, n - n // 4))
    s.set_initial_conditions(np.exp(-((x - rng.uniform(-9, 9)) / 60.0) ** 2) * np.exp(1j * 4e-3 * x))
    return s


def _read(s, nsteps, flux=True):
    out = [s.get_last_solution()] + [s.get_saved(i) for i in range(s.num_saved())]
    return out + [s.get_flux(1, nsteps)] if flux else out


def _equal(a, b):
    assert len(a) == len(b)
    for v, w in zip(a, b):
        assert np.all(np.isfinite(v)) and np.array_equal(v, w)


# 200 steps of 4096 rows are more than one window of tables
@pytest.mark.parametrize("n,nsteps,precision", [
    (60, 30, 0), (64, 40, 0), (300, 48, 0), (512, 48, 1), (1000, 30, 0), (1501, 48, 0), (2048, 48, 1),
    (4000, 200, 0), (40, 30, 0), (300, 5, 0)])
def test_splits_and_batches_give_the_same_bits(n, nsteps, precision):
    import paxpro_b200 as pxp
    with _solver(n, nsteps, precision) as s:
        s.step(nsteps)
        whole = _read(s, nsteps)
        # a second pass over the same medium
        s.set_initial_conditions(whole[0])
        s.step(nsteps)
        again = _read(s, nsteps)
    assert not np.array_equal(again[0], whole[0])
    for split in ([1] * nsteps, [nsteps // 3, 1, nsteps - 1 - nsteps // 3]):
        with _solver(n, nsteps, precision) as s:
            for k in split:
                s.step(k)
            _equal(_read(s, nsteps), whole)
            s.step(0)
            s.set_initial_conditions(whole[0])
            for k in split:
                s.step(k)
            _equal(_read(s, nsteps), again)
    # other jobs: media of their own, some of them shorter, one already under way
    jobs = [(_solver(n, nsteps, precision), nsteps)]
    jobs += [(_solver(n, nsteps - 3 * i if nsteps > 20 else nsteps, precision, seed=i), 0) for i in range(1, 4)]
    started = _solver(n, nsteps, precision)
    started.step(2)
    x = pxp.Disc(-500.0, 500.0, wl.step_for_nodes(-500.0, 500.0, 16))
    third = pxp.Solver(pxp.ProblemSpec(kind=pxp.ADI, x=x, y=x, z=pxp.Disc(0.0, 1e4, 1000.0), wavenumber=wl.K))
    third.set_initial_conditions(np.ones((16, 16), dtype=np.complex128))  # at work until waited for
    batch = pxp.Batch()
    for i, (s, _) in enumerate(jobs):
        assert batch.admit(s, nsteps - 3 * i if nsteps > 20 else nsteps)
    assert batch.admit(started, nsteps - 2)
    left = nsteps
    for k in (1, 7, nsteps):
        batch.round(k)
        left -= min(k, left)
    assert len(batch.collect()) == 5
    _equal(_read(jobs[0][0], nsteps), whole)
    _equal(_read(started, nsteps), whole)
    for i in range(1, 4):
        m = nsteps - 3 * i if nsteps > 20 else nsteps
        with _solver(n, m, precision, seed=i) as s:
            s.step(m)
            _equal(_read(jobs[i][0], m), _read(s, m))
    for s in [s for s, _ in jobs] + [started, third]:
        s.close()
    batch.close()


def test_media_of_few_and_many_steps_in_one_batch():
    """Both sampled paths, and the step-invariant one, in the same rounds."""
    import paxpro_b200 as pxp
    n, kinds = 500, [5, 60, 12, 60, 7]
    jobs = [_solver(n, m, 0, seed=i, flux=i % 2 == 0) for i, m in enumerate(kinds)]
    const = _solver(n, 60, 0, seed=9)
    const.set_material_table(np.full(n, 1e-6), np.full(n, 1e-8))
    batch = pxp.Batch()
    for s, m in zip(jobs, kinds):
        assert batch.admit(s, m)
    assert batch.admit(const, 60)
    for _ in range(6):
        batch.round(10)
    assert len(batch.collect()) == 6
    for i, (s, m) in enumerate(zip(jobs, kinds)):
        with _solver(n, m, 0, seed=i, flux=i % 2 == 0) as alone:
            alone.step(m)
            _equal(_read(s, m, i % 2 == 0), _read(alone, m, i % 2 == 0))
        s.close()
    const.close()
    batch.close()


@pytest.mark.parametrize("n,count,precision,tol", [(300, 121, 0, 1e-12), (1501, 73, 0, 1e-12), (4000, 49, 1, 1e-5)])
def test_large_groups_agree_with_alone(n, count, precision, tol):
    """One job more than take the tables: step by step, then the rest with them."""
    import paxpro_b200 as pxp
    jobs = [_solver(n, 30, precision, seed=i % 3) for i in range(count)]
    jobs[0].step(4)
    batch = pxp.Batch()
    for i, s in enumerate(jobs):
        assert batch.admit(s, 26 if i == 0 else 30 if i % 8 else 12)
    for k in (5, 7, 30):
        batch.round(k)
    assert len(batch.collect()) == count
    alone = []
    for i in range(3):
        with _solver(n, 30, precision, seed=i) as s:
            s.step(12)
            alone.append([s.get_last_solution()])
            s.step(18)
            alone[-1].append(s.get_last_solution())
    for i, s in enumerate(jobs):
        want, got = alone[i % 3][1 if i == 0 or i % 8 else 0], s.get_last_solution()
        assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)
        s.close()
    batch.close()
