"""The host side of CrankNicholson with media sampled per step, without a GPU
(tests/fake_cuda.py; launches are counted: two to factor a window of steps, one
to solve steps in it, one in all step by step): a window is factored once for
the steps in it however they are split, afresh for another pass or another
medium, and its buffer goes when its last step is done; without memory for it
the steps run one by one; captured work leaves the handle's window alone."""
from tests import fake_cuda

HEAD = """
        n = 500

        def planes(steps):
            return np.zeros((2 * steps, n))

        def solver(steps):
            s = pxp.Solver(spec(pxp.CRANK_NICHOLSON, n, nsteps=max(steps, 64)))
            s.set_material_planes(planes(steps), planes(steps), 1, steps)
            s.set_initial_conditions(np.ones(n, dtype=np.complex128))
            return s

        def launches(f, *a):
            before = fake.fake_launches()
            f(*a)
            return fake.fake_launches() - before
"""


def test_windows_of_a_solver():
    fake_cuda.run(HEAD + """
        s = solver(60)
        held = fake.fake_live()
        assert launches(s.step, 60) == 3 and fake.fake_live() == held
        s.set_initial_conditions(np.ones(n, dtype=np.complex128))
        assert [launches(s.step, 1) for _ in range(60)] == [3] + [1] * 59
        assert fake.fake_live() == held
        # another pass, and another medium, while a window is held
        s.set_initial_conditions(np.ones(n, dtype=np.complex128))
        assert launches(s.step, 7) == 3 and fake.fake_live() == held + 1
        s.set_initial_conditions(np.ones(n, dtype=np.complex128))
        assert launches(s.step, 7) == 3 and launches(s.step, 3) == 1
        s.set_material_planes(planes(50), planes(50), 1, 50)
        assert launches(s.step, 1) == 3
        s.close()
        # few steps, and many (a window holds 96 MB / (92 + 48 bytes a row) of them)
        s = solver(23)
        assert launches(s.step, 23) == 1
        s.close()
        per = 64 * (4 * 8 + 14) * 16 + 48 * 512
        most = (96 << 20) // per
        s = solver(2 * most + 30)
        held = fake.fake_live()
        assert launches(s.step, 2 * most + 30) == 9 and fake.fake_live() == held
        s.close()
    """)


def test_no_memory_for_a_window():
    fake_cuda.run(HEAD + """
        s = solver(60)
        held = fake.fake_live()
        fake.fake_fail_allocations(1)
        assert launches(s.step, 20) == 1
        fake.fake_fail_allocations(0)
        assert launches(s.step, 20) == 3 and launches(s.step, 20) == 1
        assert fake.fake_live() == held
        # in a batch: jobs without a window step by step, beside one that has its own
        jobs, b = [solver(40) for _ in range(3)], pxp.Batch()
        for j in jobs:
            assert b.admit(j, 40)
        assert launches(b.round, 1) == 3
        for j in jobs[:2]:
            j.set_material_planes(planes(40), planes(40), 1, 40)
        fake.fake_fail_allocations(1)
        assert launches(b.round, 5) == 1 + 1
        fake.fake_fail_allocations(0)
        assert launches(b.round, 40) == 3
        assert len(b.collect()) == 3
    """)


def test_windows_of_a_batch():
    fake_cuda.run(HEAD + """
        steps = [60, 60, 45, 24, 20]
        jobs, b = [solver(k) for k in steps], pxp.Batch()
        for j, k in zip(jobs, steps):
            assert b.admit(j, k)
        # four jobs in one group with windows, one step by step
        assert launches(b.round, 10) == 3 + 1
        assert launches(b.round, 14) == 1 + 1
        assert launches(b.round, 40) == 1
        assert len(b.collect()) == 5
        for j in jobs:
            j.close()
    """)


def test_captured_steps_bring_their_own_window():
    fake_cuda.run(HEAD + """
        s = solver(60)
        held = fake.fake_live()
        assert launches(s.step, 10) == 3
        fake.fake_capturing(1)
        assert launches(s.step, 5) == 3 and fake.fake_live() == held + 1
        fake.fake_capturing(0)
        assert launches(s.step, 5) == 1
        assert launches(s.step, 40) == 1 and fake.fake_live() == held
    """)


def test_large_batches_go_step_by_step():
    fake_cuda.run("""
        def solver(n, steps):
            s = pxp.Solver(spec(pxp.CRANK_NICHOLSON, n))
            z = np.zeros((2 * steps, n))
            s.set_material_planes(z, z, 1, steps)
            s.set_initial_conditions(np.ones(n, dtype=np.complex128))
            return s

        def launches(f, *a):
            before = fake.fake_launches()
            f(*a)
            return fake.fake_launches() - before

        for n, most in ((250, 148), (500, 120), (1000, 100), (2048, 72), (2049, 48)):
            b = pxp.Batch()
            jobs = [solver(n, 26) for _ in range(most + 1)]
            jobs[0].step(2)
            for i, j in enumerate(jobs):
                assert b.admit(j, 6 if i in (0, most) else 16)
            assert launches(b.round, 5) == 1, n
            assert launches(b.round, 1) == 1 and len(b.collect()) == 2
            assert launches(b.round, 6) == 3, n  # most - 1 of them
            assert b.admit(jobs[0], 4)
            assert launches(b.round, 2) == 1, n  # its window is from its first steps
            for j in jobs:
                j.close()
            b.close()
    """)


def test_a_first_step_without_a_material_can_be_captured():
    """Nothing is allocated or copied by it."""
    fake_cuda.run("""
        for n in (100, 4096):
            s = pxp.Solver(spec(pxp.CRANK_NICHOLSON, n))
            s.set_initial_conditions(np.ones(n, dtype=np.complex128))
            held, copies = fake.fake_live(), fake.fake_copies()
            fake.fake_capturing(1)
            s.step(3)
            fake.fake_capturing(0)
            assert (fake.fake_live(), fake.fake_copies()) == (held, copies)
            s.close()
    """)
