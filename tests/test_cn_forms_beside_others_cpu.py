"""How many SMs a CrankNicholson problem takes beside the other handles of the
device (the CTAs of its launch), without a GPU: several when it has the device
to itself, one beside a 3-D solver at work, whose half steps need an SM a CTA,
and fewer when 2-D handles at work need the SMs; handles that the host has
waited for, or that were given nothing to do, leave it its SMs."""
from tests import fake_cuda


def test_launch_forms():
    fake_cuda.run("""
        def cn(n):
            s = pxp.Solver(spec(pxp.CRANK_NICHOLSON, n))
            s.set_material_table(np.zeros(n), np.zeros(n))
            s.set_initial_conditions(np.ones(n, dtype=np.complex128))
            return s

        def ctas(s):
            s.step(1)
            return fake.fake_last_grid()

        s, big = cn(4096), cn(16384)
        assert (ctas(s), ctas(big)) == (4, 8)
        field = np.ones((16, 16), dtype=np.complex128)
        third = pxp.Solver(spec(pxp.ADI, 16))
        assert (ctas(s), ctas(big)) == (4, 8)  # nothing to do
        third.set_initial_conditions(field)
        assert (ctas(s), ctas(big)) == (1, 4)
        third.step(1)
        assert (ctas(s), ctas(big)) == (1, 4)
        third.synchronize()
        assert (ctas(s), ctas(big)) == (4, 8)
        third.step(1)
        assert (ctas(s), ctas(big)) == (1, 4)
        third.get_last_solution()
        assert (ctas(s), ctas(big)) == (4, 8)
        third.step(1)
        third.close()
        assert (ctas(s), ctas(big)) == (4, 8)

        def fft2d():
            f = pxp.Solver(spec(pxp.FFT_SOLVER_2D, 64))
            f.set_initial_conditions(np.ones(64, dtype=np.complex128))
            return f

        many = [fft2d() for _ in range(143)]
        assert ctas(s) == 4  # 4 SMs and 144 others
        many.append(fft2d())
        assert ctas(s) == 2
        many += [fft2d() for _ in range(2)]
        assert ctas(s) == 1
        for m in many[:2]:
            m.synchronize()
        assert ctas(s) == 2
        for m in many:
            m.close()
        b = pxp.Batch()
        jobs = [cn(4096) for _ in range(36)]
        for j in jobs[:35]:
            assert b.admit(j, 1)
        b.round(1)  # 35 problems of 4 SMs and 3 other handles
        assert fake.fake_last_grid() == 140
        b.collect()
        for j in jobs:
            assert b.admit(j, 1)
        b.round(1)  # 36 and 2: 146 SMs
        assert fake.fake_last_grid() == 144
        b.collect()
        jobs.append(cn(4096))
        for j in jobs:
            assert b.admit(j, 1)
        b.round(1)
        assert fake.fake_last_grid() == 74
        b.collect()
        jobs += [cn(4096) for _ in range(37)]
        for j in jobs:
            assert b.admit(j, 1)
        b.round(1)  # 74 of 2 SMs and 2 others
        assert fake.fake_last_grid() == 74
        b.collect()
        assert ctas(s) == 4  # the collected jobs are done
    """)


def test_pinned_forms():
    fake_cuda.run("""
        import os
        n = 4096
        s = pxp.Solver(spec(pxp.CRANK_NICHOLSON, n))
        s.set_initial_conditions(np.ones(n, dtype=np.complex128))
        for pin, want in (("0", 1), ("1", 4), ("x", 4)):
            os.environ["PXP_CN_CLUSTER"] = pin
            s.step(1)
            assert fake.fake_last_grid() == want, pin
    """)
