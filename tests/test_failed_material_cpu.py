"""A material call whose device memory cannot be had leaves no medium behind: the
next step is refused, alone and in a batch, and launches nothing, until the
medium has been set again.  Without a GPU (tests/fake_cuda.py)."""
import pytest

from tests import fake_cuda

SET = {
    "fft2d table": ("FFT_SOLVER_2D", 64, "s.set_material_table(np.zeros(n), np.zeros(n))"),
    "fft2d planes": ("FFT_SOLVER_2D", 63, "s.set_material_planes(np.zeros((30, n)), np.zeros((30, n)), 1, 30)"),
    "cn table": ("CRANK_NICHOLSON", 256, "s.set_material_table(np.zeros(n), np.zeros(n))"),
    "cn planes": ("CRANK_NICHOLSON", 256, "s.set_material_planes(np.zeros((60, n)), np.zeros((60, n)), 1, 30)"),
    "cn short": ("CRANK_NICHOLSON", 20, "s.set_material_planes(np.zeros((6, n)), np.zeros((6, n)), 1, 3)"),
    "adi spheres": ("ADI", 16, "s.set_material_spheres([pxp.Sphere(0, 0, 0, 9, 1e-5, 1e-6)])"),
    "adi planes": ("ADI", 16, "s.set_material_planes(np.zeros((6, n, n)), np.zeros((6, n, n)), 1, 3)"),
    "fft3d table": ("FFT_SOLVER_3D", 15, "s.set_material_table(np.zeros((n, n)), np.zeros((n, n)))"),
}


@pytest.mark.parametrize("failing", [1, 2])
@pytest.mark.parametrize("case", sorted(SET))
def test_no_step_through_a_medium_that_was_not_set(case, failing):
    kind, n, call = SET[case]
    fake_cuda.run(f"""
        n = {n}
        three_d = {kind!r} in ("ADI", "FFT_SOLVER_3D")
        s = pxp.Solver(spec(getattr(pxp, {kind!r}), n))
        s.set_initial_conditions(np.ones((n, n) if three_d else n, dtype=np.complex128))
        fake.fake_fail_allocations({failing})
        try:
            {call}
            failed = False
        except Exception as e:
            assert "out of memory" in str(e), e
            failed = True
        fake.fake_fail_allocations(0)
        assert failed or {failing} == 2
        before = fake.fake_launches()
        if failed:
            assert lib.pxp_step(s._h, 3) == _capi.PXP_ERR_INVALID
            assert "medium" in _capi.last_error(s._h)
            b = pxp.Batch()
            try:
                b.admit(s, 3)
                raise SystemExit("admitted")
            except Exception as e:
                assert "medium" in str(e), e
            assert fake.fake_launches() == before
        {call}
        s.step(3)
        assert fake.fake_launches() > before
    """)


def test_no_batch_round_through_a_medium_that_was_not_set():
    fake_cuda.run("""
        n = 256
        s = pxp.Solver(spec(pxp.CRANK_NICHOLSON, n))
        s.set_initial_conditions(np.ones(n, dtype=np.complex128))
        b = pxp.Batch()
        assert b.admit(s, 9)
        b.round(3)
        fake.fake_fail_allocations(1)
        try:
            s.set_material_table(np.zeros(n), np.zeros(n))
            raise SystemExit("set")
        except Exception as e:
            assert "out of memory" in str(e), e
        fake.fake_fail_allocations(0)
        before = fake.fake_launches()
        try:
            b.round(3)
            raise SystemExit("stepped")
        except Exception as e:
            assert "medium" in str(e), e
        assert fake.fake_launches() == before
        s.set_material_table(np.zeros(n), np.zeros(n))
        b.round(3)
        assert fake.fake_launches() == before + 1
    """)
