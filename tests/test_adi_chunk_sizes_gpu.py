"""The general ADI half step at the edges of its launch shapes (rows a thread,
warps a system, systems a CTA), where a system's last chunk is full, one row
long or empty and the last CTA holds fewer systems: every save against the
oracle, a sphere in every plane, Dirichlet and transparent ends."""
import numpy as np
import pytest

from test_parity_adi_gpu import FP32_INT_TOL, FP64_TOL, _int_rel, _rel, _run_both
from paxpro_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,use_tbc,precision", [
    (4, False, 0), (7, True, 0), (192, False, 0), (193, False, 0), (384, True, 0), (385, False, 0),
    (444, False, 0), (445, True, 0), (640, False, 0), (641, False, 0), (832, False, 0),
    (833, False, 0), (1088, False, 0), (1089, False, 0), (1664, False, 0), (1665, False, 0),
    (192, True, 1), (445, False, 1), (640, False, 1), (833, False, 1), (1088, False, 1)])
def test_general_half_step_at_launch_shape_edges(n, use_tbc, precision):
    sph = [(30.0, -20.0, 2375.0, 2020.0, 4.5e-5, 3.6e-6)]  # its rim crosses the first and last planes
    x = -500.0 + wl.step_for_nodes(-500.0, 500.0, n) * np.arange(n)
    g = np.exp(-((x - 40.0) / 400.0) ** 2) * np.exp(1j * 2e-3 * x)
    u0 = np.asfortranarray(g[:, None] * g[None, :])
    steps = 4 if n > 700 else 8
    out, saves, ref_out, ref_saves = _run_both(n, 0.0, steps, 500.0, sph, u0=u0, use_tbc=use_tbc,
                                               precision=precision, L=1000.0)
    assert len(saves) == len(ref_saves) == steps
    for a, b in zip(saves, ref_saves):
        if precision == 0:
            assert _rel(a, b) <= FP64_TOL
        else:
            assert _int_rel(a, b) <= FP32_INT_TOL


@pytest.mark.parametrize("n,precision", [(n, 0) for n in (257, 296, 297, 513, 592, 593, 740, 741, 769,
                                                          888, 889)] +
                         [(n, 1) for n in (5, 64, 100, 256, 296, 513, 741, 888, 1024, 2048)])
def test_vacuum_half_step_at_launch_shape_edges(n, precision):
    """The one-wave vacuum kernel where its systems a CTA change, and on
    complex64 fields (2048 nodes: the kernel above its sizes)."""
    x = -500.0 + wl.step_for_nodes(-500.0, 500.0, n) * np.arange(n)
    g = np.exp(-((x - 40.0) / 300.0) ** 2) * np.exp(1j * 2e-3 * x)
    u0 = np.asfortranarray(g[:, None] * g[None, :])
    out, saves, ref_out, ref_saves = _run_both(n, 0.0, 4, 1000.0, [], u0=u0, precision=precision)
    assert len(saves) == len(ref_saves) == 4
    for a, b in zip(saves, ref_saves):
        if precision == 0:
            assert _rel(a, b) <= FP64_TOL
        else:
            assert _int_rel(a, b) <= FP32_INT_TOL
