"""Timed cases: the calls a user's program makes, over the sizes it makes them at.

Every pass starts from the initial field, steps, and returns whole fields (and
saved slots, flux sums or the far field where the program asks for them).  The
2-D solvers' fields are small and go through host arrays (numpy in, numpy
out), as the scripts that use them do; the 3-D fields and the served jobs stay
on the device and come back as views of the resident field.

    kind      entry points
    fft2d/cn  Solver.set_initial_conditions, step, get_last_solution, get_saved, get_flux
    adi/fft3d Solver.set_initial_conditions_device, step, synchronize, field_device_ptr
    farfield  Solver.farfield with a subtracted reference, as GenericScattering calls it
    batch     Batch.admit, round, collect: one round of the serving loop

All lengths are in nm.  `exact` restates the schemes in plain torch, complex128.
"""
import math

import numpy as np
import torch

import paxpro_b200 as pxp
from paxpro_b200 import serving

LAMBDA = 0.1


def listed():
    return [
        # a short look at a small guide: launch latency and the host round trip count
        {"name": "fft2d_256", "kind": "fft2d", "n": 256, "steps": 200, "fp32": False, "medium": "guide", "save_every": 0},
        # the planar waveguide problem, 4 mm in 1 um steps, a save every 100
        {"name": "fft2d_2048", "kind": "fft2d", "n": 2048, "steps": 4000, "fp32": False, "medium": "guide", "save_every": 100},
        # the grid that a domain of 1000 steps gives: a length that is no power of two
        {"name": "fft2d_1001", "kind": "fft2d", "n": 1001, "steps": 1000, "fp32": False, "medium": "guide", "save_every": 0},
        # the same guide by finite differences, 4 mm in half-micron steps
        {"name": "cn_4096", "kind": "cn", "n": 4096, "steps": 8000, "fp32": False, "medium": "guide", "save_every": 100},
        # a curved guide: the medium changes every step, the transmitted flux is read for every step
        {"name": "cn_curved_1501", "kind": "cn", "n": 1501, "steps": 400, "fp32": False, "medium": "curved", "save_every": 0},
        # plane-wave-like beam past one small sphere: nearly every plane is vacuum
        {"name": "adi_1024", "kind": "adi", "n": 1024, "steps": 200, "fp32": False, "medium": "far", "absorber": False},
        # the scattering example's grid: the sphere fills the domain, every plane meets it
        {"name": "adi_513", "kind": "adi", "n": 513, "steps": 64, "fp32": False, "medium": "filled", "absorber": False},
        # the large field: 268 MB, few spheres a step
        {"name": "fft3d_4096", "kind": "fft3d", "n": 4096, "steps": 20, "fp32": False, "medium": "far", "absorber": False},
        # a served 3-D job in complex64
        {"name": "fft3d_1024_fp32", "kind": "fft3d", "n": 1024, "steps": 200, "fp32": True, "medium": "far", "absorber": False},
        # the scattering example with its default propagator: 513 nodes, material in every step
        {"name": "fft3d_513", "kind": "fft3d", "n": 513, "steps": 64, "fp32": False, "medium": "filled", "absorber": False},
        # the far field of that example: 512 nodes padded to 32768, a few hundredths of a degree
        {"name": "farfield_512", "kind": "farfield", "n": 512, "pad": 32768, "phi": 0.05, "fp32": False},
        # one round of the serving loop over a mixed set of jobs
        {"name": "batch_60", "kind": "batch", "n2d": 56, "n3d": 4, "nmax": 14, "steps": 200},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fft2d", "fft2d", "cn", "cn", "adi", "adi", "fft3d", "fft3d", "fft3d", "farfield", "batch"])
    fp32 = rng.random() < 0.4
    if kind == "fft2d":
        n = 2 ** rng.randint(8, 13) if rng.random() < 0.6 else _log_int(rng, 100, 3000)
        steps = _log_int(rng, 100, 1500)
        return {"kind": kind, "n": n, "steps": steps, "fp32": fp32, "medium": "guide", "save_every": rng.choice([0, 100])}
    if kind == "cn":
        if rng.random() < 0.3:
            return {"kind": kind, "n": _log_int(rng, 200, 3000), "steps": _log_int(rng, 100, 400), "fp32": fp32, "medium": "curved", "save_every": 0}
        n = 2 ** rng.randint(8, 14) if rng.random() < 0.5 else _log_int(rng, 100, 4000)
        return {"kind": kind, "n": n, "steps": _log_int(rng, 200, 3000), "fp32": fp32, "medium": "guide", "save_every": rng.choice([0, 100])}
    if kind == "adi":
        n = 2 ** rng.randint(7, 10) if rng.random() < 0.4 else _log_int(rng, 100, 1024)
        return {"kind": kind, "n": n, "steps": _log_int(rng, 20, 120), "fp32": fp32, "medium": rng.choice(["far", "filled"]), "absorber": False}
    if kind == "fft3d":
        n = 2 ** rng.randint(7, 11) if rng.random() < 0.6 else _log_int(rng, 100, 1100)
        top = 100 if n <= 600 else 20
        return {"kind": kind, "n": n, "steps": _log_int(rng, 10, top), "fp32": fp32, "medium": rng.choice(["far", "filled"]), "absorber": rng.random() < 0.3}
    if kind == "farfield":
        return {"kind": kind, "n": _log_int(rng, 128, 700), "pad": 2 ** rng.randint(11, 15), "phi": rng.uniform(0.01, 0.05), "fp32": fp32}
    return {"kind": kind, "n2d": rng.randint(4, 56), "n3d": rng.randint(0, 3), "nmax": rng.randint(10, 14), "steps": rng.choice([50, 100, 200])}


# ---- problems ---------------------------------------------------------------


def _step_for(lo, hi, n):
    """A grid step for which the truncating node count int((hi - lo) / step + 1) is n."""
    step = (hi - lo) / (n - 1)
    while int((hi - lo) / step + 1.0) != n:
        step = float(np.nextafter(step, 0.0 if int((hi - lo) / step + 1.0) < n else np.inf))
    return step


def _grid(case):
    """(xmin, xmax, dx, zmin, dz, k) of a single-solver case."""
    kind, n = case["kind"], case["n"]
    k = 2.0 * math.pi / LAMBDA
    if kind in ("fft2d", "cn"):
        return -250.0, 250.0, _step_for(-250.0, 250.0, n), 0.0, 1000.0 if kind == "fft2d" else 500.0, k
    if kind == "farfield" or case["medium"] == "filled":  # the scattering example's domain
        return -750.0, 750.0, _step_for(-750.0, 750.0, n), -525.0, 1050.0 / 256, 2.0 * math.pi / 0.1569
    half = 500.0 if kind == "adi" else 1000.0
    return -half, half, _step_for(-half, half, n), 0.0, 1000.0 if kind == "adi" else 2000.0, k


def _guide(x, core, delta_clad, centre=0.0):
    """delta, beta of a slab guide with an absorbing ramp over 25 points at each end."""
    n = len(x)
    d = np.minimum(np.arange(n), n - 1 - np.arange(n))
    beta_clad = delta_clad / 80.0
    inside = np.abs(x - centre) <= core
    delta = np.where(inside, 0.0, delta_clad)
    beta = np.where(inside, 0.0, beta_clad)
    ramp = d < 25
    beta = np.where(ramp, beta_clad + (1.0e-4 - beta_clad) * (25 - d) / 25.0, beta)
    return np.where(ramp, delta_clad, delta), beta


def _inputs_2d(case, seed):
    """Initial field and medium of a 2-D case: [1 or steps][planes a step][n] delta and beta."""
    rng = np.random.default_rng(seed)
    xmin, _, dx, zmin, dz, _ = _grid(case)
    n, steps = case["n"], case["steps"]
    x = xmin + np.arange(n) * dx
    core, dclad, waist = rng.uniform(10.0, 60.0), rng.uniform(2e-6, 3e-5), rng.uniform(5.0, 30.0)
    u0 = np.exp(-((x - rng.uniform(-5.0, 5.0)) / waist) ** 2) * np.exp(1j * rng.uniform(-2e-3, 2e-3) * x)
    if case["medium"] == "guide":
        d, b = _guide(x, core, dclad)
        return u0, d[None, None], b[None, None]
    radius = rng.uniform(2e8, 1e9)  # the guide's centre moves as z^2 / 2R
    z = zmin + np.arange(1, steps + 1) * dz
    planes = np.stack([np.stack([np.stack(_guide(x, core, dclad, zz * zz / (2.0 * radius))) for zz in (zs, zs - dz)]) for zs in z])
    return u0, planes[:, :, 0], planes[:, :, 1]


def _windows(case):
    """The flux windows of a curved guide's steps: the middle three fifths of the line."""
    n = case["n"]
    return np.full(case["steps"], n // 5), np.full(case["steps"], n - 1 - n // 5)


def _spheres(case, rng):
    """(cx, cy, cz, radius, delta, beta): one that fills the domain, or few small ones."""
    xmin, xmax, _, zmin, dz, _ = _grid(case)
    if case["kind"] == "farfield" or case["medium"] == "filled":
        return [(rng.uniform(-30, 30), rng.uniform(-30, 30), rng.uniform(-30, 30), rng.uniform(420.0, 500.0), 8.9e-6, 7e-7)]
    zmax = zmin + case["steps"] * dz
    if case["kind"] == "adi":
        # its x half step's plane at the middle step cuts the sphere
        cz = zmin + (case["steps"] // 2) * dz + rng.uniform(-100.0, 100.0)
        return [(rng.uniform(-50, 50), rng.uniform(-50, 50), cz, rng.uniform(150.0, 200.0), 4.5e-5, 3.6e-6)]
    out = []
    for _ in range(max(2, case["steps"] * 64 // 1000)):
        delta = rng.uniform(1e-6, 5e-5)
        out.append((rng.uniform(xmin, xmax), rng.uniform(xmin, xmax), rng.uniform(zmin, zmax), rng.uniform(20.0, 150.0), delta, delta / 50.0))
    return out


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _axis(case, dev):
    xmin, _, dx = _grid(case)[:3]
    return xmin + torch.arange(case["n"], dtype=torch.float64, device=dev) * dx


def _beam(case, rng, dev):
    """A wide Gaussian beam with a slight tilt, [x][y] (the layout of the resident field)."""
    x = _axis(case, dev)
    xmin, xmax = _grid(case)[:2]
    w = rng.uniform(0.4, 0.8) * (xmax - xmin)
    gx = torch.exp(-((x - rng.uniform(-20.0, 20.0)) / w) ** 2) * torch.exp(1j * rng.uniform(-1e-3, 1e-3) * x)
    gy = torch.exp(-((x - rng.uniform(-20.0, 20.0)) / w) ** 2) * torch.exp(1j * rng.uniform(-1e-3, 1e-3) * x)
    return (gx[:, None] * gy[None, :]).contiguous()


def _inputs_3d(case, seed, dev):
    rng = np.random.default_rng(seed)
    u0 = _beam(case, rng, dev)
    return u0.to(torch.complex64) if case["fp32"] else u0, _spheres(case, rng)


def _scattered(case, seed, dev):
    """An exit field with a sphere's shadow on it, and the same beam without."""
    rng = np.random.default_rng(seed)
    beam = _beam(case, rng, dev)
    cx, cy, _, r, delta, beta = _spheres(case, rng)[0]
    x, k = _axis(case, dev), _grid(case)[5]
    path = 2.0 * torch.sqrt(torch.clamp(r * r - ((x - cx) ** 2)[:, None] - ((x - cy) ** 2)[None, :], min=0.0))
    u = (beam * torch.exp(-k * complex(beta, delta) * path)).contiguous()
    return u.to(torch.complex64) if case["fp32"] else u, beam


def _jobs(case, seed):
    """The job set of a batch: kinds and sizes from the case, parameters from the seed."""
    rng = np.random.default_rng(seed)
    jobs = []
    for i in range(case["n2d"]):
        n = 2 ** (8 + i % (case["nmax"] - 7))
        jobs.append(serving.Job("cn" if i % 5 == 4 else "fft2d", n, case["steps"], i, float(rng.uniform(10.0, 60.0)),
                                float(rng.uniform(2e-6, 3e-5)), float(rng.uniform(5.0, 30.0))))
    for i in range(case["n3d"]):
        zmax = case["steps"] * 2000.0
        spheres = [(rng.uniform(-1000, 1000), rng.uniform(-1000, 1000), rng.uniform(0.0, zmax), rng.uniform(20.0, 150.0), d, d / 50.0)
                   for d in rng.uniform(1e-6, 5e-5, 8)]
        jobs.append(serving.Job("fft3d", 256 * 2 ** (i % 4), case["steps"], case["n2d"] + i, spheres=spheres))
    return jobs


# ---- what a program keeps, and one pass ---------------------------------------


class _View:
    """The resident field as an array that torch can read in place; it keeps its solver."""

    def __init__(self, solver, shape, fp32):
        self.solver = solver
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<c8" if fp32 else "<c16", "data": (solver.field_device_ptr(), False), "version": 3}


def _field(solver):
    shape = (solver.nx, solver.ny) if solver.three_d else (solver.nx,)
    return torch.as_tensor(_View(solver, shape, solver.spec.precision == pxp.FP32), device="cuda")


KINDS = {"fft2d": pxp.FFT_SOLVER_2D, "cn": pxp.CRANK_NICHOLSON, "adi": pxp.ADI, "fft3d": pxp.FFT_SOLVER_3D, "farfield": pxp.FFT_SOLVER_3D}


def _solver(case):
    xmin, xmax, dx, zmin, dz, k = _grid(case)
    x = pxp.Disc(xmin, xmax, dx)
    absorber = (0.1 * (xmax - xmin), 0.05 * (xmax - xmin)) if case.get("absorber") else (0.0, 0.0)
    s = pxp.Solver(pxp.ProblemSpec(kind=KINDS[case["kind"]], x=x, y=x, z=pxp.Disc(zmin, zmin + case.get("steps", 1) * dz, dz), wavenumber=k,
                                   precision=pxp.FP32 if case["fp32"] else pxp.FP64, save_every=case.get("save_every", 0),
                                   absorber_width=absorber[0], absorber_damping=absorber[1]))
    if (s.nx, s.ny) not in ((case["n"], 1), (case["n"], case["n"])):
        raise ValueError("the grid has %d x %d nodes" % (s.nx, s.ny))
    return s


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("fft2d", "cn"):
        u0, delta, beta = _inputs_2d(case, seed)
        s = _solver(case)
        if case["medium"] == "guide":
            s.set_material_table(delta[0, 0], beta[0, 0])
        else:
            s.set_material_planes(delta, beta, 1, case["steps"])
            s.set_flux_windows(1, *_windows(case))
        return {"case": case, "s": s, "u0": u0}
    if kind == "farfield":
        u0, ref = _scattered(case, seed, "cuda")
        s = _solver(case)
        s.set_reference(ref.t().cpu().numpy())
        torch.cuda.synchronize()
        s.set_initial_conditions_device(u0.data_ptr())
        s.synchronize()
        return {"case": case, "s": s}
    if kind == "batch":
        solvers = [serving.make_solver(j, pxp.FP32) for j in _jobs(case, seed)]
        for s in solvers:
            s.synchronize()
        u0 = [_field(s).clone() for s in solvers]
        torch.cuda.synchronize()
        return {"case": case, "s": solvers, "u0": u0, "batch": pxp.Batch()}
    u0, spheres = _inputs_3d(case, seed, "cuda")
    s = _solver(case)
    s.set_material_spheres([pxp.Sphere(*sp) for sp in spheres])
    torch.cuda.synchronize()
    return {"case": case, "s": s, "u0": u0}


def run(state):
    case, s = state["case"], state["s"]
    kind = case["kind"]
    if kind == "farfield":
        return s.farfield(pad_length=case["pad"], phi_min=-case["phi"], phi_max=case["phi"], subtract_reference=True)
    if kind == "batch":
        batch = state["batch"]
        for solver, u0 in zip(s, state["u0"]):
            solver.set_initial_conditions_device(u0.data_ptr())
            batch.admit(solver, case["steps"])
        batch.round(case["steps"])
        batch.collect()
        return [_field(solver) for solver in s]
    if kind in ("adi", "fft3d"):
        s.set_initial_conditions_device(state["u0"].data_ptr())
        s.step(case["steps"])
        s.synchronize()
        return _field(s)
    s.set_initial_conditions(state["u0"])
    s.step(case["steps"])
    u = s.get_last_solution()
    if case["fp32"]:
        u = u.astype(np.complex64)  # the served precision
    if case["medium"] == "curved":
        return {"u": u, "flux": s.get_flux(1, case["steps"]).astype(u.real.dtype)}
    if case["save_every"]:
        saved = [s.get_saved(i) for i in range(s.num_saved())]
        saved = np.stack(saved) if saved else np.empty((0, case["n"]), np.complex128)
        return {"u": u, "saved": saved.astype(u.dtype)}
    return u


# ---- work -------------------------------------------------------------------


def _work_one(kind, n, steps, fp32):
    pts = n if kind in ("fft2d", "cn") else n * n
    c = 8 if fp32 else 16
    per = {"fft2d": 2 * 5 * math.log2(n) + 14, "cn": 36, "adi": 2 * 40, "fft3d": 4 * 5 * math.log2(n) + 20}[kind]
    return 2.0 * c * pts, per * pts * steps


def work(case):
    """Fields and media in, fields out, each once; the transforms at 5 n log2 n, the tridiagonal solves as one sweep each way."""
    kind = case["kind"]
    if kind == "batch":
        total = [0.0, 0.0]
        for j in _jobs(case, 0):
            b, f = _work_one(j.kind, j.n, j.nsteps, True)
            total = [total[0] + b, total[1] + f]
        return {"bytes": total[0], "flops": total[1]}
    n = case["n"]
    if kind == "farfield":
        xmin, _, dx, _, _, k = _grid(case)
        w = min(case["pad"], 2.0 * case["pad"] * k * dx * math.sin(math.radians(case["phi"])) / (2.0 * math.pi) + 1)
        q = 2 ** math.ceil(math.log2(n))
        # n lines, then w lines, each of pad / q transforms of length q
        return {"bytes": (8 if case["fp32"] else 16) * n * n + 16 * n * n + 8 * w * w, "flops": (n + w) * 5 * case["pad"] * math.log2(q)}
    b, f = _work_one(kind, n, case["steps"], case["fp32"])
    if kind in ("fft2d", "cn"):
        planes = 2 * case["steps"] if case["medium"] == "curved" else 1
        b += 16.0 * n * planes + (8 if case["fp32"] else 16) * n * (case["steps"] // case["save_every"] if case["save_every"] else 0)
    return {"bytes": b, "flops": f}


# ---- the schemes in plain 64-bit torch ------------------------------------------


def _freq2(n, dx, dev):
    i = torch.arange(n, dtype=torch.float64, device=dev)
    i = torch.where(i > n // 2, n - i, i)
    return (2.0 * math.pi * i / (dx * n)) ** 2


def _shift(v, s, fill):
    """v moved by s places along its last axis, `fill` where nothing comes in."""
    pad = torch.full(v.shape[:-1] + (abs(s),), fill, dtype=v.dtype, device=v.device)
    return torch.cat([pad, v[..., :-s]], -1) if s > 0 else torch.cat([v[..., -s:], pad], -1)


def _tridiagonal(diag, off, rhs):
    """Systems along the last axis, constant `off` beside the diagonal: parallel cyclic reduction."""
    n = rhs.shape[-1]
    a = torch.full_like(diag, off)
    c = a.clone()
    a[..., 0] = 0
    c[..., -1] = 0
    b, d, s = diag, rhs, 1
    while s < n:
        lo, hi = -a / _shift(b, s, 1.0), -c / _shift(b, -s, 1.0)
        d = d + lo * _shift(d, s, 0.0) + hi * _shift(d, -s, 0.0)
        b = b + lo * _shift(c, s, 0.0) + hi * _shift(a, -s, 0.0)
        a, c, s = lo * _shift(a, s, 0.0), hi * _shift(c, -s, 0.0), 2 * s
    return d / b


def _fft2d_exact(u, delta, beta, dx, dz, k, steps, every):
    n = u.shape[0]
    prop = torch.exp(-0.5j * dz / k * _freq2(n, dx, u.device))
    saved = []
    for s in range(steps):
        p = s if len(delta) > 1 else 0
        u = torch.fft.ifft(torch.fft.fft(u) * prop) * torch.exp(-k * torch.complex(beta[p, 0], delta[p, 0]) * dz)
        if every and (s + 1) % every == 0:
            saved.append(u)
    return u, saved


def _cn_exact(u, delta, beta, dx, dz, k, steps, every, window=None):
    n = u.shape[0]
    rho, r = dz / (k * dx * dx), k * dz
    saved, flux = [], []
    op = None
    if len(delta) == 1 and n <= 4096:
        # one matrix for every step: its inverse times the right-hand side's matrix, once
        m = 0.5 * r * torch.complex(beta[0, 0], delta[0, 0])
        off = torch.diag(torch.full((n - 1,), 0.25j * rho, dtype=u.dtype, device=u.device), 1)
        off = off + off.t()
        op = torch.linalg.solve(torch.diag(1.0 + 0.5j * rho + m) - off, torch.diag(1.0 - 0.5j * rho - m) + off)
    for s in range(steps):
        if op is not None:
            u = op @ u
        else:
            p = s if len(delta) > 1 else 0
            m, m0 = (0.5 * r * torch.complex(beta[p, q], delta[p, q]) for q in (0, -1))
            rhs = 0.25j * rho * (_shift(u, 1, 0.0) + _shift(u, -1, 0.0)) + (1.0 - 0.5j * rho - m0) * u
            u = _tridiagonal(1.0 + 0.5j * rho + m, -0.25j * rho, rhs)
        if every and (s + 1) % every == 0:
            saved.append(u)
        if window is not None:
            w = u[window[0]:window[1] + 1].abs() ** 2
            flux.append(2.0 * w.sum() - w[0] - w[-1])
    return u, saved, flux


def _material(spheres, x, z):
    """delta, beta at [x][y] on the plane z: the first sphere that holds the point."""
    d = torch.zeros(len(x), len(x), dtype=torch.float64, device=x.device)
    b = torch.zeros_like(d)
    free = None
    for cx, cy, cz, r, delta, beta in spheres:
        dz2 = (z - cz) * (z - cz)
        if dz2 >= r * r:
            continue
        dx, dy = x - cx, x - cy
        inside = ((dx * dx)[:, None] + (dy * dy)[None, :]) + dz2 < r * r
        inside = inside if free is None else inside & free
        d[inside], b[inside] = delta, beta
        free = ~inside if free is None else free & ~inside
    return d, b, free is not None


def _step_material(spheres, x, z0, z1):
    """The medium of an FFTSolver3D step: at z1, or the sampled mean over the step where it changes."""
    if not any(cz - r <= max(z0, z1) and cz + r >= min(z0, z1) for _, _, cz, r, _, _ in spheres):
        return None
    d1, b1, _ = _material(spheres, x, z1)
    d0, b0, _ = _material(spheres, x, z0)
    changes = ((d1 - d0).abs() > 1e-10) | ((b1 - b0).abs() > 1e-10)
    if not bool(changes.any()):
        return d1, b1
    ds, bs = d0 + d1, b0 + b1
    for i in range(1, 9):
        d, b, _ = _material(spheres, x, z0 + i * ((z1 - z0) / 10))
        ds, bs = ds + 2.0 * d, bs + 2.0 * b
    return torch.where(changes, ds / 20.0, d1), torch.where(changes, bs / 20.0, b1)


def _fft3d_exact(u, spheres, x, dx, zmin, dz, k, steps, absorber=None):
    n = u.shape[0]
    f2 = _freq2(n, dx, u.device)
    prop = torch.exp(-0.5j * dz / k * (f2[:, None] + f2[None, :]))
    damp = None
    if absorber is not None:
        t = int(absorber[0] / dx + 1)
        i = torch.arange(n, dtype=torch.float64, device=u.device)
        edge = torch.minimum(i, n - 1 - i)
        damp = torch.where(edge < t, torch.exp(-(t - edge - 1) * dx / absorber[1]), torch.ones_like(edge))
    for s in range(1, steps + 1):
        u = torch.fft.ifft2(torch.fft.fft2(u) * prop)
        m = _step_material(spheres, x, zmin + (s - 1) * dz, zmin + s * dz)
        if m is not None:
            u = u * torch.exp(-k * dz * torch.complex(m[1], m[0]))
        if damp is not None:
            u = u * damp[:, None] * damp[None, :]
    return u


def _adi_half(u, diag, off, h):
    """Implicit along the last axis, explicit along the first."""
    up = torch.zeros_like(u)
    up[1:] += u[:-1]
    up[:-1] += u[1:]
    return _tridiagonal(diag.expand(u.shape), off, (1.0 / h + 2.0 * off) * u - off * up)


def _adi_exact(u, spheres, x, dx, zmin, dz, k, steps):
    h, kd = dz / 2.0, k * dx * dx
    off = -0.5j / kd
    u = u.t().contiguous()  # [y][x]
    for s in range(1, steps + 1):
        z = zmin + s * dz
        d, b, _ = _material(spheres, x, z)
        u = _adi_half(u, 1.0 / h + 1j / kd + k * torch.complex(b, d).t(), off, h)
        d, b, _ = _material(spheres, x, z + h)
        u = _adi_half(u.t().contiguous(), 1.0 / h + 1j / (kd + k * torch.complex(b, d)), off, h).t().contiguous()
    return u.t().contiguous()


def _angle_index(angle, size, k, step):
    n = int(size * k * step * math.sin(angle * math.pi / 180.0) / (2.0 * math.pi))
    if abs(n) >= size // 2:
        return size - 1 if angle > 0.0 else 0
    return n + size // 2


def _farfield_exact(u, ref, L, phi, k, dx):
    lo, hi = _angle_index(-phi, L, k, dx), _angle_index(phi, L, k, dx)
    v = torch.fft.fftshift(torch.fft.fft(u.to(torch.complex128) - ref, n=L, dim=1), dim=1)[:, lo:hi + 1]  # along y
    w = v.conj().t().contiguous()  # [window of y][x]
    out = torch.empty(w.shape[0], hi - lo + 1, dtype=torch.float64, device=u.device)
    for i in range(0, w.shape[0], 256):
        f = torch.fft.fftshift(torch.fft.fft(w[i:i + 256], n=L, dim=1), dim=1)[:, lo:hi + 1]
        out[i:i + 256] = (f.real ** 2 + f.imag ** 2) / L
    return out


def _on(a, dev, dtype):
    return torch.as_tensor(a, device=dev).to(dtype)


def exact(case, seed):
    dev = _device()
    kind = case["kind"]
    if kind == "batch":
        return [_job_exact(j, dev) for j in _jobs(case, seed)]
    xmin, xmax, dx, zmin, dz, k = _grid(case)
    if kind == "farfield":
        u, ref = _scattered(case, seed, dev)
        return _farfield_exact(u, ref, max(case["pad"], case["n"]), case["phi"], k, dx).cpu().numpy()
    if kind in ("fft2d", "cn"):
        u0, delta, beta = _inputs_2d(case, seed)
        u0 = _on(u0, dev, torch.complex128)
        delta, beta = _on(delta, dev, torch.float64), _on(beta, dev, torch.float64)
        n, steps, every = case["n"], case["steps"], case["save_every"]
        flux = []
        if kind == "fft2d":
            u, saved = _fft2d_exact(u0, delta, beta, dx, dz, k, steps, every)
        else:
            if n > 4096 and steps > 1500:
                return None
            w = _windows(case)
            u, saved, flux = _cn_exact(u0, delta, beta, dx, dz, k, steps, every, (w[0][0], w[1][0]) if case["medium"] == "curved" else None)
        u = u.cpu().numpy()
        if case["medium"] == "curved":
            return {"u": u, "flux": torch.stack(flux).cpu().numpy()}
        if every:
            return {"u": u, "saved": torch.stack(saved).cpu().numpy() if saved else np.empty((0, n), np.complex128)}
        return u
    u0, spheres = _inputs_3d(case, seed, dev)
    u0, x = u0.to(torch.complex128), _axis(case, dev)
    if kind == "adi":
        return _adi_exact(u0, spheres, x, dx, zmin, dz, k, case["steps"])
    absorber = (0.1 * (xmax - xmin), 0.05 * (xmax - xmin)) if case["absorber"] else None
    return _fft3d_exact(u0, spheres, x, dx, zmin, dz, k, case["steps"], absorber)


def _job_exact(j, dev):
    k = 2.0 * math.pi / LAMBDA
    if j.kind == "fft3d":
        dx = _step_for(-1000.0, 1000.0, j.n)
        x = -1000.0 + torch.arange(j.n, dtype=torch.float64, device=dev) * dx
        return _fft3d_exact(torch.ones(j.n, j.n, dtype=torch.complex128, device=dev), j.spheres, x, dx, 0.0, 2000.0, k, j.nsteps)
    dx = _step_for(-250.0, 250.0, j.n)
    x = -250.0 + np.arange(j.n) * dx
    d, b = (_on(v, dev, torch.float64)[None, None] for v in _guide(x, j.core_half_width, j.delta_clad))
    u0 = _on(np.exp(-(x / j.waist) ** 2), dev, torch.complex128)
    if j.kind == "fft2d":
        return _fft2d_exact(u0, d, b, dx, 1000.0, k, j.nsteps, 0)[0]
    return _cn_exact(u0, d, b, dx, 500.0, k, j.nsteps, 0)[0]
