"""What the speed of this package is measured on.

Each case is one piece of work that a program built on the package asks for
through a public entry point: a misfit with its gradient (one frequency of an
NCG update), the same with a curvature-vector product, a block of
right-hand sides on a factorized operator, the two block-LU drop-ins, the RF
preparation, the RF simulation and the NCG rules between two oracle calls.

``listed()`` names fixed sizes, ``draw(rng)`` gives others of the same ranges:
interior grids of 48 to 512 cells a side (square or not) with a PML of 8 to 20
cells, 0.25-0.5 mm cells, 4 to 10 points per wavelength, 4 to 256
transmitters, every precision profile.

``prepare`` makes the inputs from the seed (phantoms, ring arrays and
ray-traced observations; nothing of them comes out of the package), ``run`` is
one pass, ``work`` the bytes and operations that the pass cannot do without,
``exact`` the same outputs in 64 bits by plain torch and NumPy.
"""
from __future__ import annotations

import ctypes as C
import math
import os
import tempfile

import numpy as np
import torch

STENCIL_BOUNDS = (1400.0, 1700.0)
PML_STRENGTH = 10.0


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # one gradient of the full-size array in the fast profile: what every NCG update of a reconstruction costs
        dict(name="gradient 552x552 tf32", kind="misfit", ny=552, nx=552, pml=20, dx=0.25e-3, ppw=5.0, n_tx=256, n_rx=256,
             precision="tf32-refined", hessian=False),
        # the same in the reference's arithmetic, which is the default profile
        dict(name="gradient 552x552 c64", kind="misfit", ny=552, nx=552, pml=20, dx=0.25e-3, ppw=5.0, n_tx=256, n_rx=256,
             precision="c64", hessian=False),
        # a mid-size array, the gradient and a Gauss-Newton product along a direction (truncated-Newton steps)
        dict(name="hessian 288x288 tf32", kind="misfit", ny=288, nx=288, pml=16, dx=0.3e-3, ppw=6.25, n_tx=64, n_rx=128,
             precision="tf32-refined", hessian=True),
        # a few transmitters on a mid-size grid, default profile
        dict(name="gradient 224x224 c64", kind="misfit", ny=224, nx=224, pml=16, dx=0.4e-3, ppw=7.5, n_tx=32, n_rx=128,
             precision="c64", hessian=False),
        # the smallest reconstructions (tests, tutorials): launches and host work count
        dict(name="gradient 64x64 c64-refined", kind="misfit", ny=64, nx=64, pml=8, dx=0.5e-3, ppw=10.0, n_tx=6, n_rx=24,
             precision="c64-refined", hessian=False),
        # right-hand sides on a kept factorization, odd sizes: adjoint fields with the mass stencil, forward fields
        # with their virtual sources
        dict(name="solve 437x401 tf32", kind="solve", ny=437, nx=401, pml=20, dx=0.3e-3, ppw=5.5, n_src=97,
             precision="tf32-refined"),
        # the two MEX drop-ins, as the MATLAB solver calls them
        dict(name="block LU 283x251", kind="blocklu", ny=283, nx=251, pml=16, dx=0.3e-3, ppw=6.0, n_src=50),
        # RF records -> complex observations: a full array's records, float32
        dict(name="prepare 2048x256x256 f32", kind="prepare", n_time=2048, n_rx=256, n_tx=256, n_f=16, double=False),
        # a small, ragged float64 record with many frequencies
        dict(name="prepare 700x9x13 f64", kind="prepare", n_time=700, n_rx=9, n_tx=13, n_f=37, double=True),
        # RF of a full-size array on its 512 x 512 model grid
        dict(name="simulate 512x512 64 tx", kind="simulate", ny=512, nx=512, pml=20, dx=0.25e-3, n_time=200, n_tx=64,
             n_rx=256, decimation=1),
        # the smallest record: a few transmitters on a few hundred cells
        dict(name="simulate 23x27 3 tx", kind="simulate", ny=23, nx=27, pml=10, dx=0.5e-3, n_time=400, n_tx=3, n_rx=4,
             decimation=2),
        # the rules between two oracle calls of a reconstruction, on the device
        dict(name="ncg rules 552x552", kind="ncg", ny=552, nx=552, pml=20, dx=0.25e-3, cutoff=0.75),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["misfit", "misfit", "misfit", "solve", "blocklu", "prepare", "simulate", "ncg"])
    if kind == "prepare":
        return dict(kind=kind, n_time=_log(rng, 200, 2048), n_rx=_log(rng, 4, 256), n_tx=_log(rng, 3, 256),
                    n_f=_log(rng, 1, 40), double=rng.random() < 0.4)
    if kind == "simulate":
        ny = _log(rng, 20, 512)
        nx = max(20, min(512, int(ny * rng.uniform(0.8, 1.25))))
        n_tx = _log(rng, 2, 64)
        return dict(kind=kind, ny=ny, nx=nx, pml=rng.randint(8, 20), dx=rng.choice([0.25e-3, 0.4e-3, 0.5e-3]),
                    n_time=rng.randint(100, 200 if ny > 128 else 400), n_tx=n_tx, n_rx=min(256, 2 * n_tx + rng.randint(1, 9)),
                    decimation=rng.choice([1, 2]))
    interior = _log(rng, 48, 512)
    pml = 8 if interior < 100 else rng.randint(16, 20)
    ny = interior + 2 * pml
    nx = max(64, min(552, int(ny * rng.uniform(0.85, 1.15))))
    case = dict(kind=kind, ny=ny, nx=nx, pml=pml, dx=rng.choice([0.25e-3, 0.3e-3, 0.4e-3]))
    if kind == "ncg":
        return dict(case, cutoff=rng.choice([0.0, 0.5, 0.75]))
    case["ppw"] = round(rng.uniform(5.0, 10.0), 2)
    if kind == "blocklu":
        return dict(case, ny=min(ny, 400), nx=min(nx, 400), n_src=_log(rng, 1, 128))
    precision = rng.choice(["c64", "c64-refined", "tf32-refined", "tf32-refined", "bf16-refined"])
    if precision == "c64-refined":
        case.update(ny=min(ny, 420), nx=min(nx, 420))
    if kind == "solve":
        return dict(case, n_src=_log(rng, 1, 256), precision=precision)
    n_tx = _log(rng, 4, 256)
    n_rx = max(n_tx, rng.choice([24, 64, 128, 200, 256]))
    n_rx = min(n_rx, max(16, interior))                   # elements that a ring can hold apart
    return dict(case, n_tx=min(n_tx, n_rx), n_rx=n_rx, precision=precision,
                hessian=max(case["ny"], case["nx"]) <= 420 and rng.random() < 0.3)


# ---------------------------------------------------------------------------
# inputs: phantoms, ring arrays, observations
# ---------------------------------------------------------------------------

def _axis(n, d):
    return -n * d / 2 + (np.arange(n) + 0.5) * d


def _smooth(rng, shape, sigma):
    """Gaussian-filtered noise of unit deviation, sigma in cells."""
    ky, kx = np.fft.fftfreq(shape[0])[:, None], np.fft.rfftfreq(shape[1])[None, :]
    filt = np.exp(-2 * (np.pi * sigma) ** 2 * (kx ** 2 + ky ** 2))
    out = np.fft.irfft2(np.fft.rfft2(rng.standard_normal(shape)) * filt, s=shape)
    return out / max(out.std(), 1e-30)


def _phantom(rng, x, y, radius):
    """Water, a breast-like disk with round inclusions, texture (m/s)."""
    X, Y = np.meshgrid(x, y)
    c = np.full(X.shape, 1500.0)
    disk = X ** 2 + Y ** 2 < (0.8 * radius) ** 2
    c[disk] = 1470.0
    for _ in range(int(rng.integers(5, 16))):
        r0, th, rad = rng.uniform(0, 0.6 * radius), rng.uniform(0, 2 * np.pi), rng.uniform(0.04, 0.15) * radius
        c[(X - r0 * np.cos(th)) ** 2 + (Y - r0 * np.sin(th)) ** 2 < rad ** 2] = rng.uniform(1520, 1580)
    c[disk] += 5.0 * _smooth(rng, X.shape, 2.0)[disk]
    return c


def _ring(n, x, y, pml):
    """1-based column-major samples of n elements on an ellipse inside the PML, and their coordinates."""
    dx = x[1] - x[0]
    a = 0.86 * (x.size / 2 - pml) * dx
    b = 0.86 * (y.size / 2 - pml) * dx
    th = 2 * np.pi * np.arange(n) / n
    ix = np.clip(np.round((a * np.cos(th) - x[0]) / dx), pml, x.size - 1 - pml).astype(np.int64)
    iy = np.clip(np.round((b * np.sin(th) - y[0]) / dx), pml, y.size - 1 - pml).astype(np.int64)
    lin = iy + y.size * ix + 1
    _, first = np.unique(lin, return_index=True)          # elements that fall on one sample are one element
    keep = np.sort(first)
    return lin[keep], np.stack([x[ix[keep]], y[iy[keep]]], 1)


def _traced(c, x, y, src, rec, f):
    """Observations of a phantom: straight-ray travel times, 2-D spreading."""
    dx = x[1] - x[0]
    s = torch.as_tensor(1.0 / c, device="cuda")
    a, b = torch.as_tensor(src, device="cuda"), torch.as_tensor(rec, device="cuda")
    r = torch.sqrt(((a[:, None] - b[None]) ** 2).sum(-1)).clamp_min(dx)
    mean = torch.zeros_like(r)
    steps = 96
    for i in range(steps):
        t = (i + 0.5) / steps
        p = a[:, None] * (1 - t) + b[None] * t
        ix = ((p[..., 0] - x[0]) / dx).round().long()
        iy = ((p[..., 1] - y[0]) / dx).round().long()
        mean = mean + s[iy, ix]
    tau = r * mean / steps
    k = 2 * math.pi * f / 1500.0
    amp = dx * dx / torch.sqrt(8 * math.pi * k * r)
    ph = -2 * math.pi * f * tau - math.pi / 4
    return torch.complex(amp * torch.cos(ph), amp * torch.sin(ph)).cpu().numpy()


def _model(case, seed):
    rng = np.random.default_rng(seed)
    x, y = _axis(case["nx"], case["dx"]), _axis(case["ny"], case["dx"])
    radius = (min(case["ny"], case["nx"]) / 2 - case["pml"]) * case["dx"]
    true = _phantom(rng, x, y, radius)
    # an iterate between the homogeneous start and the phantom: what every update after the first one sees
    return rng, x, y, true, 1500.0 + 0.5 * (true - 1500.0)


def _frequency(case):
    return 1500.0 / (case["ppw"] * case["dx"])


def _misfit_inputs(case, seed):
    rng, x, y, true, c = _model(case, seed)
    f = _frequency(case)
    rx, at = _ring(case["n_rx"], x, y, case["pml"])
    pick = np.unique((np.arange(case["n_tx"]) * rx.size) // case["n_tx"])
    tx = rx[pick]
    Y = _traced(true, x, y, at[pick], at, f).astype(np.complex64)[:, :, None]
    mask = rng.random(Y.shape) > 0.02                       # dead traces
    mask[np.arange(tx.size), pick] = False                  # a transmitter does not hear itself
    slowness = torch.as_tensor(1.0 / c, device="cuda").to(torch.float32)
    v = torch.as_tensor(1e-5 * _smooth(rng, c.shape, 6.0), device="cuda").to(torch.float32) if case["hessian"] else None
    return dict(x=x, y=y, f=f, tx=tx, rx=rx, Y=Y, mask=mask, slowness=slowness, v=v)


def _solve_inputs(case, seed):
    _, x, y, _, c = _model(case, seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    src = torch.zeros((case["n_src"], case["nx"], case["ny"], 2), device="cuda")
    src[:, 1:-1, 1:-1] = torch.randn((case["n_src"], case["nx"] - 2, case["ny"] - 2, 2), generator=g, device="cuda")
    return dict(x=x, y=y, c=c, f=_frequency(case), src=torch.view_as_complex(src).permute(2, 1, 0))


def _blocklu_inputs(case, seed):
    q = _solve_inputs(case, seed)
    op = _operator(q["x"], q["y"], q["c"], q["f"], case["pml"] * case["dx"])
    names = ("Ld", "Ll", "Lu", "Dd", "Dl", "Du", "Ud", "Ul", "Uu")
    return dict(blocks=[torch.as_tensor(op[n], device="cuda").to(torch.complex64).t().contiguous().t() for n in names],
                src=q["src"])


def _prepare_inputs(case, seed):
    rng = np.random.default_rng(seed)
    dt = 1.0 / 12.5e6
    t = -2e-6 + np.arange(case["n_time"]) * dt
    f = np.linspace(0.3e6, 1.2e6, case["n_f"]) if case["n_f"] > 1 else np.array([0.8e6])
    f = f[rng.permutation(f.size)]
    dtype = torch.float64 if case["double"] else torch.float32
    g = torch.Generator(device="cuda").manual_seed(seed)
    n_tr = case["n_rx"] * case["n_tx"]
    # a tone burst at its own arrival in each trace, with noise
    tt = torch.as_tensor(t, device="cuda")
    rf = torch.empty((n_tr, case["n_time"]), dtype=dtype, device="cuda")
    arrive = torch.rand((n_tr, 1), generator=g, device="cuda", dtype=torch.float64) * (t[-1] - t[0]) * 0.8 + t[0]
    for first in range(0, n_tr, 8192):
        u = tt[None] - arrive[first:first + 8192]
        rf[first:first + 8192] = (torch.sin(2 * math.pi * 0.7e6 * u) * torch.exp(-((u - 2e-6) / 1e-6) ** 2)).to(dtype)
    rf += 0.01 * torch.randn(rf.shape, generator=g, device="cuda", dtype=torch.float32).to(dtype)
    active = rng.random((case["n_tx"], case["n_rx"])) > 0.03
    return dict(t=t, f=f, rf=rf.view(case["n_tx"], case["n_rx"], case["n_time"]).permute(2, 1, 0), active=active)


def _simulate_inputs(case, seed):
    rng = np.random.default_rng(seed)
    x, y = _axis(case["nx"], case["dx"]), _axis(case["ny"], case["dx"])
    radius = min(case["ny"], case["nx"]) / 2 * case["dx"]
    c = _phantom(rng, x, y, radius)
    rx, _ = _ring(case["n_rx"], x, y, 1)
    tx = rx[np.unique((np.arange(case["n_tx"]) * rx.size) // case["n_tx"])]
    dt = 0.25 * case["dx"] / 1650.0
    t = np.arange(case["n_time"]) * dt
    f0 = 1500.0 / (6 * case["dx"])
    source = np.sin(2 * np.pi * f0 * t) * np.exp(-((t - 1.5 / f0) * f0) ** 2)
    model = dict(c_mps=c, x_m=x, y_m=y, tx_index=tx, rx_index=rx, dt_s=dt, source_pressure=source)
    cfg = dict(backend="native-batch", pml_size=case["pml"], density_kg_m3=1000.0, sound_speed_ref_mps=1650.0,
               downsample_factor=case["decimation"], time_offset_s=0.0, work_dir=os.path.join(tempfile.gettempdir(), "wust_rf"))
    return model, cfg


def _ncg_inputs(case, seed):
    rng, x, y, _, c = _model(case, seed)
    shape = c.shape
    X, Y = np.meshgrid(x, y)
    mask = X ** 2 + Y ** 2 < (0.8 * (min(shape) / 2 - case["pml"]) * case["dx"]) ** 2
    g = 1e-9 * (_smooth(rng, shape, 3.0) + 0.3 * rng.standard_normal(shape))
    prev_z = np.where(mask, 1e-9 * _smooth(rng, shape, 4.0), 0.0)
    direction = -prev_z
    prev_gz = 0.9 * float(np.sum(prev_z ** 2))
    slope = float(np.sum((g * mask) ** 2))
    return dict(x=x, y=y, c=c, mask=mask, g=g, prev_z=prev_z, direction=direction, prev_gz=prev_gz, f=0.6e6,
                curvature=slope / 2e3, c0=1500.0)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------

_size_in_pool = [None]


def _one_size_in_the_pool(case):
    """The package keeps a solver per grid and profile; a program works on one grid at a time."""
    from waveforminversionust_b200.objective import POOL
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if _size_in_pool[0] != key:
        POOL.clear()
        _size_in_pool[0] = key


def prepare(case, seed):
    kind = case["kind"]
    if kind == "misfit":
        from waveforminversionust_b200.objective import POOL, Observations, default_config
        _one_size_in_the_pool(case)
        q = _misfit_inputs(case, seed)
        obs = Observations(q["x"], q["y"], q["tx"], q["rx"], np.array([q["f"]]), q["Y"], q["mask"])
        cfg = default_config(pml_m=case["pml"] * case["dx"], pml_strength=PML_STRENGTH, stencil_bounds=STENCIL_BOUNDS,
                             precision=case["precision"])
        POOL.get(1.0 / q["slowness"].double().cpu().numpy(), obs, 0, cfg)      # the solver that a program keeps
        return dict(kind=kind, slowness=q["slowness"].requires_grad_(True), obs=obs, cfg=cfg, v=q["v"])
    if kind == "solve":
        from waveforminversionust_b200.solver import HelmholtzSolver
        q = _solve_inputs(case, seed)
        solver = HelmholtzSolver(q["x"], q["y"], q["c"], None, q["f"], -1, PML_STRENGTH, case["pml"] * case["dx"],
                                 dict(backend="gpu", stencil_bounds=STENCIL_BOUNDS), precision=case["precision"],
                                 max_sources=case["n_src"])
        return dict(kind=kind, solver=solver, src=q["src"])
    if kind == "blocklu":
        return dict(_blocklu_inputs(case, seed), kind=kind)
    if kind == "prepare":
        return dict(_prepare_inputs(case, seed), kind=kind)
    if kind == "simulate":
        model, cfg = _simulate_inputs(case, seed)
        return dict(kind=kind, model=model, cfg=cfg)
    from waveforminversionust_b200.solver import HelmholtzSolver
    q = _ncg_inputs(case, seed)
    solver = HelmholtzSolver(q["x"], q["y"], q["c"], None, 0.3e6, -1, PML_STRENGTH, case["pml"] * case["dx"],
                             dict(backend="gpu", stencil_bounds=STENCIL_BOUNDS), max_sources=1)
    dev = {k: torch.as_tensor(np.ascontiguousarray(q[k].T), device="cuda") for k in ("c", "g", "prev_z", "direction")}
    mask = torch.as_tensor(np.ascontiguousarray(q["mask"].T).astype(np.uint8), device="cuda")
    return dict(q, **dev, mask=mask, roi=torch.empty_like(dev["c"]), z=torch.empty_like(dev["c"]), kind=kind, solver=solver,
                cutoff=case["cutoff"])


def run(state):
    kind = state["kind"]
    if kind == "misfit":
        from waveforminversionust_b200.autograd import misfit
        s = state["slowness"]
        loss = misfit(s, state["obs"], 0, state["cfg"])
        if state["v"] is None:
            (g,) = torch.autograd.grad(loss, s)
            return dict(loss=loss.detach().to(s.dtype), gradient=g)
        (g,) = torch.autograd.grad(loss, s, create_graph=True)
        (h,) = torch.autograd.grad(g, s, state["v"])
        return dict(loss=loss.detach().to(s.dtype), gradient=g.detach(), product=h)
    if kind == "solve":
        solver = state["solver"]
        u, v = solver.solve(state["src"], want_virtual=True)
        lam = solver.massApply(solver.solve(state["src"], adjoint=True), True)
        return dict(u=u, v=v, lam=lam)
    if kind == "blocklu":
        from waveforminversionust_b200.solver import applyBlockLU, decompBlockLU
        b = state["blocks"]
        inv = decompBlockLU(*b)
        sides = [b[i] for i in (0, 1, 2, 6, 7, 8)]
        return dict(inv=inv, u=applyBlockLU(state["src"], *sides, inv, False),
                    lam=applyBlockLU(state["src"], *sides, inv, True))
    if kind == "prepare":
        from waveforminversionust_b200.prepare import dtft_device
        return dict(Y=dtft_device(state["t"], state["f"], state["rf"], state["active"]))
    if kind == "simulate":
        from waveforminversionust_b200.simulate import wust_simulate
        return dict(pressure=wust_simulate(state["model"], state["cfg"])["pressure"])
    return _run_ncg(state)


def _run_ncg(state):
    """What the device-resident reconstruction loop does between two oracle calls."""
    from waveforminversionust_b200 import _lib
    from waveforminversionust_b200.ncg import linearized_step_length
    lib, check = _lib.load(), _lib.check
    h = C.c_void_p(state["solver"].handle)

    def ptr(t):
        return C.c_void_p(t.data_ptr())

    c, direction = state["c"].clone(), state["direction"].clone()       # the loop updates them in place
    roi, z, mask = state["roi"], state["z"], state["mask"]
    check(lib.wust_ncg_roi_gradient(h, ptr(state["g"]), ptr(mask), state["c0"], state["f"], state["cutoff"], 4.0, ptr(roi), ptr(z)))
    beta, gz, slope, rel = C.c_double(), C.c_double(), C.c_double(), C.c_double()
    check(lib.wust_ncg_direction(h, ptr(roi), ptr(z), ptr(state["prev_z"]), C.c_double(state["prev_gz"]), 1,
                                 ptr(direction), C.byref(beta), C.byref(gz)))
    check(lib.wust_ncg_dot(h, ptr(roi), ptr(direction), C.byref(slope)))
    alpha = linearized_step_length(slope.value, state["curvature"])
    check(lib.wust_ncg_project(h, ptr(c), ptr(direction), C.c_double(alpha), 1.0, 12.0, 1350.0, 1750.0, ptr(mask),
                               C.byref(rel)))
    return dict(c=c, direction=direction, z=z, beta=beta.value, gz=gz.value, relative_update=rel.value)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    if kind == "prepare":
        n, tr = case["n_time"], case["n_rx"] * case["n_tx"]
        return dict(bytes=n * tr * (8 if case["double"] else 4) + tr * (1 + 8 * case["n_f"]), flops=4.0 * n * tr * case["n_f"])
    N = case["ny"] * case["nx"]
    if kind == "simulate":
        M = (case["ny"] + 2 * case["pml"]) * (case["nx"] + 2 * case["pml"])
        out = case["n_tx"] * case["n_rx"] * -(-case["n_time"] // case["decimation"])
        # per transmitter and step: the split velocity and density fields read and written, seven real transforms
        steps = case["n_tx"] * case["n_time"]
        return dict(bytes=steps * M * 32.0 + 4.0 * out, flops=steps * M * (7 * 2.5 * math.log2(M) + 40))
    if kind == "ncg":
        return dict(bytes=N * (8 * 7 + 1), flops=N * (60 + (5 * math.log2(N) if case["cutoff"] else 0)))
    n, nx = case["ny"] - 2, case["nx"]
    factor = 8.0 * n ** 3 * nx
    pair = lambda s: 16.0 * n * n * s * nx                    # one forward and one backward substitution
    if kind == "blocklu":
        return dict(bytes=8.0 * (9 * N + case["ny"] ** 2 * nx + 3 * N * case["n_src"]), flops=factor + 2 * pair(case["n_src"]))
    if kind == "solve":
        return dict(bytes=8.0 * (case["ny"] ** 2 * nx + 4 * N * case["n_src"]), flops=2 * pair(case["n_src"]))
    pairs = 4 if case["hessian"] else 2
    return dict(bytes=4.0 * N * (3 if case["hessian"] else 2) + 9.0 * case["n_tx"] * case["n_rx"],
                flops=factor + pairs * pair(case["n_tx"]))


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _stencil_weights(f, h, g=1.0):
    """Least-squares mass weights of the nine-point stencil between the two speeds."""
    lo, hi = (v / (f * h) for v in STENCIL_BOUNDS)
    th = np.arange(100) * np.pi / 396
    G = 1.0 / (1.0 / hi + np.arange(10) / 9 * (1.0 / lo - 1.0 / hi))
    th, G = np.meshgrid(th, G)
    P, Q = np.cos(2 * np.pi * g * np.cos(th) / G), np.cos(2 * np.pi * np.sin(th) / G)
    b = 5.0 / 6.0
    A = np.stack([(np.pi ** 2 * (2 - P - Q)).ravel(), (2 * np.pi ** 2 * (1 - P * Q)).ravel()], 1)
    rhs = (2 * np.pi ** 2 + G ** 2 * ((1 + 1 / g ** 2) * P * Q - P - Q / g ** 2)
           - b * (1 + 1 / g ** 2) * G ** 2 * (1 - P - Q + P * Q)).ravel()
    d, e = np.linalg.lstsq(A, rhs, rcond=None)[0]
    return b, float(d), float(e)


def _operator(x, y, c, f, pml_m):
    """The nine coefficient arrays of the PML Helmholtz operator (square cells, time sign -1), the factor of the
    virtual sources and the mass weights."""
    ny, nx = c.shape
    h = float(np.mean(np.diff(x)))
    b, d, e = _stencil_weights(f, h)

    def stretch(v):
        p = np.linspace(v[0], v[-1], 2 * v.size - 1)
        mid, half = (v[0] + v[-1]) / 2, (v[-1] - v[0]) / 2
        return 1 - 1j * PML_STRENGTH * (np.maximum(np.abs(p - mid) - half + pml_m, 0) / pml_m) ** 2

    ex, ey = stretch(x)[None, :], stretch(y)[:, None]
    A = (ey / ex)[0::2, 1::2] * b / h ** 2             # (ny, nx-1)
    B = (ex / ey)[1::2, 0::2] * b / h ** 2             # (ny-1, nx)
    r = (1 - b) / (2 * b)
    Cm = (ex * ey)[0::2, 0::2]
    q = Cm * (2 * np.pi * f / c) ** 2
    z = lambda m, n: np.zeros((m, n), complex)
    o = dict(Dd=z(ny, nx), Dl=z(ny - 1, nx), Du=z(ny - 1, nx), Ld=z(ny, nx - 1), Ll=z(ny - 1, nx - 1), Lu=z(ny - 1, nx - 1),
             Ud=z(ny, nx - 1), Ul=z(ny - 1, nx - 1), Uu=z(ny - 1, nx - 1))
    i, I = slice(1, ny - 1), slice(1, nx - 1)           # interior rows, columns
    up, dn = slice(0, ny - 2), slice(2, ny)
    lf, rt = slice(0, nx - 2), slice(2, nx)
    o["Dd"][[0, -1], :] = 1
    o["Dd"][:, [0, -1]] = 1
    o["Dd"][i, I] = (1 - d - e) * q[i, I] - (A[i, 1:] + A[i, :-1] + B[1:, I] + B[:-1, I])
    o["Dl"][up, I] = B[up, I] - r * (A[up, 1:] + A[up, :-1]) + d / 4 * q[up, I]
    o["Du"][i, I] = B[i, I] - r * (A[dn, 1:] + A[dn, :-1]) + d / 4 * q[dn, I]
    o["Ld"][i, lf] = A[i, lf] - r * (B[1:, lf] + B[:-1, lf]) + d / 4 * q[i, lf]
    o["Ll"][up, lf] = r * (A[up, lf] + B[up, lf]) + e / 4 * q[up, lf]
    o["Lu"][i, lf] = r * (A[dn, lf] + B[i, lf]) + e / 4 * q[dn, lf]
    o["Ud"][i, I] = A[i, I] - r * (B[1:, rt] + B[:-1, rt]) + d / 4 * q[i, rt]
    o["Ul"][up, I] = r * (A[up, I] + B[up, rt]) + e / 4 * q[up, rt]
    o["Uu"][i, I] = r * (A[dn, I] + B[i, rt]) + e / 4 * q[dn, rt]
    return dict(o, mult=Cm * 8 * np.pi ** 2 * f ** 2 / c, d=d, e=e)


def _cols(a):
    """(rows, columns) -> a list of columns, on the GPU in complex128."""
    t = a if isinstance(a, torch.Tensor) else torch.as_tensor(a, device="cuda")
    return t.to(torch.complex128).t().contiguous()


def _tri(dg, lo, up, v):
    """A tridiagonal matrix (diagonal, below, above) times v (rows, n)."""
    out = dg[:, None] * v
    out[1:] += lo[:, None] * v[:-1]
    out[:-1] += up[:, None] * v[1:]
    return out


class _Exact:
    """Block LU of the operator in complex128: pages inv(T_j) with zero border rows and columns."""

    def __init__(self, op):
        for n in ("Dd", "Dl", "Du", "Ld", "Ll", "Lu", "Ud", "Ul", "Uu"):
            setattr(self, n, _cols(op[n]))
        self.nx, self.ny = self.Dd.shape
        self.inv = torch.zeros((self.nx, self.ny, self.ny), dtype=torch.complex128, device="cuda")
        for j in range(self.nx):
            T = torch.diag(self.Dd[j]) + torch.diag(self.Dl[j], -1) + torch.diag(self.Du[j], 1)
            if j:
                right = _tri(self.Ud[j - 1], self.Uu[j - 1], self.Ul[j - 1], self.inv[j - 1].t()).t()
                T = T - self.L(j - 1, right)
            self.inv[j, 1:-1, 1:-1] = torch.linalg.inv(T[1:-1, 1:-1])

    def L(self, j, v):
        return _tri(self.Ld[j], self.Ll[j], self.Lu[j], v)

    def U(self, j, v):
        return _tri(self.Ud[j], self.Ul[j], self.Uu[j], v)

    def LH(self, j, v):
        return _tri(self.Ld[j].conj(), self.Lu[j].conj(), self.Ll[j].conj(), v)

    def UH(self, j, v):
        return _tri(self.Ud[j].conj(), self.Uu[j].conj(), self.Ul[j].conj(), v)

    def solve(self, src, adjoint=False, inv=None):
        """src (nx, ny, n) -> the block sweeps, column 0 and n - 1 as the drop-in leaves them."""
        inv = self.inv if inv is None else inv
        u = torch.zeros(src.shape, dtype=torch.complex128, device="cuda")
        last = self.nx - 1
        if not adjoint:
            for j in range(1, self.nx):
                u[j] = inv[j] @ (src[j] - self.L(j - 1, u[j - 1]))
            for j in range(last - 1, -1, -1):
                u[j] -= inv[j] @ self.U(j, u[j + 1])
        else:
            for j in range(1, self.nx):
                u[j] = src[j] - self.UH(j - 1, inv[j - 1].mH @ u[j - 1])
            for j in range(last - 1, -1, -1):
                u[j] = inv[j].mH @ (u[j] - self.LH(j, u[j + 1]))
        return u


def _mass(v, d, e, adjoint):
    """The mass stencil on (nx, ny, n) fields: the ring is zero before (adjoint) or after it."""
    def ring(a):
        a[[0, -1]] = 0
        a[:, [0, -1]] = 0
        return a
    if adjoint:
        v = ring(v.clone())
    pad = torch.zeros((v.shape[0] + 2, v.shape[1] + 2, v.shape[2]), dtype=v.dtype, device=v.device)
    pad[1:-1, 1:-1] = v
    out = torch.zeros_like(v)
    for a in range(3):
        for b in range(3):
            w = (1 - d - e, d / 4, e / 4)[(a != 1) + (b != 1)]
            out += w * pad[a:a + v.shape[0], b:b + v.shape[1]]
    return out if adjoint else ring(out)


def _exact_misfit(case, seed):
    q = _misfit_inputs(case, seed)
    s = q["slowness"].double().cpu().numpy()
    op = _operator(q["x"], q["y"], 1.0 / s, q["f"], case["pml"] * case["dx"])
    lu = _Exact(op)
    ny, nx, S = case["ny"], case["nx"], q["tx"].size
    tx, rx = torch.as_tensor(q["tx"] - 1, device="cuda"), torch.as_tensor(q["rx"] - 1, device="cuda")
    Y = torch.as_tensor(q["Y"][:, :, 0], device="cuda").to(torch.complex128)
    m = torch.as_tensor(q["mask"][:, :, 0], device="cuda").double()
    Y = Y * m
    src = torch.zeros((nx * ny, S), dtype=torch.complex128, device="cuda")
    src[tx, torch.arange(S, device="cuda")] = 1
    u = lu.solve(src.view(nx, ny, S))
    p = u.view(nx * ny, S)[rx].t() * m
    a = (p.conj() * Y).sum(1) / (p.abs() ** 2).sum(1)
    res = (a[:, None] * p - Y) * m
    av = a * torch.as_tensor(op["mult"], device="cuda").t()[:, :, None] * u

    def back(r):                                            # -Re(conj(a v) . M^T H^-H r), summed over transmitters
        b = torch.zeros((nx * ny, S), dtype=torch.complex128, device="cuda")
        b[rx] = r.t()
        lam = _mass(lu.solve(b.view(nx, ny, S), True), op["d"], op["e"], True)
        return -(av.real * lam.real + av.imag * lam.imag).sum(2).t()

    out = dict(loss=0.5 * (res.abs() ** 2).sum(), gradient=back(res))
    if case["hessian"]:
        v = q["v"].double().t()[:, :, None]
        # J v with the source scales frozen: -a H^-1 M (mult u v) at the receivers
        w = lu.solve(_mass(torch.as_tensor(op["mult"], device="cuda").t()[:, :, None] * u * v, op["d"], op["e"], False))
        out["product"] = back(-a[:, None] * w.view(nx * ny, S)[rx].t() * m)
    return out


def _exact_ncg(case, seed):
    q = _ncg_inputs(case, seed)
    roi = np.where(q["mask"], q["g"], 0.0)
    z = roi
    if case["cutoff"]:
        ky = np.fft.fftfreq(case["ny"], np.mean(np.diff(q["y"])))[:, None]
        kx = np.fft.fftfreq(case["nx"], np.mean(np.diff(q["x"])))[None, :]
        kc = 2 * q["f"] / q["c0"] * case["cutoff"]
        z = np.real(np.fft.ifft2(np.fft.fft2(roi) / (1 + ((kx ** 2 + ky ** 2) / kc ** 2) ** 4)))
        z = np.where(q["mask"], z, 0.0)
    gz = float(np.sum(roi * z))
    beta = min(max(float(np.sum(roi * (z - q["prev_z"]))) / q["prev_gz"], 0.0), gz / q["prev_gz"])
    d = -z + beta * q["direction"]
    if float(np.sum(roi * d)) >= 0:
        d, beta = -z, 0.0
    alpha = max(0.0, -float(np.sum(roi * d)) / q["curvature"])
    lo, hi = np.maximum(q["c"] - 12.0, 1350.0), np.minimum(q["c"] + 12.0, 1750.0)
    new = np.clip(1 / q["c"] + alpha * d, 1 / hi, 1 / lo)
    c = np.where(q["mask"], 1 / new, q["c"])
    old = 1 / q["c"][q["mask"]]
    rel = float(np.linalg.norm(1 / c[q["mask"]] - old) / np.linalg.norm(old))
    T = lambda v: np.ascontiguousarray(v.T)
    return dict(c=T(c), direction=T(d), z=T(z), beta=beta, gz=gz, relative_update=rel)


def _exact_simulate(case, seed):
    model, cfg = _simulate_inputs(case, seed)
    P, dt, c_ref, rho0, d = case["pml"], model["dt_s"], cfg["sound_speed_ref_mps"], cfg["density_kg_m3"], case["dx"]
    ny, nx, nt = case["ny"], case["nx"], case["n_time"]
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")
    c2 = dev(np.pad(model["c_mps"], P, mode="edge") ** 2)
    Ny, Nx = c2.shape
    # complex transforms throughout, so that the unpaired frequencies are what the method says
    ky, kx = 2 * np.pi * np.fft.fftfreq(Ny, d)[:, None], 2 * np.pi * np.fft.fftfreq(Nx, d)[None, :]
    kappa = np.sinc(c_ref * dt * np.sqrt(ky ** 2 + kx ** 2) / (2 * np.pi))
    deriv = {n + s: dev(1j * k * np.exp((0.5j if s == "+" else -0.5j) * k * d) * kappa)
             for n, k in (("y", ky), ("x", kx)) for s in "+-"}

    def absorb(n, shift):
        out = np.ones(n)
        i = np.arange(P)
        out[:P] = np.exp(-dt * c_ref / d * ((i + shift - P) / P) ** 4)
        out[n - P:] = np.exp(-dt * c_ref / d * ((i + shift + 1) / P) ** 4)
        return out

    py, pys = dev(absorb(Ny, 0.0)[:, None]), dev(absorb(Ny, 0.5)[:, None])
    px, pxs = dev(absorb(Nx, 0.0)[None, :]), dev(absorb(Nx, 0.5)[None, :])

    def at(index):
        i = np.asarray(index) - 1
        return torch.as_tensor(i % ny + P, device="cuda"), torch.as_tensor(i // ny + P, device="cuda")

    ty, tx = at(model["tx_index"])
    ry, rx = at(model["rx_index"])
    S = ty.numel()
    uy, ux, dy, dx, p = (torch.zeros((S, Ny, Nx), dtype=torch.float64, device="cuda") for _ in range(5))
    rec = torch.zeros((nt, rx.numel(), S), dtype=torch.float64, device="cuda")
    each = torch.arange(S, device="cuda")
    back = lambda v: torch.fft.ifft2(v).real
    for t in range(nt):
        F = torch.fft.fft2(p)
        uy = pys * (pys * uy - dt / rho0 * back(deriv["y+"] * F))
        ux = pxs * (pxs * ux - dt / rho0 * back(deriv["x+"] * F))
        dy = py * (py * dy - dt * rho0 * back(deriv["y-"] * torch.fft.fft2(uy)))
        dx = px * (px * dx - dt * rho0 * back(deriv["x-"] * torch.fft.fft2(ux)))
        sv = float(model["source_pressure"][t]) / 2
        dy[each, ty, tx] = sv / c2[ty, tx]
        dx[each, ty, tx] = sv / c2[ty, tx]
        p = c2 * (dy + dx)
        rec[t] = p[:, ry, rx].t()
    rec = rec.cpu().numpy()
    q = case["decimation"]
    if q > 1:
        L = 48 * q + 1
        h = np.sinc((np.arange(L) - 24 * q) / q) / q * np.kaiser(L, 8.6)
        h /= h.sum()
        pad = np.pad(rec, ((24 * q, 24 * q + q), (0, 0), (0, 0)))
        rec = np.stack([np.tensordot(h[::-1], pad[m * q:m * q + L], 1) for m in range(-(-nt // q))])
    return dict(pressure=rec)


def exact(case, seed):
    kind = case["kind"]
    if kind == "misfit":
        return _exact_misfit(case, seed)
    if kind == "ncg":
        return _exact_ncg(case, seed)
    if kind == "simulate":
        return _exact_simulate(case, seed) if case["n_tx"] * case["n_time"] * case["ny"] * case["nx"] < 4e9 else None
    if kind == "prepare":
        q = _prepare_inputs(case, seed)
        dt = q["t"][1] - q["t"][0]
        K = torch.as_tensor(np.exp(-2j * np.pi * q["f"][None, :] * q["t"][:, None]) * dt, device="cuda")
        rf = q["rf"].permute(2, 1, 0) * torch.as_tensor(q["active"], device="cuda")[:, :, None]
        Y = torch.stack([torch.complex(r.double() @ K.real, r.double() @ K.imag) for r in rf])
        return dict(Y=Y)
    if kind == "solve":
        q = _solve_inputs(case, seed)
        op = _operator(q["x"], q["y"], q["c"], q["f"], case["pml"] * case["dx"])
        lu = _Exact(op)
        src = q["src"].permute(1, 0, 2).to(torch.complex128).contiguous()
        u = lu.solve(src)
        lam = _mass(lu.solve(src, True), op["d"], op["e"], True)
        v = torch.as_tensor(op["mult"], device="cuda").t()[:, :, None] * u
        T = lambda a: a.permute(1, 0, 2)
        return dict(u=T(u), v=T(v), lam=T(lam))
    q = _blocklu_inputs(case, seed)
    lu = _Exact(dict(zip(("Ld", "Ll", "Lu", "Dd", "Dl", "Du", "Ud", "Ul", "Uu"), q["blocks"])))
    src = q["src"].permute(1, 0, 2).to(torch.complex128).contiguous()
    T = lambda a: a.permute(1, 0, 2)
    return dict(inv=lu.inv.permute(1, 2, 0), u=T(lu.solve(src)), lam=T(lu.solve(src, True)))
