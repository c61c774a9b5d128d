"""Workloads whose time is tracked: pressure solves, RK3 steps of the
stratified shear layer (DNS, Smagorinsky and dynamic LES), batched solves
and ensemble cohorts, through the package's public entry points.

All grids are the shear-layer domain 4 pi x 2 pi x 20 (periodic x and y,
Neumann / free-slip z walls, z tanh-stretched unless the reference's own
uniform-spacing operator is asked for).  The mixed-precision solves run to
a relative residual of 1e-11 where nz is 32 times a small count and 1e-12 on
the other column lengths (whose error is about 100 times the residual): ten
and a hundred times below the benchmark's setting, so that pressure holds
the 1e-9 that the solver is asked for, and above the FP64 rounding floor of
the residual.  A pressure is determined up to a constant, so every program
below fixes it to zero interior mean before it uses it.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from anelastic_solve_b200 import abi
from anelastic_solve_b200 import grid as G
from anelastic_solve_b200.mg import MGSolver
from anelastic_solve_b200.ns import NSSolver

LX, LY, HALF = 4.0 * math.pi, 2.0 * math.pi, 10.0
FIELDS = ("u", "v", "w", "p", "rho")


def listed():
    return [
        # one pressure solve of the smallest test configuration: latency
        dict(name="solve_small", kind="solve", nx=64, ny=32, nz=64, method="mixed"),
        # a grid whose column length is not a multiple of 32
        dict(name="solve_ragged", kind="solve", nx=96, ny=48, nz=100, method="mixed"),
        # the standalone Poisson benchmark
        dict(name="solve_large", kind="solve", nx=512, ny=256, nz=512, method="mixed"),
        # the one-for-one replacement of the reference's mg_solver: FP64,
        # point smoother, uniform-spacing operator, its own stop test
        dict(name="solve_fp64", kind="solve", nx=256, ny=128, nz=128, method="literal"),
        # a serving bucket's standalone solves in one batch
        dict(name="batch_16", kind="batch", nx=64, ny=64, nz=64, members=16),
        # a short run on the CPU-runnable configuration: latency of a step
        dict(name="dns_small", kind="step", nx=64, ny=32, nz=64, model="dns", method="mixed", steps=4),
        # the DNS benchmark
        dict(name="dns_large", kind="step", nx=512, ny=256, nz=512, model="dns", method="mixed", steps=1),
        # the plain FP64 path a Fortran driver switches to first
        dict(name="dns_fp64", kind="step", nx=128, ny=64, nz=128, model="dns", method="fp64", steps=1),
        # a driver that keeps its state in host memory
        dict(name="dns_host", kind="host", nx=192, ny=96, nz=192, model="dns", method="mixed", steps=1),
        # the LES benchmark's models on half its resolution
        dict(name="les_ssm", kind="step", nx=384, ny=192, nz=192, model="ssm", method="mixed", steps=1),
        # the reference runfile's dynamic models
        dict(name="les_dsm", kind="step", nx=192, ny=96, nz=96, model="dsm", method="mixed", steps=1),
        # an ensemble of one serving bucket stepping together
        dict(name="cohort_8", kind="cohort", nx=64, ny=64, nz=64, members=8, steps=2),
    ]


def _extent(rng, lo, hi):
    """An extent {1, 3, 5} * 2^a in [lo, hi] (the level rule asks for a
    coarse grid of a few cells), log-uniform."""
    al = sorted(m << a for m in (1, 3, 5) for a in range(2, 10) if lo <= m << a <= hi)
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(al, key=lambda n: abs(math.log(n / x)))


def draw(rng):
    kind = rng.choice(("solve", "solve", "batch", "step", "step", "step", "host", "cohort"))
    c = dict(kind=kind)
    nx = _extent(rng, 16, {"solve": 512, "step": 512, "host": 256}.get(kind, 128))
    # cells up to four times longer or shorter in x than in y
    ny = _extent(rng, max(16, nx // 4), min(nx, 256))
    hi = {"solve": 512, "step": 512, "host": 256}.get(kind, 128)
    # columns of any length, and the longer ones in multiples of 32
    nz = int(math.exp(rng.uniform(math.log(24), math.log(130))))
    if kind in ("batch", "cohort"):
        # these need columns of 32 * {2, 3, 4} cells
        nz = rng.choice((64, 96, 128))
        c["members"] = rng.randint(2, 16 if kind == "batch" else 8)
    elif rng.random() < 0.6:
        nz = rng.choice([32 * m for m in (2, 3, 4, 6, 8, 12, 16) if 32 * m <= hi])
    if kind in ("solve", "step", "host"):
        c["method"] = rng.choice(("mixed", "mixed", "mixed", "fp64", "literal" if kind == "solve" else "mixed"))
        if c["method"] != "mixed":
            # the point smoother coarsens z too
            nx, ny = min(nx, 128), min(ny, 64)
            nz = _extent(rng, 32, 128)
    if kind in ("step", "host", "cohort"):
        c["steps"] = 1
    if kind in ("step", "host"):
        c["model"] = rng.choice(("dns", "dns", "ssm", "dsm"))
        if c["model"] != "dns":
            # the subgrid models cost several times a DNS step
            nx, ny, nz = min(nx, 192), min(ny, 96), min(nz, 192)
    c.update(nx=nx, ny=ny, nz=nz)
    return c


# ------------------------------------------------------------------ set-up
def _levels(nx, ny, nz, zline):
    out = []
    for n in (nx, ny, nz):
        L = 1
        while n % 2 == 0 and n // 2 >= 2:
            n //= 2
            L += 1
        out.append(L)
    if zline:
        out[2] = 1
    return tuple(out)


def _mg_params(c):
    method = c.get("method", "mixed")
    lv = _levels(c["nx"], c["ny"], c["nz"], method == "mixed")
    if method == "mixed":
        tol = 1e-11 if c["nz"] in (64, 96, 128, 192, 256, 384, 512) else 1e-12
        return abi.make_mg_params(lv, maxcy=400, tolmax=tol, precision=abi.PREC_MIXED, stop=abi.STOP_RESID,
                                  smoother=abi.SMOOTHER_ZLINE, mode=abi.MODE_METRIC)
    if method == "fp64":
        return abi.make_mg_params(lv, maxcy=400, tolmax=1e-10, stop=abi.STOP_RESID, mode=abi.MODE_METRIC)
    return abi.make_mg_params(lv, maxcy=400, tolmax=1e-9)


def _ns_params(c, Re=2000.0, Ri=0.1):
    model = c.get("model", "dns")
    les = model != "dns"
    return abi.make_ns_params(Re=50000.0 if les else Re, g=-Ri, cfl=0.5, dtmax=1e9, ew=1, scal1_on=0, les=les,
                              ssm_const=0.0289, pr_sgs=0.7,
                              models=(abi.MODEL_DSM,) * 3 if model == "dsm" else None, stretched=(0, 0, 1),
                              interp=abi.DIAG_CORRECTED)


def _grid(c):
    return G.shear_layer_grid(c["nx"], c["ny"], c["nz"], stretched=c.get("method") != "literal")


def _smooth_noise(gen, nz, ny, nx, zc):
    """A random field with the spectrum of a resolved flow (energy in the
    large scales, falling off well before the grid scale), concentrated on
    the shear layer as its pressure sources are."""
    dev = "cuda"
    kx = torch.fft.rfftfreq(nx, LX / nx / (2 * math.pi), device=dev, dtype=torch.float64)
    ky = torch.fft.fftfreq(ny, LY / ny / (2 * math.pi), device=dev, dtype=torch.float64)
    k2 = kx[None, :] ** 2 + ky[:, None] ** 2
    env = 1.0 / torch.cosh(zc / 2.0) ** 2
    out = torch.zeros(nz, ny, nx, dtype=torch.float64, device=dev)
    # a few vertical structures, each with its own horizontal pattern
    for m in range(4):
        a = torch.randn(ny, nx, generator=gen, device=dev, dtype=torch.float64)
        a = torch.fft.irfft2(torch.fft.rfft2(a) * torch.exp(-k2 / 16.0) * torch.sqrt(k2 + 0.25), s=(ny, nx))
        a = a / a.std()
        ph = 2.0 * math.pi * torch.rand(1, generator=gen, device=dev, dtype=torch.float64)
        out += (env * torch.cos(0.6 * (m + 1) * zc + ph))[:, None, None] * a
    return out


def _rhs(c, g, seed):
    """A pressure source with zero volume mean (Neumann/periodic problems
    are solvable only then), as a ghosted device array."""
    nx, ny, nz = g.shape
    gen = torch.Generator("cuda").manual_seed(seed)
    f = _smooth_noise(gen, nz, ny, nx, torch.from_numpy(g.z.xc[1:-1].copy()).cuda())
    dz = torch.from_numpy(g.z.dxc[1:-1].copy()).cuda()
    f -= (f.mean(dim=(1, 2)) * dz).sum() / dz.sum()
    out = torch.zeros(g.ghosted[::-1], dtype=torch.float64, device="cuda")
    out[1:-1, 1:-1, 1:-1] = f
    return out


def _flow(g, seed):
    """A rolled-up shear layer: the mean profile, smooth finite-amplitude
    perturbations and the benchmark's grid-scale noise on |z| < 2."""
    gen = torch.Generator("cuda").manual_seed(seed)
    Z, Y, X = g.ghosted[::-1]
    zc = torch.from_numpy(g.z.xc.copy()).cuda()
    noise = (zc.abs() < 2.0).to(torch.float64)[:, None, None]
    f = {}
    for name, amp in (("u", 0.1), ("v", 0.05), ("w", 0.1)):
        a = torch.zeros(Z, Y, X, dtype=torch.float64, device="cuda")
        a[1:-1, 1:-1, 1:-1] = amp * _smooth_noise(gen, Z - 2, Y - 2, X - 2, zc[1:-1])
        a += 1e-3 * noise * (2.0 * torch.rand(Z, Y, X, generator=gen, device="cuda", dtype=torch.float64) - 1.0)
        f[name] = a
    th = torch.tanh(zc)[:, None, None]
    f["u"] += th
    f["rho"] = (-th).expand(Z, Y, X).contiguous()
    f["p"] = torch.zeros(Z, Y, X, dtype=torch.float64, device="cuda")
    return f


def _stepper(c, g, seed, **phys):
    s = NSSolver(g, _mg_params(c), _ns_params(c, **phys))
    f = _flow(g, seed)
    torch.cuda.synchronize()
    s.set_fields(f)
    s.project()
    return s, f


def prepare(case, seed):
    g = _grid(case)
    st = {"case": case, "stream": torch.cuda.Stream()}
    if case["kind"] == "solve":
        st["solver"] = MGSolver(g, _mg_params(case))
        st["rhs"] = _rhs(case, g, seed)
        st["phi"] = torch.zeros_like(st["rhs"])
    elif case["kind"] == "batch":
        st["solver"] = MGSolver(g, _mg_params(case))
        st["rhs"] = [_rhs(case, g, 1000 * seed + b) for b in range(case["members"])]
        st["phi"] = [torch.zeros_like(r) for r in st["rhs"]]
    elif case["kind"] == "cohort":
        st["members"], st["out"] = [], []
        for b in range(case["members"]):
            # members of one bucket differ in their physics and their state
            s, f = _stepper(case, g, 1000 * seed + b, Re=500.0 * (1 + b), Ri=0.05 + 0.02 * b)
            st["members"].append(s)
            st["out"].append(f)
    else:
        st["solver"], st["out"] = _stepper(case, g, seed)
        if case["kind"] == "host":
            host = {k: torch.zeros(g.ghosted[::-1], dtype=torch.float64, pin_memory=True).numpy().T for k in FIELDS}
            st["solver"].get_into(host)
            st["host"] = host
            del st["out"]
    torch.cuda.synchronize()
    return st


# --------------------------------------------------------------- one pass
def _gauge(p):
    q = p[1:-1, 1:-1, 1:-1]
    return q - q.mean()


def run(state):
    c, stream = state["case"], state["stream"]
    h = stream.cuda_stream
    if c["kind"] in ("solve", "batch"):
        with torch.cuda.stream(stream):
            if c["kind"] == "solve":
                state["phi"].zero_()
                state["solver"].solve(state["phi"], state["rhs"], stream=h)
                return _gauge(state["phi"])
            for p in state["phi"]:
                p.zero_()
            state["solver"].solve_batch(state["phi"], state["rhs"], stream=h)
            return [_gauge(p) for p in state["phi"]]
    if c["kind"] == "host":
        state["solver"].step_host(state["host"], state["host"], c["steps"], stream=h)
        out = dict(state["host"])
        p = out["p"][1:-1, 1:-1, 1:-1]
        out["p"] = p - p.mean()
        return out
    if c["kind"] == "cohort":
        NSSolver.step_cohort(state["members"], c["steps"], stream=h)
        pairs = list(zip(state["members"], state["out"]))
    else:
        state["solver"].step(c["steps"], stream=h)
        pairs = [(state["solver"], state["out"])]
    res = []
    for s, f in pairs:
        s.get_into(f)
        o = dict(f)
        with torch.cuda.stream(stream):
            o["p"] = _gauge(f["p"])
        res.append(o)
    return res


def work(case):
    cells = case["nx"] * case["ny"] * case["nz"] * case.get("members", 1)
    if case["kind"] in ("solve", "batch"):
        # right-hand side in, solution out; 13 flops apply the operator once
        return {"bytes": 16.0 * cells, "flops": 13.0 * cells}
    n = case["steps"]
    # u, v, w, p, rho in and out once per step; three sub-steps of about
    # 250 flops per cell (right-hand sides, column solves, projection)
    return {"bytes": 80.0 * n * cells, "flops": 750.0 * n * cells}


# ------------------------------------------------- solves in plain torch
def _exact_solution(case, rhs):
    """A p = f in 64 bits: Fourier in x and y, a tridiagonal system in z."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case.get("method") == "literal":
        edges = -HALF + 2.0 * HALF / nz * np.arange(nz + 1)
    else:
        s = -1.0 + 2.0 * np.arange(nz + 1) / nz
        edges = HALF * np.tanh(2.0 * s) / math.tanh(2.0)
    dz = np.diff(edges)
    dc = np.diff(0.5 * (edges[1:] + edges[:-1]))
    lo, up = np.zeros(nz), np.zeros(nz)
    lo[1:] = 1.0 / (dz[1:] * dc)
    up[:-1] = 1.0 / (dz[:-1] * dc)
    lx = (2.0 * torch.cos(2 * math.pi * torch.arange(nx // 2 + 1, device="cuda", dtype=torch.float64) / nx) - 2.0)
    ly = (2.0 * torch.cos(2 * math.pi * torch.arange(ny, device="cuda", dtype=torch.float64) / ny) - 2.0)
    lam = lx[None, :] / (LX / nx) ** 2 + ly[:, None] / (LY / ny) ** 2
    f = torch.fft.rfft2(rhs[1:-1, 1:-1, 1:-1])
    cp = torch.empty(nz, *lam.shape, dtype=torch.float64, device="cuda")
    prev = None
    for k in range(nz):
        b = lam - (lo[k] + up[k])
        d = f[k]
        if k == nz - 1:
            # the constant mode is singular: its last row pins the constant
            b[0, 0] += 1.0
        if k:
            b = b - lo[k] * cp[k - 1]
            d = d - lo[k] * prev
        cp[k] = up[k] / b
        f[k] = prev = d / b
    for k in range(nz - 2, -1, -1):
        f[k] -= cp[k] * f[k + 1]
    p = torch.fft.irfft2(f, s=(ny, nx))
    return p - p.mean()


def exact(case, seed):
    if case["kind"] not in ("solve", "batch"):
        return None
    g = _grid(case)
    if case["kind"] == "solve":
        return _exact_solution(case, _rhs(case, g, seed))
    return [_exact_solution(case, _rhs(case, g, 1000 * seed + b)) for b in range(case["members"])]
