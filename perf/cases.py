"""Performance cases of the framework: whole calls of its public entry points.

Every case is one segment of a run as a user's program makes it: the
primitive state goes in from pinned host arrays, a number of CFL time steps
run on the GPU, the primitive state comes back.  The entry points are
``Simulation.set_prim / advance / get_prim`` (one problem, FP64 or FP32-mixed),
``Simulation.step_host`` (a host code that owns the state and asks for one
step at a time) and the ``fvgpu_batch_*`` calls (many problems together).

FP64 outputs are returned as the FP64 arrays the call fills.  The FP32-mixed
form computes its fluxes in FP32; its snapshots go on as float32 to an
analysis on the GPU (spectra, rendering), which is what the case returns.

``exact`` is a plain torch FP64 restatement of the scheme (2-cell ghost
fill, minmod PLM or PCM states, HLL / HLLC, gravity, constant conduction,
the reference's viscous terms, Euler or RK2, the CFL time step), literal 3-D
formulas in which a shift along a one-cell axis reads the cell itself.
"""
import ctypes
import math

import numpy as np
import torch

import fv3d_gb300 as fv
from fv3d_gb300 import _abi

_BC = {"absorbing": _abi.FV_BC_ABSORBING, "reflecting": _abi.FV_BC_REFLECTING, "periodic": _abi.FV_BC_PERIODIC}

# Per problem: boundaries (x, y, z), solver, reconstruction, stepping, CFL,
# gamma, g, kappa, mu -- the settings of the repository's own configurations.
_PROBLEMS = {
    "sod": dict(bc=("reflecting", "reflecting", "periodic"), solver="hllc", gamma=1.4),
    "sedov": dict(bc=("absorbing", "absorbing", "periodic"), solver="hllc", gamma=1.4),
    "rayleigh_taylor": dict(bc=("periodic", "periodic", "reflecting"), solver="hll", gamma=1.4, g=-0.1),
    "rayleigh_taylor_tc_visc": dict(bc=("periodic", "periodic", "reflecting"), solver="hll", gamma=1.4, g=-0.1,
                                    kappa=1e-4, mu=1e-4),
    "thermal_pulse": dict(bc=("periodic",) * 3, solver="hllc", gamma=1.4, kappa=0.01, mu=0.005),
    "shear_layer": dict(bc=("periodic",) * 3, solver="hllc", gamma=5.0 / 3.0, kappa=1e-4, mu=1e-4),
    "blast": dict(bc=("periodic",) * 3, solver="hllc", gamma=1.4, recon="pcm", stepping="euler", cfl=0.1),
    "flow_3d": dict(bc=("periodic",) * 3, solver="hllc", gamma=5.0 / 3.0, kappa=1e-3, mu=1e-3),
}


def listed():
    return [
        # a host code that keeps its own state and asks for one step: the smallest call, all latency
        dict(name="fp64 step_host sod 96x64", call="step_host", precision="fp64", problem="sod", nx=96, ny=64, nz=1,
             steps=1),
        # the point blast of the plain FP64 configuration, between two snapshots
        dict(name="fp64 sedov 256^2", call="advance", precision="fp64", problem="sedov", nx=256, ny=256, nz=1,
             steps=32),
        # the benchmark workload: Rayleigh-Taylor with gravity in the x-z plane
        dict(name="fp64 rt 512x1536", call="advance", precision="fp64", problem="rayleigh_taylor", nx=512, ny=1,
             nz=1536, steps=16),
        # conduction and viscosity on an odd, ragged 2-D grid
        dict(name="fp64 pulse 1001x713", call="advance", precision="fp64", problem="thermal_pulse", nx=1001, ny=713,
             nz=1, steps=8),
        # the reference's own 3-D example: blast, PCM, Euler steps
        dict(name="fp64 blast 64^3", call="advance", precision="fp64", problem="blast", nx=64, ny=64, nz=64,
             steps=48),
        # a ragged 3-D flow with every physical term, RK2
        dict(name="fp64 flow 101x83x61", call="advance", precision="fp64", problem="flow_3d", nx=101, ny=83, nz=61,
             steps=8),
        # many small FP64 problems together: Sod tubes and blasts of uneven sizes
        dict(name="fp64 batch 48 sod sedov", call="batch", precision="fp64", problem="sod_sedov", n=48, lo=64, hi=256,
             steps=16),
        # FP32-mixed: a small grid, bound by the latency of its steps
        dict(name="mixed sedov 256^2", call="advance", precision="mixed", problem="sedov", nx=256, ny=256, nz=1,
             steps=200),
        # FP32-mixed: the mid-size gravity run
        dict(name="mixed rt 512x1536", call="advance", precision="mixed", problem="rayleigh_taylor", nx=512, ny=1,
             nz=1536, steps=64),
        # FP32-mixed: the largest grid, shear layer with conduction and viscosity
        dict(name="mixed shear 4096^2", call="advance", precision="mixed", problem="shear_layer", nx=4096, ny=4096,
             nz=1, steps=100),
        # FP32-mixed 3-D with every physical term
        dict(name="mixed flow 192^3", call="advance", precision="mixed", problem="flow_3d", nx=192, ny=192, nz=192,
             steps=24),
        # many uneven problems advanced together in the FP32-mixed form
        dict(name="mixed batch 64 sod sedov", call="batch", precision="mixed", problem="sod_sedov", n=64, lo=64,
             hi=256, steps=200),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    precision = rng.choice(["fp64", "mixed"])
    call = rng.choice(["step_host", "advance", "advance", "advance3d", "batch"])
    if call == "step_host":
        problem = rng.choice(["sod", "sedov"])
        return dict(call=call, precision=precision, problem=problem, nx=_spread(rng, 40, 700),
                    ny=_spread(rng, 40, 700), nz=1, steps=1)
    if call == "advance":
        problem = rng.choice(["sod", "sedov", "rayleigh_taylor", "rayleigh_taylor_tc_visc", "thermal_pulse",
                              "shear_layer"])
        a, b = _spread(rng, 64, 1100), _spread(rng, 64, 1100)
        steps = max(8, min(64, (1 << 24) // (a * b))) if precision == "mixed" else max(8, min(32, (1 << 22) // (a * b)))
        if problem.startswith("rayleigh"):
            return dict(call=call, precision=precision, problem=problem, nx=a, ny=1, nz=b, steps=steps)
        return dict(call=call, precision=precision, problem=problem, nx=a, ny=b, nz=1, steps=steps)
    if call == "advance3d":
        problem = rng.choice(["blast", "flow_3d"])
        a, b, c = (_spread(rng, 24, 120) for _ in range(3))
        return dict(call="advance", precision=precision, problem=problem, nx=a, ny=b, nz=c,
                    steps=24 if precision == "mixed" else 8)
    return dict(call="batch", precision=precision, problem="sod_sedov", n=_spread(rng, 4, 48), lo=rng.randrange(40, 80),
                hi=rng.randrange(120, 260), steps=rng.choice([16, 32]))


# ---- settings and initial states -------------------------------------------

def _settings(problem, nx, ny, nz):
    s = dict(recon="plm", stepping="rk2", cfl=0.8, g=0.0, kappa=0.0, mu=0.0)
    s.update(_PROBLEMS[problem])
    s.update(problem=problem, n=(nx, ny, nz), lo=(0.0, 0.0, 0.0), hi=(1.0, 1.0, 1.0))
    if problem.startswith("rayleigh"):
        s["hi"] = (0.5, 1.0, 1.5)
    s["d"] = tuple((h - l) / k for h, l, k in zip(s["hi"], s["lo"], s["n"]))
    return s


def _problems(case):
    """The settings of each problem of the case."""
    if case["call"] != "batch":
        return [_settings(case["problem"], case["nx"], case["ny"], case["nz"])]
    out = []
    for i in range(case["n"]):
        # five sides between lo and hi, Sod tubes and blasts alternating, gamma spread over 1.1 .. 1.67
        side = case["lo"] + (case["hi"] - case["lo"]) * ((i // 2 * 7) % 5) // 4
        s = _settings("sod" if i % 2 == 0 else "sedov", side, side, 1)
        s["gamma"] = 1.1 + 0.57 * ((i * 0.6180339887498949) % 1.0)
        out.append(s)
    return out


def _params(s, precision):
    p = fv.parse_ini("")
    p.Nx, p.Ny, p.Nz = s["n"]
    (p.xmin, p.ymin, p.zmin), (p.xmax, p.ymax, p.zmax), (p.dx, p.dy, p.dz) = s["lo"], s["hi"], s["d"]
    p.boundary_x, p.boundary_y, p.boundary_z = (_BC[b] for b in s["bc"])
    p.riemann_solver = _abi.FV_HLL if s["solver"] == "hll" else _abi.FV_HLLC
    p.reconstruction = _abi.FV_PLM if s["recon"] == "plm" else _abi.FV_PCM
    p.time_stepping = _abi.FV_TS_RK2 if s["stepping"] == "rk2" else _abi.FV_TS_EULER
    p.CFL, p.gamma0, p.tend = s["cfl"], s["gamma"], 1.0e30
    p.gravity, p.g = int(s["g"] != 0.0), s["g"]
    p.thermal_conductivity_active, p.kappa = int(s["kappa"] != 0.0), s["kappa"]
    p.viscosity_active, p.mu = int(s["mu"] != 0.0), s["mu"]
    p.precision = _abi.FV_PREC_FP64 if precision == "fp64" else _abi.FV_PREC_FP32_MIXED
    return p


def _state(s, seed):
    """The initial primitives (rho, u, v, w, p) on the GPU, each (Nz, Ny, Nx); None for a field that is zero."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    nx, ny, nz = s["n"]
    ax = [torch.arange(k, device="cuda", dtype=torch.float64).add_(0.5).mul_(d).add_(l)
          for k, d, l in zip(s["n"], s["d"], s["lo"])]
    X, Y, Z = ax[0].view(1, 1, nx), ax[1].view(1, ny, 1), ax[2].view(nz, 1, 1)
    one = torch.ones((nz, ny, nx), device="cuda", dtype=torch.float64)

    def noise():
        return torch.rand((nz, ny, nx), device="cuda", dtype=torch.float64, generator=gen).mul_(2).sub_(1)

    def shift():  # the same flow at another place
        return float(torch.rand((), device="cuda", generator=gen)) - 0.5

    name = s["problem"]
    if name == "sod":
        left = (X + 0.0 * Y <= 0.5 + 0.1 * shift()).expand(nz, ny, nx)
        rho = torch.where(left, 1.0 * one, 0.125 * one) * (1 + 1e-3 * noise())
        u, v = (0.1 * torch.sin(math.pi * x).expand(nz, ny, nx) for x in (X, Y))
        return [rho, u, v, None, torch.where(left, 1.0 * one, 0.1 * one)]
    if name == "sedov":
        r = torch.sqrt((X - 0.5 - 0.1 * shift()) ** 2 + (Y - 0.5 - 0.1 * shift()) ** 2).expand(nz, ny, nx)
        hot = (s["gamma"] - 1.0) / (math.pi * 0.02 ** 2)
        return [one * (1 + 1e-2 * noise()), None, None, None, torch.where(r < 0.02, hot * one, 1e-5 * one)]
    if name.startswith("rayleigh"):
        rho = torch.where((Z > 0.75).expand(nz, ny, nx), 2.0 * one, one)
        p = 2.5 + s["g"] * rho * (Z - 0.75)
        # the usual perturbation, grown to a tenth, in layers that drift sideways
        w = 0.1 * (1 + torch.cos(4 * math.pi * (X - 0.5 * shift()))) * (1 + torch.cos(2 * math.pi * Z)) / 4
        v = 0.1 * one if s["mu"] else None
        return [rho, 0.3 * one + 1e-3 * noise(), v, w.expand(nz, ny, nx) + 1e-4 * noise(), p]
    if name == "thermal_pulse":
        r2 = (X - 0.5 - 0.2 * shift()) ** 2 + (Y - 0.5 - 0.2 * shift()) ** 2
        T = (1.0 + torch.exp(-r2 / (2 * 0.05 ** 2))).expand(nz, ny, nx)
        # carried along by a uniform flow
        return [one, 0.4 * one + 1e-3 * noise(), 0.3 * one, 0.1 * one, T * (1 + 1e-4 * noise())]
    if name == "shear_layer":
        inner = ((Y - 0.5).abs() < 0.25).expand(nz, ny, nx)
        v = 1e-2 * torch.sin(4 * math.pi * (X - 0.2 * shift())) + 1e-3 * noise()
        w = 0.1 * torch.cos(2 * math.pi * Y).expand(nz, ny, nx)
        return [torch.where(inner, 2 * one, one), torch.where(inner, 0.5 * one, -0.5 * one), 0.1 * one + v, w, 2.5 * one]
    if name == "blast":
        r = torch.sqrt((X - 0.5 - 0.1 * shift()) ** 2 + (Y - 0.5) ** 2 + (Z - 0.5) ** 2)
        inside = r < 0.2
        rho = torch.where(inside, one, 1.2 * one) * (1 + 1e-3 * noise())
        return [rho, None, None, None, torch.where(inside, 10.0 * one, 0.1 * one)]
    out = []  # flow_3d: a few long waves per field and small noise, subsonic and supersonic regions
    for base, amp in ((1.25, 0.5), (0.0, 0.8), (0.0, 0.8), (0.0, 0.8), (1.25, 0.5)):
        f = sum(torch.sin(2 * math.pi * ((1 + k % 2) * X + (1 + k // 2) * Y + (2 - k % 2) * Z + shift()))
                for k in range(3)) / 3
        out.append(base + amp * f + 1e-2 * noise())
    return out


def _pinned(t):
    if t is None:
        return None
    h = torch.empty(t.shape, dtype=torch.float64, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _ptrs(fields):
    dp = ctypes.POINTER(ctypes.c_double)
    return [None if f is None else f.ctypes.data_as(dp) for f in fields]


def prepare(case, seed):
    probs = _problems(case)
    params = [_params(s, case["precision"]) for s in probs]
    ins, outs = [], []
    for i, s in enumerate(probs):
        nx, ny, nz = s["n"]
        ins.append([_pinned(f) for f in _state(s, 1000003 * int(seed) + i)])
        outs.append([torch.empty((nz, ny, nx), dtype=torch.float64, pin_memory=True).numpy() for _ in range(5)])
    if case["call"] == "step_host":  # its arrays are all given
        zero = torch.zeros(outs[0][0].shape, dtype=torch.float64)
        ins[0] = [_pinned(zero) if f is None and k in (1, 2) else f for k, f in enumerate(ins[0])]
    solver = fv.Batch(params) if case["call"] == "batch" else fv.Simulation(params[0])
    return dict(case=case, solver=solver, ins=ins, outs=outs)


def _result(st, extra):
    outs = [torch.from_numpy(f) for fields in st["outs"] for f in fields]
    if st["case"]["call"] == "batch":  # one array per field over all problems
        outs = [torch.cat([torch.from_numpy(fields[v]).reshape(-1) for fields in st["outs"]]) for v in range(5)]
    if st["case"]["precision"] != "fp64":
        outs = [t.to("cuda").float() for t in outs]
    return {"prim": outs, "time": extra}


def run(st):
    case, solver = st["case"], st["solver"]
    if case["call"] == "step_host":
        _, dt = solver.step_host(st["ins"][0], 0.0, st["outs"][0])
        return _result(st, dt)
    if case["call"] == "advance":
        solver.set_prim(*st["ins"][0])
        t, _ = solver.advance(1.0e30, max_steps=case["steps"])
        solver.get_prim(st["outs"][0])
        return _result(st, t)
    t0 = solver.times()  # a batch's clocks go on from pass to pass
    for i, f in enumerate(st["ins"]):
        solver.set_prim(i, *f)
    solver.run(case["steps"])
    t1 = solver.times()
    for i, f in enumerate(st["outs"]):
        solver._check(solver.lib.fvgpu_batch_get_prim(solver._h, i, *_ptrs(f)), "batch_get_prim")
    return _result(st, (t1 - t0).astype(np.float32))


def work(case):
    """Bytes: the host state in and out, and per step the state read and
    written once (8 bytes per value).  Operations: per face two states of
    slopes and a Riemann solve, per cell conversions, update and sources."""
    total_b = total_f = 0.0
    for s in _problems(case):
        cells = float(np.prod(s["n"]))
        dims = sum(k > 1 for k in s["n"])
        fields = 5 if dims == 3 or s["mu"] else 4
        stages = 2 if s["stepping"] == "rk2" else 1
        face = (8 * fields if s["recon"] == "plm" else 0) + 90
        cell = 25 + 6 * fields * dims + (10 * dims if s["kappa"] else 0) + (60 * dims if s["mu"] else 0)
        total_b += cells * (10 * 8 + case["steps"] * 2 * fields * 8)
        total_f += cells * case["steps"] * (stages * (dims * face + cell) + 25)
    return {"bytes": total_b, "flops": total_f}


# ---- the scheme in plain torch, FP64 ---------------------------------------

def _minmod(a, b):
    return torch.where(a * b < 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _pad(q, s):
    """Two ghost layers along every axis of more than one cell (X, then Y, then Z)."""
    for a in range(3):
        n, bc = s["n"][a], s["bc"][a]
        if n == 1:
            continue
        i = torch.arange(-2, n + 2, device=q[0].device)
        ghost = (i < 0) | (i >= n)
        if bc == "periodic":
            i = i % n
        elif bc == "reflecting":
            i = torch.where(i < 0, -i - 1, torch.where(i >= n, 2 * n - 1 - i, i))
        else:
            i = i.clamp(0, n - 1)
        q = [f.index_select(3 - a, i) for f in q]
        if bc == "reflecting":
            sign = torch.where(ghost, -1.0, 1.0).to(torch.float64)
            q[1 + a] = q[1 + a] * sign.view([-1 if k == 3 - a else 1 for k in range(4)])
    return q


def _win(f, s, off, extra=None):
    """The interior window of a padded field shifted by `off` (x, y, z); one more cell along axis `extra`."""
    for a in range(3):
        if s["n"][a] > 1:
            f = f.narrow(3 - a, 2 + off[a], s["n"][a] + (1 if extra == a else 0))
    return f


def _euler_flux(r, un, t1, t2, p, gm1):
    E = p / gm1 + 0.5 * r * (un * un + t1 * t1 + t2 * t2)
    m = r * un
    return [r, m, r * t1, r * t2, E], [m, m * un + p, m * t1, m * t2, (p + E) * un]


def _hll(L, R, gamma):
    gm1 = gamma - 1
    aL, aR = torch.sqrt(gamma * L[4] / L[0]), torch.sqrt(gamma * R[4] / R[0])
    SL = torch.minimum(L[1] - aL, R[1] - aR).clamp(max=0.0)  # a zero speed gives the one-sided flux
    SR = torch.maximum(L[1] + aL, R[1] + aR).clamp(min=0.0)
    UL, FL = _euler_flux(*L, gm1)
    UR, FR = _euler_flux(*R, gm1)
    return [(SR * fl - SL * fr + SL * SR * (ur - ul)) / (SR - SL) for ul, fl, ur, fr in zip(UL, FL, UR, FR)]


def _hllc(L, R, gamma):
    (rL, uL, aL, bL, pL), (rR, uR, aR, bR, pR) = L, R
    gm1 = gamma - 1
    EL = 0.5 * rL * (uL * uL + aL * aL) + pL / gm1  # two velocities, as the reference
    ER = 0.5 * rR * (uR * uR + aR * aR) + pR / gm1
    c = torch.sqrt(torch.maximum(gamma * pL / rL, gamma * pR / rR))
    SL, SR = torch.minimum(uL, uR) - c, torch.maximum(uL, uR) + c
    kL, kR = rL * (uL - SL), rR * (SR - uR)
    uS = (kR * uR + kL * uL + (pL - pR)) / (kR + kL)
    pS = (kR * pL + kL * pR + kL * kR * (uL - uR)) / (kR + kL)
    left = uS > 0
    r, u, p, E = (torch.where(left, x, y) for x, y in ((rL, rR), (uL, uR), (pL, pR), (EL, ER)))
    t1, t2 = torch.where(left, aL, aR), torch.where(left, bL, bR)
    S = torch.where(left, SL, SR)
    outside = (SL > 0) | (~left & (SR <= 0))
    sr = torch.where(outside, r, r * (S - u) / (S - uS))
    sE = torch.where(outside, E, ((S - u) * E - p * u + pS * uS) / (S - uS))
    su, sp = torch.where(outside, u, uS), torch.where(outside, p, pS)
    m = sr * su
    return [m, m * su + sp, m * t1, m * t2, (sE + sp) * su]


# velocity fields (normal, first, second transverse) of the sweeps along x, y, z
_SWEEP = ((1, 2, 3), (2, 1, 3), (3, 2, 1))


def _faces(Q, s, a, gamma):
    """The fluxes (rho, m_x, m_y, m_z, E) of the n + 1 faces along axis a."""
    cells = []
    for k in range(4):
        off = [0, 0, 0]
        off[a] = k - 2
        cells.append([_win(f, s, off, extra=a) for f in Q])
    if s["recon"] == "plm":
        L, R = [], []
        for q0, q1, q2, q3 in zip(*cells):
            d = q2 - q1
            L.append(q1 + 0.5 * _minmod(q1 - q0, d))
            R.append(q2 - 0.5 * _minmod(d, q3 - q2))
    else:
        L, R = cells[1], cells[2]
    un, t1, t2 = _SWEEP[a]
    f = (_hll if s["solver"] == "hll" else _hllc)([L[0], L[un], L[t1], L[t2], L[4]],
                                                 [R[0], R[un], R[t1], R[t2], R[4]], gamma)
    out = [f[0], None, None, None, f[4]]
    out[un], out[t1], out[t2] = f[1], f[2], f[3]
    return out


def _viscous(Q, s):
    """The viscous increments (u, v, w, E) per unit time: flux differences without 1/d and
    with the reference's mixed-up indices in the z branch."""
    ox, oy, oz = (1.0 / d for d in s["d"])
    mu = s["mu"]
    U, V, W = 1, 2, 3

    def P(k, j, i, var):
        return _win(Q[var], s, (i - 1, j - 1, k - 1))

    acc = [0.0, 0.0, 0.0, 0.0]

    def add(sign, tx, ty, tz, qu, qv, qw):
        for c, t in enumerate((tx, ty, tz, tx * qu + ty * qv + tz * qw)):
            acc[c] = acc[c] + sign * mu * t

    for e in (1, 2):
        sign = -1.0 if e == 1 else 1.0
        q = [0.5 * (P(1, 1, e, c) + P(1, 1, e - 1, c)) for c in (U, V, W)]
        dx = [ox * (P(1, 1, e, c) - P(1, 1, e - 1, c)) for c in (U, V, W)]
        dy = [oy / 4 * (P(1, 2, e, c) - P(1, 0, e, c) + P(1, 2, e - 1, c) - P(1, 0, e - 1, c)) for c in (U, V)]
        dz = [oz / 4 * (P(2, 1, e, c) - P(0, 1, e, c) + P(2, 1, e - 1, c) - P(0, 1, e - 1, c)) for c in (U, W)]
        add(sign, 4 / 3 * dx[0] - 2 / 3 * (dy[1] + dz[1]), dx[1] + dy[0], dx[2] + dz[0], *q)
        q = [0.5 * (P(1, e, 1, c) + P(1, e - 1, 1, c)) for c in (U, V, W)]
        dy = [oy * (P(1, e, 1, c) - P(1, e - 1, 1, c)) for c in (U, V, W)]
        dx = [ox / 4 * (P(1, e, 2, c) - P(1, e, 0, c) + P(1, e - 1, 2, c) - P(1, e - 1, 0, c)) for c in (U, V)]
        dz = [oz / 4 * (P(2, e, 1, c) - P(0, e, 1, c) + P(2, e - 1, 1, c) - P(0, e - 1, 1, c)) for c in (V, W)]
        add(sign, dx[1] + dy[0], 4 / 3 * dy[1] - 2 / 3 * (dx[0] + dz[1]), dz[0] + dy[2], *q)
        q = [0.5 * (P(e, 1, 1, c) + P(e - 1, 1, 1, c)) for c in (U, V, W)]
        dz = [oz * (P(e, 1, 1, c) - P(e - 1, 1, 1, c)) for c in (U, V, W)]
        dudx = ox / 4 * (P(e, 1, 2, U) - P(1, e, 0, U) + P(e - 1, 1, 2, U) - P(1, e - 1, 0, U))
        dwdx = ox / 4 * (P(e, 1, 2, V) - P(1, e, 0, W) + P(e - 1, 1, 2, V) - P(1, e - 1, 0, W))
        dvdy = oz / 4 * (P(e, 2, 1, W) - P(e, 0, 1, V) + P(e - 1, 2, 1, W) - P(e - 1, 0, 1, V))
        dwdy = oz / 4 * (P(e, 2, 1, V) - P(e, 0, 1, W) + P(e - 1, 2, 1, V) - P(e - 1, 0, 1, W))
        add(sign, dz[0] + dwdx, dz[1] + dwdy, 4 / 3 * dz[2] - 2 / 3 * (dudx + dvdy), *q)
    return acc


def _to_prim(C, gamma):
    r = C[0]
    u, v, w = (m / r for m in C[1:4])
    return [r, u, v, w, (C[4] - 0.5 * r * (u * u + v * v + w * w)) * (gamma - 1)]


def _to_cons(q, gamma):
    r, u, v, w, p = q
    return [r, r * u, r * v, r * w, p / (gamma - 1) + 0.5 * r * (u * u + v * v + w * w)]


def _stage(C, s, dt, gamma):
    Q = _pad(_to_prim(C, gamma), s)
    C = list(C)
    for a in range(3):
        n = s["n"][a]
        if n == 1:
            continue
        F = _faces(Q, s, a, gamma)
        for v in range(5):
            C[v] = C[v] + (F[v].narrow(3 - a, 0, n) - F[v].narrow(3 - a, 1, n)) * dt / s["d"][a]
        if a == 2 and s["g"]:
            C[3] = C[3] + dt * s["g"] * _win(Q[0], s, (0, 0, 0))
            C[4] = C[4] + 0.5 * dt * s["g"] * (F[0].narrow(1, 0, n) + F[0].narrow(1, 1, n))
    C[0] = C[0].clamp(min=1e-6)
    if s["kappa"]:
        T = Q[4] / Q[0]
        c = _win(T, s, (0, 0, 0))
        for a in range(3):
            if s["n"][a] > 1:
                off = [0, 0, 0]
                off[a] = 1
                up, dn = _win(T, s, off), _win(T, s, [-o for o in off])
                C[4] = C[4] + dt * s["kappa"] / s["d"][a] ** 2 * (up - 2 * c + dn)
    if s["mu"]:
        for v, x in enumerate(_viscous(Q, s)):
            C[1 + v] = C[1 + v] + x * dt
    return C


def _advance(q, s, steps, gamma):
    """`steps` CFL steps of a stack of problems (leading axis); the primitives and the time of each."""
    C = _to_cons(q, gamma)
    t = 0.0
    fixed = 0.0
    for c in (s["kappa"], s["mu"]):
        fixed = max(fixed, 2 * c / min(s["d"]) ** 2)
    for _ in range(steps):
        r, u, v, w, p = _to_prim(C, gamma)
        cs = torch.sqrt(gamma * p / r)
        inv = sum((cs + x.abs()) / d for x, d in zip((u, v, w), s["d"]))
        dt = (s["cfl"] / inv.amax(dim=(1, 2, 3), keepdim=True).clamp(min=fixed))
        C1 = _stage(C, s, dt, gamma)
        if s["stepping"] == "rk2":
            C2 = _stage(C1, s, dt, gamma)
            C = [0.5 * (a + b) for a, b in zip(C, C2)]
        else:
            C = C1
        t = t + dt
    return _to_prim(C, gamma), t.view(-1)


def exact(case, seed):
    probs = _problems(case)
    groups = {}
    for i, s in enumerate(probs):
        groups.setdefault((s["problem"], s["n"]), []).append(i)
    prim, time = [None] * len(probs), [None] * len(probs)
    for members in groups.values():
        states = []
        for i in members:
            q = _state(probs[i], 1000003 * int(seed) + i)
            states.append([torch.zeros_like(q[0]) if f is None else f for f in q])
        q = [torch.stack([st[v] for st in states]) for v in range(5)]
        gamma = torch.tensor([probs[i]["gamma"] for i in members], device="cuda", dtype=torch.float64)
        got, t = _advance(q, probs[members[0]], case["steps"], gamma.view(-1, 1, 1, 1))
        for k, i in enumerate(members):
            prim[i], time[i] = [f[k] for f in got], float(t[k])
    if case["call"] == "batch":
        return {"prim": [torch.cat([p[v].reshape(-1) for p in prim]) for v in range(5)], "time": np.array(time)}
    return {"prim": prim[0], "time": time[0]}
