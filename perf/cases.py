"""Timed cases: what users of the library run, through its public entry points.

Every case is one call (or one short loop of calls) that the examples, the benchmark or the
gradient drivers make: the explicit diffusion example's loop through `Launcher`, a run of
explicit diffusion steps, PT iterations and solves of viscoelastic Stokes in 2D and 3D (FP64, FP32
and FP32 inside FP64 defect correction, with and without the thermal coupling), implicit PT
diffusion, and the shallow-ice time loop with the gradient of an ensemble.

`listed()` are the timed cases, `draw(rng)` another one of the same ranges. `prepare` makes device
fields and inputs from a seed, `run` is the user's call, `exact` the same result in plain FP64
torch, and `work` the bytes and operations of one pass: an explicit step or a PT iteration reads its
inputs once and writes its results once.
"""

from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "chmy.jl_gb300"))

from chmy_gb300 import (  # noqa: E402
    Arch,
    Field,
    FunctionField,
    GB300Backend,
    Launcher,
    Neumann,
    UniformGrid,
    VectorField,
    _abi,
    batch,
    compute_q,
    stokes_fields,
    stokes_params,
    update_C,
)
from chmy_gb300.adjoint import SIAEnsemble  # noqa: E402
from chmy_gb300.bcs import Dirichlet, to_cg_bc  # noqa: E402
from chmy_gb300.configs import StokesProblem  # noqa: E402
from chmy_gb300.functions import ball  # noqa: E402
from chmy_gb300.grids import Center, Vertex  # noqa: E402
from chmy_gb300.solvers import StokesSolver  # noqa: E402

DEV = "cuda"
C, V = Center(), Vertex()


def listed():
    return [
        # the explicit diffusion example as its user writes it: two launches a step, 126^2
        {"name": "diffusion_launcher_126", "kind": "diffusion_launcher", "nx": 126, "ny": 126, "steps": 4},
        # the same loop as one call, an ordinary 2D size with odd rows
        {"name": "diffusion_run_1023", "kind": "diffusion_run", "nx": 1023, "ny": 769, "steps": 50, "f32": False},
        # the VE Stokes example itself: scalar viscosity, buoyant ball, thermal coupling, FP64
        {"name": "stokes2d_thermal_254", "kind": "stokes2d_thermal", "nx": 254, "ny": 254, "iters": 60},
        # a chunk of FP64 PT iterations between two convergence checks, 2D with inclusions
        {"name": "stokes2d_f64_511", "kind": "stokes2d_f64", "nx": 511, "ny": 511, "iters": 64},
        # a whole 2D solve to 1e-8, FP32 inside FP64 defect correction
        {"name": "stokes2d_solve_191", "kind": "stokes2d_solve", "nx": 191, "ny": 191},
        # the FP32 ping-pong iterations of a large 2D model
        {"name": "stokes2d_pp_f32_2047", "kind": "stokes_pp", "nx": 2047, "ny": 1535, "nz": 0, "iters": 20},
        # FP64 PT iterations in 3D, ragged sizes
        {"name": "stokes3d_f64_95", "kind": "stokes3d_f64", "nx": 95, "ny": 80, "nz": 112, "iters": 16},
        # the FP32 ping-pong iterations of a 3D model
        {"name": "stokes3d_pp_f32_192", "kind": "stokes_pp", "nx": 192, "ny": 160, "nz": 176, "iters": 10},
        # one implicit step of 3D variable diffusion, a fixed number of FP64 PT iterations
        {"name": "ptdiff3d_f64_191", "kind": "ptdiff_run", "nx": 191, "ny": 160, "nz": 128, "iters": 24, "f32": False},
        # one implicit step of 3D variable diffusion solved to 1e-10, FP32 inside FP64 refinement
        {"name": "ptdiff3d_solve_128", "kind": "ptdiff_solve", "nx": 128, "ny": 128, "nz": 128},
        # the shallow-ice time loop of one glacier
        {"name": "sia_run_383", "kind": "sia_run", "nx": 383, "ny": 255, "steps": 60},
        # forward and reverse sweep of a small ensemble of uneven glaciers
        {"name": "sia_gradient_10", "kind": "sia_gradient", "members": 10, "nmin": 64, "nmax": 224, "steps": 24},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["diffusion_launcher", "diffusion_run", "stokes2d_thermal", "stokes2d_f64", "stokes2d_solve", "stokes_pp",
                       "stokes3d_f64", "ptdiff_run", "ptdiff_solve", "sia_run", "sia_gradient"])
    c = {"kind": kind}
    if kind == "diffusion_launcher":
        c.update(nx=size(40, 400), ny=size(40, 400), steps=rng.randint(2, 6))
    elif kind == "diffusion_run":
        c.update(nx=size(64, 1600), ny=size(64, 1600), steps=rng.randint(20, 60), f32=rng.random() < 0.3)
    elif kind == "stokes2d_thermal":
        c.update(nx=size(62, 700), ny=size(62, 700), iters=rng.randint(20, 60))
    elif kind == "stokes2d_f64":
        c.update(nx=size(64, 1100), ny=size(64, 1100), iters=rng.randint(16, 64))
    elif kind == "stokes2d_solve":
        c.update(nx=size(64, 240), ny=size(64, 240))
    elif kind == "stokes_pp":
        if rng.random() < 0.5:
            c.update(nx=size(128, 2500), ny=size(128, 2500), nz=0, iters=2 * rng.randint(5, 12))
        else:
            c.update(nx=size(40, 200), ny=size(40, 200), nz=size(40, 200), iters=2 * rng.randint(3, 6))
    elif kind == "stokes3d_f64":
        c.update(nx=size(32, 130), ny=size(32, 130), nz=size(32, 130), iters=rng.randint(8, 20))
    elif kind == "ptdiff_run":
        c.update(nx=size(40, 220), ny=size(40, 220), nz=size(40, 220), iters=rng.randint(12, 30), f32=rng.random() < 0.3)
    elif kind == "ptdiff_solve":
        c.update(nx=size(48, 140), ny=size(48, 140), nz=size(48, 140))
    elif kind == "sia_run":
        c.update(nx=size(64, 600), ny=size(64, 600), steps=rng.randint(20, 60))
    else:
        lo = size(32, 96)
        c.update(members=rng.randint(3, 12), nmin=lo, nmax=lo + size(16, 128), steps=rng.randint(10, 28))
    return c


# ---- inputs (padded arrays [z, y, x], logical index I at I + 1) ------------------------------


def _dims(c):
    return (c["nx"], c["ny"], c["nz"]) if c.get("nz") else (c["nx"], c["ny"])


def _ext(n, loc):
    """Padded extents, x first, of a field whose dimension d is at Vertex where loc[d] is 1."""
    return tuple(m + v + 4 for m, v in zip(n, loc))


def _zeros(n, loc, dtype=torch.float64):
    return torch.zeros(tuple(reversed(_ext(n, loc))), dtype=dtype, device=DEV)


def _coords(n, loc, org, length):
    """Coordinate of every padded point, as arrays that broadcast to the padded [z, y, x] shape."""
    nd, out = len(n), []
    for d in range(nd):
        h = length / n[d]
        x = org + (torch.arange(-1, n[d] + loc[d] + 3, dtype=torch.float64, device=DEV) - (1.0 if loc[d] else 0.5)) * h
        shape = [1] * nd
        shape[nd - 1 - d] = x.numel()
        out.append(x.reshape(shape))
    return out


def _smooth(xs, gen, modes=12, kmax=4.0):
    """A smooth random field of zero mean and about unit variance: a sum of random plane waves."""
    r = torch.rand((modes, len(xs) + 1), generator=gen, device=DEV, dtype=torch.float64).tolist()
    out = 0.0
    for row in r:
        phase = 2.0 * math.pi * row[-1]
        for x, k in zip(xs, row):
            phase = phase + 2.0 * math.pi * kmax * (2.0 * k - 1.0) * x
        out = out + torch.sin(phase)
    return out * math.sqrt(2.0 / modes)


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _face(nd, d):
    return tuple(int(e == d) for e in range(nd))


_EDGES = {2: [(0, 1)], 3: [(0, 1), (0, 2), (1, 2)]}


def _tau_locs(nd):
    return [(0,) * nd] * nd + [tuple(int(e in ab) for e in range(nd)) for ab in _EDGES[nd]]


def _loc(bits):
    return tuple(V if b else C for b in bits)


def _pt_params(n, G=1.0, dt=1e-2, re_pi=4.0):
    """The examples' PT parameters (examples/stokes_2d_inc_ve_T.jl:86-93) on the unit box."""
    dx, nd = 1.0 / max(n), len(n)
    lt, r, vdt = 1.0 / (re_pi * math.pi), 0.5, dx / math.sqrt(nd * 1.1)
    th = lt * (r + 4.0 / 3.0) / vdt
    return {"G": G, "dt": dt, "dtau_Pr": r / th, "dtau_r": 1.0 / (th + 1.0), "nu_dtau": vdt * lt}


def _stokes_inputs(case, seed):
    """VE Stokes on [-0.5, 0.5]^N. 2D: 8 viscous inclusions under pure shear. 3D: a smooth random
    log-viscosity, a buoyant ball and free slip. tau_old holds the previous step's stress."""
    n, g, T = _dims(case), _gen(seed), torch.float32 if case["kind"] == "stokes_pp" else torch.float64
    nd = len(n)
    x = _coords(n, (0,) * nd, -0.5, 1.0)
    if nd == 2:
        eta = torch.ones(tuple(reversed(_ext(n, (0, 0)))), dtype=torch.float64, device=DEV)
        for cx, cy, r, le in torch.rand((8, 4), generator=g, device=DEV, dtype=torch.float64).tolist():
            r = 0.02 + 0.06 * r
            eta[(x[0] - cx + 0.5) ** 2 + (x[1] - cy + 0.5) ** 2 < r * r] = 10.0 ** (4.0 * le - 2.0)
    else:
        eta = torch.exp(_smooth(x, g))
    s = {"eta": eta, "P": _zeros(n, (0,) * nd), "V": [], "rho": [None] * nd}
    for d in range(nd):
        v = _zeros(n, _face(nd, d))
        if nd == 2:
            v += (-1.0 if d == 0 else 1.0) * _coords(n, _face(nd, d), -0.5, 1.0)[d]
        s["V"].append(v)
    s["tau"] = [_zeros(n, l) for l in _tau_locs(nd)]
    s["tau_old"] = [0.1 * _smooth(_coords(n, l, -0.5, 1.0), g) + _zeros(n, l) for l in _tau_locs(nd)]
    if nd == 3:
        z = _coords(n, (0, 0, 1), -0.5, 1.0)
        s["rho"][2] = torch.where(z[0] ** 2 + z[1] ** 2 + z[2] ** 2 < 0.01, 1.0, 0.0).to(torch.float64) + _zeros(n, (0, 0, 1))
    for k, v in s.items():
        s[k] = [None if a is None else a.to(T) for a in v] if isinstance(v, list) else v.to(T)
    s["inv_eta"] = 1.0 / s["eta"]
    # (kind, left value, right value) per component and dimension
    if nd == 2:
        bc = [[("D", 0.5, -0.5), ("N", 0.0, 0.0)], [("N", 0.0, 0.0), ("D", -0.5, 0.5)]]
    else:
        bc = [[("D" if e == d else "N", 0.0, 0.0) for e in range(3)] for d in range(3)]
    return n, s, _pt_params(n), bc


def _thermal_inputs(case, seed):
    n, g = _dims(case), _gen(seed)
    lam, dx = 1e-4, 1.0 / max(n)
    p = _pt_params(n, dt=dx * dx / lam / 4.2)
    u = torch.rand(4, generator=g, device=DEV, dtype=torch.float64).tolist()
    p.update(eta=1.0, eta_ve=1.0 / (1.0 + 1.0 / p["dt"]), lam=lam, ball=(0.2 * u[0] - 0.1, 0.2 * u[1] - 0.1, 0.1 + 0.1 * u[2], 1.0, 0.0))
    x = _coords(n, (0, 0), -0.5, 1.0)
    s = {"P": _zeros(n, (0, 0)), "V": [0.05 * _smooth(_coords(n, _face(2, d), -0.5, 1.0), g) + _zeros(n, _face(2, d)) for d in range(2)]}
    s["tau"] = [_zeros(n, l) for l in _tau_locs(2)]
    s["tau_old"] = [0.1 * _smooth(_coords(n, l, -0.5, 1.0), g) + _zeros(n, l) for l in _tau_locs(2)]
    s["T"] = torch.exp(-((x[0] - 0.1 * u[3]) ** 2 + x[1] ** 2) / 0.02)
    s["T_old"] = s["T"] + 0.01 * _smooth(x, g)
    return n, s, p, [[("D", 0.0, 0.0), ("N", 0.0, 0.0)], [("N", 0.0, 0.0), ("D", 0.0, 0.0)]]


def _ptdiff_inputs(case, seed):
    n, g, T = _dims(case), _gen(seed), torch.float32 if case.get("f32") else torch.float64
    x = _coords(n, (0, 0, 0), -0.5, 1.0)
    D = torch.exp(0.5 * _smooth(x, g, kmax=6.0))
    C0 = torch.exp(-(x[0] ** 2 + x[1] ** 2 + x[2] ** 2) / 0.01) * (1.0 + 0.1 * _smooth(x, g))
    bc = [("D", 0.0, 0.0), ("N", 0.0, 0.0), ("N", 0.0, 0.0)]
    _bc(C0, n, (0, 0, 0), bc)
    dt, Dmax, dx = 1e-3, float(D.max()), 1.0 / max(n)
    vdt = dx / math.sqrt(3 * 1.1)
    re = math.pi + math.sqrt(math.pi**2 + 1.0 / (Dmax * dt))
    p = {"dt": dt, "omega_q": 1.0 / (1.0 + 1.0 / (re * vdt)), "dtau_C": 1.0 / (re * Dmax / vdt + 1.0 / dt)}
    return n, C0.to(T), D.to(T), p, bc


def _sia_inputs(n, seed, steps=0):
    """A bed of smooth hills on [-1, 1]^2, a glacier on it, linear mass balance."""
    g = _gen(seed)
    x = _coords(n, (0, 0), -1.0, 2.0)
    B = 0.4 + 0.2 * _smooth(x, g, kmax=1.5)
    H = torch.relu(0.25 - 0.4 * (x[0] ** 2 + x[1] ** 2) + 0.05 * _smooth(x, g, kmax=1.0))
    _bc(H, n, (0, 0), [("N", 0.0, 0.0)] * 2)
    ela = 0.3 + 0.4 * torch.rand(1, generator=g, device=DEV, dtype=torch.float64).item()
    return B, H, {"Gamma": 1.0, "ela": ela, "beta": 0.5, "m_max": 0.25, "dt_max": 0.5, "cfl": 4.1}


def _member_sizes(case):
    r = np.random.default_rng(case["members"] + case["nmin"])
    return [tuple(int(v) for v in r.integers(case["nmin"], case["nmax"] + 1, 2)) for _ in range(case["members"])]


# ---- the user's side -------------------------------------------------------------------------

_ARCH = []


def _arch():
    if not _ARCH:
        _ARCH.append(Arch(GB300Backend(), device_id=1))
    return _ARCH[0]


def _grid(n, T=np.float64, org=-0.5, length=1.0):
    return UniformGrid(origin=(T(org),) * len(n), extent=(T(length),) * len(n), dims=n, dtype=T)


def _np(t):
    return np.float32 if t.dtype == torch.float32 else np.float64


def _field(grid, bits, t=None, T=None):
    f = Field(_arch(), grid, _loc(bits), T or _np(t))
    if t is not None:
        f.data.copy_(t)
    return f


def _cg_bc(nd, spec):
    make = {"D": Dirichlet, "N": Neumann}
    return to_cg_bc(nd, {"xyz"[d]: (make[k](l), make[k](r)) for d, (k, l, r) in enumerate(spec)})


def _stokes_device(n, s, T):
    """Fields of a VE Stokes state and their descriptor."""
    grid, nd = _grid(n, T), len(n)
    f = {"V": [_field(grid, _face(nd, d), s["V"][d]) for d in range(nd)], "r_V": [_field(grid, _face(nd, d), T=T) for d in range(nd)],
         "P": _field(grid, (0,) * nd, s["P"]), "divV": _field(grid, (0,) * nd, T=T)}
    for k in ("tau", "tau_old"):
        f[k] = [_field(grid, l, a) for l, a in zip(_tau_locs(nd), s[k])]
    for k in ("eta", "inv_eta", "T", "T_old"):
        if k in s:
            f[k] = _field(grid, (0,) * nd, s[k])
    if "rho" in s and any(a is not None for a in s["rho"]):
        f["rho_g"] = [None if a is None else _field(grid, _face(nd, d), a) for d, a in enumerate(s["rho"])]
    return grid, f


def prepare(case, seed):
    kind, arch = case["kind"], _arch()
    if kind == "diffusion_launcher":
        n = _dims(case)
        grid = _grid(n, org=-1.0, length=2.0)
        Cf, q = Field(arch, grid, C), VectorField(arch, grid)
        Cf.data.copy_(_diffusion_C0(case, seed))
        return {"case": case, "launch": Launcher(arch, grid), "grid": grid, "C": Cf, "q": q, "dt": min(grid.spacing()) ** 2 / 2 / 2.1}
    if kind == "diffusion_run":
        T = np.float32 if case["f32"] else np.float64
        grid = _grid(_dims(case), T, -1.0, 2.0)
        A, B = Field(arch, grid, C), Field(arch, grid, C)
        A.data.copy_(_diffusion_C0(case, seed))
        B.data.copy_(A.data)
        return {"case": case, "grid": grid, "A": A, "B": B, "bc": to_cg_bc(2, Neumann()), "dt": float(min(grid.spacing())) ** 2 / 2 / 2.1}
    if kind == "stokes2d_thermal":
        n, s, p, bc = _thermal_inputs(case, seed)
        grid, f = _stokes_device(n, s, np.float64)
        par = stokes_params(p["eta"], p["eta_ve"], p["G"], p["dt"], p["dtau_Pr"], p["dtau_r"], p["nu_dtau"], p["lam"])
        par.rho_g_fn[1] = FunctionField(ball, grid, (C, V), parameters=p["ball"]).desc()
        return {"case": case, "grid": grid, "f": f, "desc": stokes_fields(**f), "par": par,
                "bc": (_abi.cg_bc * 3)(*[_cg_bc(2, b) for b in bc]), "bc_T": to_cg_bc(2, Neumann())}
    if kind in ("stokes2d_f64", "stokes2d_solve", "stokes3d_f64"):
        n, s, p, bc = _stokes_inputs(case, seed)
        nd, h = len(n), {}
        for k in ("V", "tau", "tau_old"):
            h[k] = [a.cpu().numpy() for a in s[k]]
        h["eta"], h["P"] = s["eta"].cpu().numpy(), s["P"].cpu().numpy()
        h["r_V"], h["divV"] = [np.zeros_like(a) for a in h["V"]], np.zeros_like(h["P"])
        if nd == 3:
            h["rho_g"] = [None, None, s["rho"][2].cpu().numpy()]
        par = stokes_params(1.0, 1.0, p["G"], p["dt"], p["dtau_Pr"], p["dtau_r"], p["nu_dtau"])
        pb = StokesProblem(grid=_grid(n), host=h, params=par, bc_V=[_cg_bc(nd, b) for b in bc], ncheck=max(n) // 4, max_iter=200 * max(n))
        solver = StokesSolver(arch, pb)
        start = {k: [f.data.clone() for f in solver.fields[k]] for k in ("V", "tau")}
        start["P"] = solver.fields["P"].data.clone()
        return {"case": case, "solver": solver, "start": start}
    if kind == "stokes_pp":
        n, s, p, bc = _stokes_inputs(case, seed)
        grid, f = _stokes_device(n, s, np.float32)
        other = {k: [_field(grid, l, a) for l, a in zip(ls, s[k])] for k, ls in
                 (("V", [_face(len(n), d) for d in range(len(n))]), ("tau", _tau_locs(len(n))))}
        other["P"] = _field(grid, (0,) * len(n), s["P"])
        del f["eta"]
        par = stokes_params(1.0, 1.0, p["G"], p["dt"], p["dtau_Pr"], p["dtau_r"], p["nu_dtau"])
        return {"case": case, "grid": grid, "f": f, "other": other, "a": stokes_fields(**f), "b": stokes_fields(**other), "par": par,
                "bc": (_abi.cg_bc * 3)(*[_cg_bc(len(n), b) for b in bc])}
    if kind in ("ptdiff_run", "ptdiff_solve"):
        n, C0, D, p, bc = _ptdiff_inputs(case, seed)
        T = _np(C0)
        grid = _grid(n, T)
        f = {"C": _field(grid, (0, 0, 0), C0), "C_old": _field(grid, (0, 0, 0), C0), "D": _field(grid, (0, 0, 0), D),
             "q": [_field(grid, _face(3, d), T=T) for d in range(3)]}
        s = _abi.cg_ptdiff_fields()
        s.C, s.C_old, s.D = f["C"].desc(), f["C_old"].desc(), f["D"].desc()
        s.q = (_abi.cg_field * 3)(*[q.desc() for q in f["q"]])
        par = _abi.cg_ptdiff_params()
        par.dt, par.omega_q, par.dtau_C = p["dt"], p["omega_q"], p["dtau_C"]
        return {"case": case, "grid": grid, "f": f, "desc": s, "par": par, "bc": _cg_bc(3, bc), "C0": C0}
    if kind == "sia_run":
        n = _dims(case)
        B, H, p = _sia_inputs(n, seed)
        grid = _grid(n, org=-1.0, length=2.0)
        q = [_field(grid, _face(2, d), T=np.float64) for d in range(2)]
        return {"case": case, "grid": grid, "H": _field(grid, (0, 0), H), "B": _field(grid, (0, 0), B), "q": q,
                "qd": (_abi.cg_field * 3)(q[0].desc(), q[1].desc(), _abi.cg_field()), "par": _sia_params(p)}
    members, H0, obs = [], [], []
    for k, n in enumerate(_member_sizes(case)):
        B, H, p = _sia_inputs(n, seed * 1000 + k)
        members.append((_grid(n, org=-1.0, length=2.0), B.cpu().numpy(), _sia_params(p)))
        H0.append(H.cpu().numpy())
        obs.append(0.9 * H0[-1])
    return {"case": case, "sia": SIAEnsemble(arch, members), "H0": H0, "obs": obs}


def _sia_params(p):
    o = _abi.cg_sia_params()
    o.Gamma, o.As, o.n, o.beta, o.ela, o.m_max, o.dt_max, o.cfl = p["Gamma"], 0.0, 3, p["beta"], p["ela"], p["m_max"], p["dt_max"], p["cfl"]
    return o


def _diffusion_C0(case, seed):
    n, g = _dims(case), _gen(seed)
    x = _coords(n, (0, 0), -1.0, 2.0)
    C0 = torch.exp(-(x[0] ** 2 + x[1] ** 2) / 0.1) + 0.1 * _smooth(x, g)
    _bc(C0, n, (0, 0), [("N", 0.0, 0.0)] * 2)
    return C0.to(torch.float32) if case.get("f32") else C0


def run(state):
    case, arch = state["case"], _arch()
    kind = case["kind"]
    if kind == "diffusion_launcher":
        grid, Cf, q, launch = state["grid"], state["C"], state["q"], state["launch"]
        for _ in range(case["steps"]):
            launch(arch, grid, (compute_q, (q, Cf, 1.0, grid)))
            launch(arch, grid, (update_C, (Cf, q, state["dt"], grid)), bc=batch(grid, (Cf, Neumann())))
        return [Cf.data, q.x.data, q.y.data]
    if kind == "diffusion_run":
        A, B = state["A"], state["B"]
        arch.call("cg_diffusion_run", ctypes.byref(state["grid"].desc()), ctypes.byref(A.desc()), ctypes.byref(B.desc()), 1.0, state["dt"],
                  ctypes.byref(state["bc"]), case["steps"])
        return [A.data, B.data]
    if kind == "stokes2d_thermal":
        arch.call("cg_stokes_pt_iterations_thermal", ctypes.byref(state["grid"].desc()), ctypes.byref(state["desc"]),
                  ctypes.byref(state["par"]), state["bc"], ctypes.byref(state["bc_T"]), case["iters"])
        return _stokes_out(state["f"]) + [state["f"]["T"].data]
    if kind in ("stokes2d_f64", "stokes3d_f64"):
        solver = state["solver"]
        solver.iterate(case["iters"])
        err = solver.residual()
        return _stokes_out(solver.fields) + [np.array(err)]
    if kind == "stokes2d_solve":
        solver, start = state["solver"], state["start"]
        for k in ("V", "tau"):
            for f, a in zip(solver.fields[k], start[k]):
                f.data.copy_(a)
        solver.fields["P"].data.copy_(start["P"])
        solver.solve(precision=_abi.CG_F32)
        return [f.data for f in solver.fields["V"] + solver.fields["tau"]] + [solver.fields["P"].data]
    if kind == "stokes_pp":
        arch.call("cg_stokes_pt_iterations_pp", ctypes.byref(state["grid"].desc()), ctypes.byref(state["a"]), ctypes.byref(state["b"]),
                  ctypes.byref(state["par"]), state["bc"], case["iters"])
        return _stokes_out(state["f"])
    if kind == "ptdiff_run":
        arch.call("cg_ptdiff_run", ctypes.byref(state["grid"].desc()), ctypes.byref(state["desc"]), ctypes.byref(state["par"]),
                  ctypes.byref(state["bc"]), 1, case["iters"])
        f = state["f"]
        return [f["C"].data, f["C_old"].data] + [q.data for q in f["q"]]
    if kind == "ptdiff_solve":
        f = state["f"]
        f["C"].data.copy_(state["C0"])
        f["C_old"].data.copy_(state["C0"])
        o, res = _abi.cg_solve_opts(), _abi.cg_solve_result()
        o.max_iter, o.ncheck, o.eps, o.precision, o.max_outer, o.inner_rtol = 20000, 50, 1e-10, _abi.CG_F32, 20, 1e-3
        arch.call("cg_ptdiff_solve", ctypes.byref(state["grid"].desc()), ctypes.byref(state["desc"]), ctypes.byref(state["par"]),
                  ctypes.byref(state["bc"]), ctypes.byref(o), ctypes.byref(res))
        return [f["C"].data]
    if kind == "sia_run":
        t = ctypes.c_double()
        arch.call("cg_sia_run", ctypes.byref(state["grid"].desc()), ctypes.byref(state["H"].desc()), ctypes.byref(state["B"].desc()),
                  state["qd"], ctypes.byref(state["par"]), case["steps"], ctypes.byref(t))
        return [state["H"].data, state["q"][0].data, state["q"][1].data, t.value]
    obs = state["obs"]
    dG, de, gH, HN = state["sia"].gradient(state["H0"], case["steps"], lambda m, H: H - obs[m])
    return [np.array(dG), np.array(de), [g[2:-2, 2:-2] for g in gH], HN]


def _stokes_out(f):
    return [a.data for a in f["V"] + f["tau"] + f["r_V"]] + [f["P"].data, f["divV"].data]


# ---- the same in plain FP64 torch ------------------------------------------------------------


def _at(f, n, off=None):
    """The values at I + off over the launch range [0, n+1]^N."""
    nd = len(n)
    off = off or (0,) * nd
    return f[tuple(slice(1 + off[d], n[d] + 3 + off[d]) for d in reversed(range(nd)))]


def _unit(nd, d, s=1):
    return tuple(s * int(e == d) for e in range(nd))


def _bc(f, n, loc, spec):
    """Dirichlet and Neumann planes of one field, last dimension first, over tangential 0..n+2."""
    nd = len(n)
    for d in reversed(range(nd)):
        kind, left, right = spec[d]
        ext = n[d] + loc[d]

        def plane(i):
            return tuple(i + 1 if e == d else slice(1, n[e] + 4) for e in reversed(range(nd)))

        for side, v in enumerate((left, right)):
            if kind is None:
                continue
            if kind == "D" and loc[d]:
                f[plane(1 if side == 0 else ext)] = v
            else:
                src = f[plane(1 if side == 0 else ext)]
                f[plane(0 if side == 0 else ext + 1)] = 2.0 * v - src if kind == "D" else src
    return f


def _d(f, n, d, idx, fwd):
    """Difference along d over the launch range: f[I+1] - f[I] (fwd) or f[I] - f[I-1]."""
    nd = len(n)
    if fwd:
        return (_at(f, n, _unit(nd, d)) - _at(f, n)) * idx[d]
    return (_at(f, n) - _at(f, n, _unit(nd, d, -1))) * idx[d]


def _exact_stokes(n, s, p, bc, iters=None, tol=None, thermal=False):
    nd, idx = len(n), [float(m) for m in n]
    f64 = lambda a: None if a is None else a.double().clone()  # noqa: E731
    s = {k: [f64(a) for a in v] if isinstance(v, list) else f64(v) for k, v in s.items()}
    Vel, tau, to, P = s["V"], s["tau"], s["tau_old"], s["P"]
    rV, divV = [torch.zeros_like(v) for v in Vel], torch.zeros_like(P)
    g = 1.0 / (p["G"] * p["dt"])
    edges = _EDGES[nd]
    if thermal:
        x = _coords(n, (0, 1), -0.5, 1.0)
        cx, cy, r, vin, vout = p["ball"]
        rho = [None, torch.where((x[0] - cx) ** 2 + (x[1] - cy) ** 2 < r * r, vin, vout).double() + _zeros(n, (0, 1))]
        ieta_c, eve_c = 1.0 / p["eta"], p["eta_ve"]
        ieta_e, eve_e = [ieta_c], [eve_c]
        step = [p["nu_dtau"] / p["eta_ve"]] * 2
    else:
        rho, ie = s["rho"], s["inv_eta"]
        ieta_c = _at(ie, n)
        eve_c = 1.0 / (ieta_c + g)
        ieta_e = []
        for a, b in edges:
            ua, ub = _unit(nd, a, -1), _unit(nd, b, -1)
            uab = tuple(i + j for i, j in zip(ua, ub))
            ieta_e.append(0.25 * (ieta_c + _at(ie, n, ua) + _at(ie, n, ub) + _at(ie, n, uab)))
        eve_e = [1.0 / (v + g) for v in ieta_e]
        step = [p["nu_dtau"] * (torch.minimum(ieta_c, _at(ie, n, _unit(nd, d, -1))) + g) for d in range(nd)]
    it = 0
    while True:
        e = [_d(Vel[d], n, d, idx, True) for d in range(nd)]
        dv = sum(e[1:], e[0])
        _at(divV, n).copy_(dv)
        _at(P, n).sub_(dv * eve_c * p["dtau_Pr"])
        for c in range(nd):
            t = _at(tau[c], n)
            t.add_((-(t - _at(to[c], n)) * g - t * ieta_c + 2.0 * (e[c] - dv / 3.0)) * eve_c * p["dtau_r"])
        for k, (a, b) in enumerate(edges):
            t = _at(tau[nd + k], n)
            eod = 0.5 * (_d(Vel[a], n, b, idx, False) + _d(Vel[b], n, a, idx, False))
            t.add_((-(t - _at(to[nd + k], n)) * g - t * ieta_e[k] + 2.0 * eod) * eve_e[k] * p["dtau_r"])
        for d in range(nd):
            r = _d(tau[d], n, d, idx, False) - _d(P, n, d, idx, False)
            for k, (a, b) in enumerate(edges):
                if d in (a, b):
                    r = r + _d(tau[nd + k], n, b if d == a else a, idx, True)
            if rho[d] is not None:
                r = r - _at(rho[d], n)
            _at(rV[d], n).copy_(r)
        for d in range(nd):
            _at(Vel[d], n).add_(_at(rV[d], n) * step[d])
            _bc(Vel[d], n, _face(nd, d), bc[d])
        if thermal:
            T, dq = s["T"], 0.0
            for d in range(2):
                q, v, l = torch.zeros_like(Vel[d]), _at(Vel[d], n), _at(T, n, _unit(2, d, -1))
                _at(q, n).copy_(-p["lam"] * _d(T, n, d, idx, False) + torch.relu(v) * l - torch.relu(-v) * _at(T, n))
                dq = dq + _d(q, n, d, idx, True)
            Tn = T.clone()
            _at(Tn, n).copy_(_at(s["T_old"], n) - p["dt"] * dq)
            s["T"] = _bc(Tn, n, (0, 0), [("N", 0.0, 0.0)] * 2)
        it += 1
        if iters is not None and it == iters:
            break
        if tol is not None and it % 500 == 0:
            inner = lambda a, l: a[tuple(slice(2 + l[d], n[d] + 2) for d in reversed(range(nd)))]  # noqa: E731
            worst = [float(inner(divV, (0,) * nd).abs().max())] + [float(inner(r, _face(nd, d)).abs().max()) for d, r in enumerate(rV)]
            if max(worst) < tol or it >= 60000:
                break
    return Vel, tau, rV, P, divV, s.get("T"), step


def _sia_steps(S_B, H, p, idx, steps, Gamma, ela):
    """Steps of the shallow-ice loop on H over cells [0, n+1]^2 (Neumann ghosts); gradients flow."""
    t, qx, qy = 0.0, None, None
    dx2 = (1.0 / max(idx)) ** 2
    pad = lambda a: torch.nn.functional.pad(a[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]  # noqa: E731
    for _ in range(steps):
        Hp = pad(H)
        S = S_B + Hp
        gx, gy = (S[:, 1:] - S[:, :-1]) * idx[0], (S[1:, :] - S[:-1, :]) * idx[1]
        ax, ay = 0.5 * (gx[1:-1, 1:] + gx[1:-1, :-1]), 0.5 * (gy[1:, 1:-1] + gy[:-1, 1:-1])
        D = Gamma * H**5 * (ax * ax + ay * ay)
        flat = D.reshape(-1)
        top = flat[torch.argmax(flat)]
        dt = dx2 / top / p["cfl"] if float(top) > 0 else torch.as_tensor(p["dt_max"], dtype=torch.float64, device=DEV)
        dt = dt if float(dt) < p["dt_max"] else torch.as_tensor(p["dt_max"], dtype=torch.float64, device=DEV)
        qx = torch.nn.functional.pad(-0.5 * (D[:, 1:] + D[:, :-1]) * gx[1:-1, 1:-1], (1, 1, 0, 0))
        qy = torch.nn.functional.pad(-0.5 * (D[1:, :] + D[:-1, :]) * gy[1:-1, 1:-1], (0, 0, 1, 1))
        x = p["beta"] * (S[1:-1, 1:-1] - ela)
        m = torch.where(x < p["m_max"], x, torch.full_like(x, p["m_max"]))
        W = m - (qx[:, 1:] - qx[:, :-1]) * idx[0] - (qy[1:, :] - qy[:-1, :]) * idx[1]
        H = torch.relu(H + dt * W)
        t = t + float(dt)
    return H, qx, qy, t


def _sia_padded(H0, H, n):
    out = H0.clone()
    out[2:-2, 2:-2] = H
    return _bc(out, n, (0, 0), [("N", 0.0, 0.0)] * 2)


def exact(case, seed):
    kind = case["kind"]
    n = _dims(case) if "nx" in case else None
    if kind in ("diffusion_launcher", "diffusion_run"):
        C0 = _diffusion_C0(case, seed).double()
        idx = [m / 2.0 for m in n]
        dt = (2.0 / max(n)) ** 2 / 2 / 2.1
        A, B = C0, C0.clone()
        q = [_zeros(n, _face(2, d)) for d in range(2)]
        for _ in range(case["steps"]):
            for d in range(2):
                _at(q[d], n).copy_(-_d(A, n, d, idx, False))
            _at(B, n).copy_(_at(A, n) - dt * (_d(q[0], n, 0, idx, True) + _d(q[1], n, 1, idx, True)))
            _bc(B, n, (0, 0), [("N", 0.0, 0.0)] * 2)
            A, B = B, A
        if kind == "diffusion_launcher":
            return [A] + q
        return [B, A] if case["steps"] % 2 else [A, B]
    if kind == "stokes2d_thermal":
        n, s, p, bc = _thermal_inputs(case, seed)
        Vel, tau, rV, P, divV, T, _ = _exact_stokes(n, s, p, bc, iters=case["iters"], thermal=True)
        return Vel + tau + rV + [P, divV, T]
    if kind in ("stokes2d_f64", "stokes3d_f64", "stokes_pp"):
        n, s, p, bc = _stokes_inputs(case, seed)
        Vel, tau, rV, P, divV, _, _ = _exact_stokes(n, s, p, bc, iters=case["iters"])
        if kind == "stokes_pp":
            return Vel + tau + rV + [P, divV]
        nd = len(n)
        for d in range(nd):
            _bc(rV[d], n, _face(nd, d), [("D" if e == d else None, 0.0, 0.0) for e in range(nd)])
        mid = lambda f, l: f[tuple(slice(2, n[d] + l[d] + 2) for d in reversed(range(nd)))]  # noqa: E731
        err = [float(mid(divV, (0,) * nd).abs().max())] + [float(mid(r, _face(nd, d)).abs().max()) for d, r in enumerate(rV)]
        return Vel + tau + rV + [P, divV] + [np.array(err)]
    if kind == "stokes2d_solve":
        # the pressure is defined up to a constant, and the state at the stopping test only to it
        if n[0] * n[1] > 200 * 200:
            return None
        n, s, p, bc = _stokes_inputs(case, seed)
        Vel, tau, _, _, _, _, _ = _exact_stokes(n, s, p, bc, tol=1e-9)
        return Vel + tau + [None]
    if kind in ("ptdiff_run", "ptdiff_solve"):
        n, C0, D, p, bc = _ptdiff_inputs(case, seed)
        idx, D, Co = [float(m) for m in n], D.double(), C0.double()
        Df = [0.5 * (_at(D, n) + _at(D, n, _unit(3, d, -1))) for d in range(3)]
        c, q = Co.clone(), [_zeros(n, _face(3, d)) for d in range(3)]
        if kind == "ptdiff_run":
            for _ in range(case["iters"]):
                for d in range(3):
                    qd = _at(q[d], n)
                    qd.add_((-(Df[d] * _d(c, n, d, idx, False)) - qd) * p["omega_q"])
                dv = _d(q[0], n, 0, idx, True) + _d(q[1], n, 1, idx, True) + _d(q[2], n, 2, idx, True)
                cc = _at(c, n)
                cc.add_((-(cc - _at(Co, n)) / p["dt"] - dv) * p["dtau_C"])
                _bc(c, n, (0, 0, 0), bc)
            return [c, Co] + q
        inner = (slice(2, -2),) * 3

        def apply(u):  # u - dt divg(D grad u) on the interior cells
            w = torch.zeros_like(c)
            w[inner] = u
            _bc(w, n, (0, 0, 0), bc)
            for d in range(3):
                _at(q[d], n).copy_(-Df[d] * _d(w, n, d, idx, False))
            dv = _d(q[0], n, 0, idx, True) + _d(q[1], n, 1, idx, True) + _d(q[2], n, 2, idx, True)
            return u + p["dt"] * dv[(slice(1, -1),) * 3]

        b = Co[inner].clone()
        u = b.clone()
        r = b - apply(u)
        d, rr = r.clone(), float((r * r).sum())
        for _ in range(4000):
            if rr < 1e-26 * float((b * b).sum()):
                break
            Ad = apply(d)
            a = rr / float((d * Ad).sum())
            u, r = u + a * d, r - a * Ad
            new = float((r * r).sum())
            d, rr = r + (new / rr) * d, new
        c[inner] = u
        return [_bc(c, n, (0, 0, 0), bc)]
    if kind == "sia_run":
        B, H0, p = _sia_inputs(n, seed)
        H, qx, qy, t = _sia_steps(B[1:-1, 1:-1], H0[2:-2, 2:-2], p, [m / 2.0 for m in n], case["steps"], p["Gamma"], p["ela"])
        q = [_zeros(n, (1, 0)), _zeros(n, (0, 1))]
        q[0][2:-2, 2:-2], q[1][2:-2, 2:-2] = qx, qy
        return [_sia_padded(H0, H, n)] + q + [t]
    dG, de, gH, HN = [], [], [], []
    for k, n in enumerate(_member_sizes(case)):
        B, H0, p = _sia_inputs(n, seed * 1000 + k)
        v = [torch.tensor(x, dtype=torch.float64, device=DEV, requires_grad=True) for x in (p["Gamma"], p["ela"])]
        h = H0[2:-2, 2:-2].clone().requires_grad_(True)
        H, _, _, _ = _sia_steps(B[1:-1, 1:-1], h, p, [m / 2.0 for m in n], case["steps"], *v)
        grads = torch.autograd.grad(0.5 * ((H - 0.9 * H0[2:-2, 2:-2]) ** 2).sum(), v + [h])
        dG.append(float(grads[0]))
        de.append(float(grads[1]))
        gH.append(grads[2].cpu().numpy())
        HN.append(_sia_padded(H0, H.detach(), n).cpu().numpy())
    return [np.array(dG), np.array(de), gH, HN]


# ---- bytes and operations of one pass --------------------------------------------------------


def work(case):
    """Arrays read and written once per step or iteration, and the operations of the update.
    Solves count one pass over their inputs and results for each FP64 cycle and 19 FP32 arrays
    (2D Stokes) or 10 (3D diffusion) per inner iteration, at the iteration counts of these sizes:
    about 30 per point of the longer side (Stokes) and 3 (diffusion)."""
    kind = case["kind"]
    if kind == "sia_gradient":
        cells = case["members"] * ((case["nmin"] + case["nmax"]) / 2.0) ** 2
        return {"bytes": cells * case["steps"] * (3 + 2 * 9 + 2) * 8.0, "flops": cells * case["steps"] * 160.0}
    cells = float(math.prod(_dims(case)))
    b = 4.0 if case.get("f32") or kind in ("stokes_pp", "stokes2d_solve", "ptdiff_solve") else 8.0
    arrays, flops, reps = {
        "diffusion_launcher": (2, 13, case.get("steps")),
        "diffusion_run": (2, 13, case.get("steps")),
        "stokes2d_thermal": (18, 85, case.get("iters")),
        "stokes2d_f64": (18, 65, case.get("iters")),
        "stokes2d_solve": (19, 65, 30 * max(_dims(case))),
        "stokes3d_f64": (28, 130, case.get("iters")),
        "stokes_pp": (28 if case.get("nz") else 18, 130 if case.get("nz") else 65, case.get("iters")),
        "ptdiff_run": (10, 40, case.get("iters")),
        "ptdiff_solve": (10, 40, 3 * max(_dims(case))),
        "sia_run": (3, 57, case.get("steps")),
    }[kind]
    return {"bytes": cells * arrays * b * reps, "flops": cells * flops * reps}
