"""The work a user of this framework has it do, as cases that can be timed.

Every case goes through the public entry points (``Solver``, ``Batch``,
``RadialBatch``) with device-resident arrays, as a program that keeps its
fields on the GPU calls them.  Kinds:

  derivatives  the compact derivatives of a field in all three directions,
               with and without accumulation, first and second derivative
  filters      one state through the compact filter and one field pair
               through the Gaussian filter (what every RK stage ends with)
  solvers      the general tridiagonal / pentadiagonal line solvers
  stage        the right-hand-side routines of one RK stage, called one by
               one as lddrk4_nonperiodic_mf.f does
  output       the diagnostics that Output runs after each step
  step         one main-loop step (Compute_CFL, Compute_Tstep, LDDRK4)
  batch        one step of several same-size cases at once (serving)
  radial       steps of many 1-D radial problems of uneven length
"""
import math

import numpy as np
import torch

from shock_turbulence_b200 import Batch, Solver, default_params, periodic_params
from shock_turbulence_b200.initial import radial_blast
from shock_turbulence_b200.radial import RadialBatch

FP32 = 1   # precision: FP32 intermediates, FP64 state


def _grid(nx, ny=None, nz=None):
    return {"nx": nx, "ny": ny or nx, "nz": nz or nx}


def listed():
    return [
        # latency: three first derivatives of the smallest grid in use (the
        # per-call cost of a host program that calls the operators one by one)
        {"name": "derivatives 32^3", "kind": "derivatives", "family": "octant", "second": False, **_grid(32)},
        # the operators of a viscous code on an uneven grid of the octant
        {"name": "derivatives 112x176x208", "kind": "derivatives", "family": "octant", "second": True,
         **_grid(112, 176, 208)},
        # the same on the periodic box of a spectral-like turbulence run
        {"name": "derivatives box 256^3", "kind": "derivatives", "family": "periodic", "second": True, **_grid(256)},
        # end of a stage: the state's compact filter, the sensors' Gaussian
        {"name": "filters 240x192x336", "kind": "filters", "family": "octant", **_grid(240, 192, 336)},
        # line systems with coefficients of their own, bounded and periodic
        {"name": "solvers 384x16384", "kind": "solvers", "n": 384, "lot": 16384},
        # one RK stage through the single routines
        {"name": "stage 144x176x160", "kind": "stage", **_grid(144, 176, 160)},
        # the analyses after each step of a production run
        {"name": "output 192^3", "kind": "output", **_grid(192)},
        # decaying turbulence, the small plain run: 64^3 periodic, FP64
        {"name": "step box 64^3", "kind": "step", "family": "periodic", "precision": 0, **_grid(64)},
        # FP32 mode on a mid-size octant with a material interface
        {"name": "step blast 256^3 fp32", "kind": "step", "family": "octant", "precision": FP32, **_grid(256)},
        # the production run: expanding blast in turbulence, 384^3, FP64
        {"name": "step blast 384^3", "kind": "step", "family": "octant", "precision": 0, **_grid(384)},
        # serving: same-size requests stepped together, FP32 mode
        {"name": "batch 6 x 96^3 fp32", "kind": "batch", "cases": 6, "precision": FP32, **_grid(96)},
        # uneven radial problems, 128 to 4096 points each
        {"name": "radial 512 problems", "kind": "radial", "problems": 512, "nmin": 128, "nmax": 4096, "steps": 4},
    ]


def draw(rng):
    def size(lo, hi, unit=16):
        return unit * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / unit))

    kind = rng.choice(["derivatives", "filters", "solvers", "stage", "output", "step", "batch", "radial"])
    if kind == "solvers":
        # lines times rows bounded by the listed case's four-fold
        n = int(round(math.exp(rng.uniform(math.log(24), math.log(1024)))))
        return {"kind": kind, "n": n, "lot": int(round(math.exp(rng.uniform(math.log(256), math.log(8e6 / n)))))}
    if kind == "radial":
        nmin = int(round(math.exp(rng.uniform(math.log(32), math.log(1024)))))
        nmax = int(round(math.exp(rng.uniform(math.log(nmin + 1), math.log(4096)))))
        return {"kind": kind, "problems": int(round(math.exp(rng.uniform(math.log(8), math.log(1024))))),
                "nmin": nmin, "nmax": nmax, "steps": rng.randint(1, 6)}
    if kind == "batch":
        n = size(32, 128, 32)
        return {"kind": kind, "cases": rng.randint(2, 8), "precision": rng.choice([0, FP32]), **_grid(n)}
    if kind == "step":
        p = rng.choice([0, FP32])
        return {"kind": kind, "family": rng.choice(["octant", "periodic"]), "precision": p,
                **_grid(size(48, 272, 32), size(48, 272, 32), size(48, 272, 32))}
    top = {"derivatives": 448, "filters": 400, "stage": 272, "output": 320}[kind]
    g = _grid(*(size(32, top) for _ in range(3)))
    if kind == "derivatives":
        return {"kind": kind, "family": rng.choice(["octant", "periodic"]), "second": rng.random() < 0.7, **g}
    if kind == "filters":
        return {"kind": kind, "family": rng.choice(["octant", "periodic"]), **g}
    return {"kind": kind, **g}


# ---- inputs -------------------------------------------------------------------
def _gen(seed, device="cuda"):
    return torch.Generator(device=device).manual_seed(int(seed))


def _turbulence(shape, k0, urms, gen):
    """Solenoidal velocity with E(k) ~ k^4 exp(-2 (k/k0)^2), three fields."""
    nx, nz, ny = shape
    dev = "cuda"
    kx = torch.fft.fftfreq(nx, 1.0 / nx, device=dev, dtype=torch.float64)[:, None, None]
    kz = torch.fft.fftfreq(nz, 1.0 / nz, device=dev, dtype=torch.float64)[None, :, None]
    ky = torch.fft.rfftfreq(ny, 1.0 / ny, device=dev, dtype=torch.float64)[None, None, :]
    k2 = kx * kx + kz * kz + ky * ky
    amp = k2 * torch.exp(-k2 / (k0 * k0)) / torch.sqrt(k2.clamp(min=1.0))
    amp[0, 0, 0] = 0.0
    h = [torch.fft.rfftn(torch.randn(shape, dtype=torch.float64, device=dev, generator=gen)) * amp for _ in range(3)]
    dot = (h[0] * kx + h[1] * ky + h[2] * kz) / k2.clamp(min=1.0)
    out = []
    for hq, kq in zip(h, (kx, ky, kz)):
        out.append(torch.fft.irfftn(hq - dot * kq, s=shape))
    rms = torch.sqrt(sum((f * f).mean() for f in out) / 3.0)
    return [f * (urms / rms) for f in out]


def _state(p, seed, blast, interface):
    """Conserved state Q (5, nx, nz, ny) and mass fraction Y: turbulence, with
    a Gaussian energy deposit at the symmetry corner and a spherical material
    interface where asked."""
    shape = (p.nx, p.nz, p.ny)
    g = _gen(seed)
    k0 = min(8.0, min(shape) / 8.0)
    u, v, w = _turbulence(shape, k0, 0.1 / math.sqrt(3.0), g)

    def axis(n, length, view):
        return (torch.arange(n, dtype=torch.float64, device="cuda") * (length / (n - 1))).view(view)

    r2 = axis(p.nx, p.x_leng, (-1, 1, 1)) ** 2 + axis(p.nz, p.z_leng, (1, -1, 1)) ** 2 + \
        axis(p.ny, p.y_leng, (1, 1, -1)) ** 2
    dx = p.x_leng / (p.nx - 1)
    Y = 0.5 - 0.5 * torch.tanh((torch.sqrt(r2) - 2.5) / (6.0 * dx)) if interface else \
        torch.ones(shape, dtype=torch.float64, device="cuda")
    pr = 1.0 / p.gamma1
    P = pr * (1.0 + 19.0 * torch.exp(-r2 / (4.0 * dx) ** 2)) if blast else torch.full_like(r2, pr)
    # a weak density fluctuation on top of the uniform background
    rho = 1.0 + 0.01 * torch.sin(axis(p.nx, 2.0 * math.pi, (-1, 1, 1)) + axis(p.ny, 2.0 * math.pi, (1, 1, -1)))
    if blast or interface:
        rho = torch.ones_like(P)
    g1, g2, eps = p.gamma1, p.gamma2, p.epsilon
    geff = (Y * g1 / (g1 - 1) + eps * (1 - Y) * g2 / (g2 - 1)) / (Y / (g1 - 1) + eps * (1 - Y) / (g2 - 1))
    Q = torch.empty((5,) + shape, dtype=torch.float64, device="cuda")
    Q[0], Q[1], Q[2], Q[3] = rho * u, rho * v, rho * w, rho
    Q[4] = P / (geff - 1.0) + 0.5 * rho * (u * u + v * v + w * w)
    return Q, Y


def _smooth(shape, gen, n):
    """n turbulent-looking scalar fields."""
    return torch.stack([_turbulence(shape, min(8.0, min(shape) / 8.0), 1.0, gen)[0] for _ in range(n)])


def _params(case):
    sizes = (case["nx"], case["ny"], case["nz"])
    if case.get("family") == "periodic":
        return periodic_params(*sizes, re=100.0, precision=case.get("precision", 0))
    return default_params(*sizes, re=100.0, c_beta_scale=1.75, precision=case.get("precision", 0))


def _new(p, *lead):
    return torch.zeros(lead + (p.nx, p.nz, p.ny), dtype=torch.float64, device="cuda")


# ---- prepare --------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "solvers":
        return _prepare_solvers(case, seed)
    if kind == "radial":
        return _prepare_radial(case, seed)
    p = _params(case)
    s = {"case": case, "p": p}
    if kind == "batch":
        n = case["cases"]
        s["batch"] = b = Batch(p, n)
        for k in range(n):
            Q, Y = _state(p, 1000 * seed + k, True, False)
            torch.cuda.synchronize()
            b.start(k, Q, Y)
        s["Q"], s["Y"] = _new(p, n, 5), _new(p, n)
        torch.cuda.synchronize()
        return s
    s["solver"] = sol = Solver(p)
    shape = (p.nx, p.nz, p.ny)
    periodic = case.get("family") == "periodic"
    if kind == "derivatives":
        s["F"] = _smooth(shape, _gen(seed), 3)
        s["d"], s["d2"], s["div"] = _new(p, 3), _new(p, 3), _new(p)
    elif kind == "filters":
        s["Q"] = _smooth(shape, _gen(seed), 7)
        s["Qf"], s["Eg"] = _new(p, 5), _new(p, 2)
    elif kind == "stage":
        s["Q"], s["Y"] = _state(p, seed, True, True)
        s["Qrhs"], s["Yrhs"] = _new(p, 5), _new(p)
        torch.cuda.synchronize()
        sol.Compute_gamma(s["Y"])
    else:
        Q, Y = _state(p, seed, not periodic, not periodic and case.get("precision", 0) == FP32)
        torch.cuda.synchronize()
        sol.set_state(Q, None if periodic else Y)
        if not periodic:
            sol.Compute_gamma(Y)
        if kind == "output":
            sol.step(0.0, 0)
            s["Grad"] = _new(p, 4)
        else:
            sol.RHS(Q, _new(p, 5), None if periodic else Y)   # /GRAD/ of the start, for Compute_hyper
            sol.Compute_hyper(Q, None if periodic else Y)
            s["Q"], s["Y"] = Q, Y
        s["time"], s["step"] = 0.0, 0
    torch.cuda.synchronize()
    return s


def _solver_coefficients(case, seed):
    """Diagonally dominant rows near the compact schemes' own, each line and
    row different: (A, B, C, R) and (A, B, C, D, E, R), layout (n, lot)."""
    n, lot = case["n"], case["lot"]
    g = _gen(seed)

    def rows(mid, spread):
        return mid + spread * (torch.rand((n, lot), dtype=torch.float64, device="cuda", generator=g) - 0.5)

    tri = [rows(1.0 / 3.0, 0.1), rows(1.0, 0.05), rows(1.0 / 3.0, 0.1)]
    pen = [rows(0.05, 0.02), rows(0.3, 0.1), rows(1.0, 0.05), rows(0.3, 0.1), rows(0.05, 0.02)]
    R = [rows(0.0, 2.0) for _ in range(4)]
    return tri, pen, R


def _prepare_solvers(case, seed):
    tri, pen, R = _solver_coefficients(case, seed)
    s = {"case": case, "solver": Solver(default_params(32)), "tri": tri, "pen": pen, "R": R,
         "X": [torch.empty_like(r) for r in R]}
    torch.cuda.synchronize()
    return s


def _prepare_radial(case, seed):
    n = case["problems"]
    lengths = np.random.default_rng(7).integers(case["nmin"], case["nmax"] + 1, size=n).astype(np.int32)
    rng = np.random.default_rng(seed)
    Q = np.concatenate([radial_blast(int(m), 2.0, float(rng.uniform(10.0, 200.0)), rng=rng).ravel() for m in lengths])
    rb = RadialBatch(lengths, np.full(n, 2.0))
    rb.set_state(np.ascontiguousarray(Q))
    s = {"case": case, "rb": rb, "Q": torch.zeros(Q.size, dtype=torch.float64, device="cuda")}
    torch.cuda.synchronize()
    return s


# ---- run ------------------------------------------------------------------------
def run(s):
    return _RUN[s["case"]["kind"]](s)


def _run_derivatives(s):
    sol, F, d, d2, div = s["solver"], s["F"], s["d"], s["d2"], s["div"]
    if s["case"]["family"] == "periodic":
        d1 = grad = (sol.DFDX, sol.DFDY, sol.DFDZ)
        dd = (sol.D2FDX2, sol.D2FDY2, sol.D2FDZ2)
    else:
        # a symmetric scalar's gradient; the velocity's own direction is antisymmetric
        d1 = (sol.DFDX_sym, sol.DFDY_sym, sol.DFDZ_sym)
        grad = (sol.DFDX_asym, sol.DFDY_asym, sol.DFDZ_asym)
        dd = (sol.D2FDX2_sym, sol.D2FDY2_sym, sol.D2FDZ2_sym)
    if not s["case"]["second"]:
        for k in range(3):
            d1[k](F[0], d[k], 0, 1.0)
        return {"d": d}
    for k in range(3):                       # first and second derivative of a scalar
        dd[k](F[0], d[k], d2[k], 1)
    for k in range(3):                       # divergence, accumulated direction by direction
        grad[k](F[k], div, int(k > 0), -1.0)
    return {"d": d, "d2": d2, "div": div}


def _run_filters(s):
    s["solver"].Compact_Filter(s["Q"][:5], s["Qf"], 5)
    s["solver"].Gaussian_Filter(s["Q"][5:], s["Eg"], 2)
    return {"Qf": s["Qf"], "Eg": s["Eg"]}


def _run_solvers(s):
    sol, n, lot = s["solver"], s["case"]["n"], s["case"]["lot"]
    for x, r in zip(s["X"], s["R"]):
        x.copy_(r)                           # the solvers work in place
    torch.cuda.current_stream().synchronize()
    for k, per in enumerate((0, 1)):
        sol.tridiagonal(*s["tri"], s["X"][k], n, lot, per)
    for k, per in enumerate((0, 1)):
        sol.pentadiagonal(*s["pen"], s["X"][2 + k], n, lot, per)
    return s["X"]


def _run_stage(s):
    sol, Q, Y, Qrhs, Yrhs = s["solver"], s["Q"], s["Y"], s["Qrhs"], s["Yrhs"]
    sol.Compute_gamma(Y)
    sol.RHS(Q, Qrhs, Y)
    sol.Hyper_RHS(Q, Qrhs, Y)
    sol.Species_RHS(Q, Qrhs, Y, Yrhs)
    sol.bc_RHS(Q, Qrhs, Y, Yrhs)
    sol.Sponge_Forcing(Q, Qrhs, Y, Yrhs)
    return {"Q": Q, "Qrhs": Qrhs, "Yrhs": Yrhs}


def _run_output(s):
    sol = s["solver"]
    Grad, maxdil, enstrophy = sol.Compute_Grad(s["Grad"])
    hmix, tke, ur, ya = sol.Compute_SRM_Stats()
    rad, skew = sol.Generate_Shock_Surface()
    return {"Grad": Grad, "scalars": [maxdil, enstrophy, hmix, tke, rad, skew], "ur": np.nan_to_num(ur),
            "ya": np.nan_to_num(ya), "monitors": sol.monitors()}


def _run_step(s):
    sol = s["solver"]
    s["time"], s["step"] = sol.step(s["time"], s["step"])
    sol.get_state(s["Q"], s["Y"])
    return {"Q": s["Q"], "Y": s["Y"], "time": s["time"]}


def _run_batch(s):
    b = s["batch"]
    b.step_async()
    times = [b.get(k, s["Q"][k], s["Y"][k])[2] for k in range(s["case"]["cases"])]
    return {"Q": s["Q"], "Y": s["Y"], "times": times}


def _run_radial(s):
    s["rb"].step(s["case"]["steps"])
    s["rb"].get_state(s["Q"])
    return {"Q": s["Q"], "times": s["rb"].get_time()[0]}


_RUN = {"derivatives": _run_derivatives, "filters": _run_filters, "solvers": _run_solvers, "stage": _run_stage,
        "output": _run_output, "step": _run_step, "batch": _run_batch, "radial": _run_radial}


# ---- work -----------------------------------------------------------------------
def work(case):
    """Inputs read once, outputs written once.  A step is 10 (octant) or 11
    (periodic) RK stages; every stage depends on the whole field of the one
    before, so each reads and writes the state and the RK registers once."""
    kind = case["kind"]
    if kind == "solvers":
        N = case["n"] * case["lot"]
        return {"bytes": 8.0 * N * (2 * 5 + 2 * 7), "flops": N * (8.0 + 14.0 + 20.0 + 36.0)}
    if kind == "radial":
        lengths = np.random.default_rng(7).integers(case["nmin"], case["nmax"] + 1, size=case["problems"])
        pts = float(lengths.sum())
        # state and RK register stay on chip over the steps of a problem
        return {"bytes": 8.0 * pts * (3 + 3 + 2), "flops": pts * case["steps"] * 11 * 600.0}
    n3 = float(case["nx"] * case["ny"] * case["nz"])
    if kind == "derivatives":
        if not case["second"]:
            return {"bytes": n3 * 8.0 * 4, "flops": n3 * 3 * 13.0}
        return {"bytes": n3 * 8.0 * (3 + 3 + 3 + 1), "flops": n3 * (3 * 27.0 + 3 * 14.0)}
    if kind == "filters":
        return {"bytes": n3 * 8.0 * 14, "flops": n3 * (15 * 26.0 + 6 * 13.0)}
    if kind == "stage":
        return {"bytes": n3 * 8.0 * (6 + 3 + 6), "flops": n3 * 2200.0}
    if kind == "output":
        return {"bytes": n3 * 8.0 * (6 + 1 + 4), "flops": n3 * 250.0}
    fields, stages = (10, 11) if case.get("family") == "periodic" else (12, 10)
    c = case.get("cases", 1)
    return {"bytes": c * n3 * 8.0 * 2 * fields * stages, "flops": c * n3 * stages * 2500.0}


# ---- exact ----------------------------------------------------------------------
# The line operators as dense matrices (explicit stencil, then the compact
# left-hand side inverted in 64 bits), applied along an axis.
def _stencil(n, rows, symmetric, wrap):
    """Dense matrix of an interior stencil {offset: weight}; outside the low
    end the field continues as an even (+1) or odd (-1) one."""
    M = np.zeros((n, n))
    for i in range(n):
        for o, wgt in rows.items():
            j = i + o
            if wrap:
                M[i, j % n] += wgt
            elif j < 0:
                M[i, -j] += symmetric * wgt
            elif j < n:
                M[i, j] += wgt
    return M


def _set(M, i, entries):
    M[i] = 0.0
    for j, v in entries.items():
        M[i, j] = v


def _band(n, rows, wrap):
    M = np.zeros((n, n))
    for i in range(n):
        for o, wgt in rows.items():
            j = i + o
            if wrap:
                M[i, j % n] += wgt
            elif 0 <= j < n:
                M[i, j] += wgt
    return M


def _d_matrix(n, length, order, odd, wrap):
    sg = -1.0 if odd else 1.0
    if order == 1:
        a, b, al = 14.0 / 18.0, 1.0 / 36.0, 1.0 / 3.0
        B, A = _stencil(n, {1: a, -1: -a, 2: b, -2: -b}, sg, wrap), _band(n, {-1: al, 0: 1.0, 1: al}, wrap)
        if not wrap:
            if odd:
                _set(A, 0, {0: 1.0, 1: 2.0 * al})
                # the odd field's own value at the plane enters row 1 as it is
                _set(B, 0, {2: 2.0 * b, 1: 2.0 * a})
                _set(B, 1, {3: b, 1: b, 2: a, 0: -a})
            else:
                _set(A, 0, {0: 1.0})
                _set(B, 0, {})
                _set(B, 1, {3: b, 1: -b, 2: a, 0: -a})
            _set(A, n - 2, {n - 3: 0.5, n - 2: 1.0, n - 1: 1.0 / 6.0})
            _set(B, n - 2, {n - 1: 5.0 / 9.0, n - 2: 0.5, n - 3: -1.0, n - 4: -1.0 / 18.0})
            _set(A, n - 1, {n - 2: 2.0, n - 1: 1.0})
            _set(B, n - 1, {n - 1: 2.5, n - 2: -2.0, n - 3: -0.5})
    else:
        a, b, al = 12.0 / 11.0, 3.0 / 44.0, 2.0 / 11.0
        B = _stencil(n, {1: a, -1: a, 2: b, -2: b, 0: -2.0 * (a + b)}, sg, wrap)
        A = _band(n, {-1: al, 0: 1.0, 1: al}, wrap)
        if not wrap:
            _set(A, 0, {0: 1.0, 1: 2.0 * al})
            _set(B, 0, {2: 2.0 * b, 1: 2.0 * a, 0: -2.0 * (a + b)})
            _set(B, 1, {3: b, 1: -b - 2.0 * a, 2: a, 0: a})
            _set(A, n - 2, {n - 3: -0.35, n - 2: 1.0, n - 1: 0.1})
            _set(B, n - 2, {n - 1: 1.2375, n - 2: -3.0, n - 3: 2.325, n - 4: -0.6, n - 5: 0.0375})
            _set(A, n - 1, {n - 2: 11.0, n - 1: 1.0})
            _set(B, n - 1, {n - 1: 13.0, n - 2: -27.0, n - 3: 15.0, n - 4: -1.0})
    return np.linalg.solve(A, B) * ((n - 1) / length) ** order


def _filter_matrix(n, odd, wrap):
    sg = -1.0 if odd else 1.0
    f = [9.9965e-01, 0.66652, 0.16674, 4.0e-05, -5.0e-06]
    af, bf, ab = 6.6624e-01, 1.6688e-01, 0.45
    # mirrored weights of the symmetric formulas: f(-k) = f(k)
    B = _stencil(n, {k: f[abs(k)] for k in range(-4, 5)}, sg, wrap)
    A = _band(n, {-2: bf, -1: af, 0: 1.0, 1: af, 2: bf}, wrap)
    if wrap:
        return np.linalg.solve(A, B)
    if odd:
        _set(A, 0, {0: 1.0})
        _set(B, 0, {})
        _set(A, 1, {0: af, 1: 1.0 - bf, 2: af, 3: bf})
        # the odd formulas keep the reference's weights on f(0) and below
        _set(B, 1, {5: f[4], 3: -f[4], 4: f[3], 2: -f[3] + f[1], 1: f[0] - f[2], 0: f[1]})
        B[1, 3] += f[2]
        _set(B, 2, {6: f[4], 2: f[0] - f[4], 5: f[3], 1: f[1] - f[3], 0: f[2], 4: f[2], 3: f[1]})
        _set(B, 3, {7: f[4], 1: f[2] - f[4], 0: f[3], 6: f[3], 5: f[2], 2: f[1], 4: f[1], 3: f[0]})
    else:
        _set(A, 0, {0: 1.0, 1: 2.0 * af, 2: 2.0 * bf})
        _set(A, 1, {0: af, 1: 1.0 + bf, 2: af, 3: bf})
    _set(A, n - 3, {n - 4: ab, n - 3: 1.0, n - 2: ab})
    _set(A, n - 2, {n - 3: ab, n - 2: 1.0, n - 1: ab})
    _set(A, n - 1, {n - 1: 1.0})
    _set(B, n - 1, {n - 1: 15 / 16, n - 2: 1 / 4, n - 3: -3 / 8, n - 4: 1 / 4, n - 5: -1 / 16})
    _set(B, n - 2, {n - 1: 1 / 16 + 7 / 8 * ab, n - 2: 3 / 4 + ab / 2, n - 3: 3 / 8 + ab / 4, n - 4: -1 / 4 + ab / 2,
                    n - 5: 1 / 16 - ab / 8})
    c = [5 / 8 + 3 / 4 * ab, (1 / 2 + ab) / 2, (-1 / 8 + ab / 4) / 2]
    _set(B, n - 3, {n - 3 + k: c[abs(k)] for k in range(-2, 3)})
    c = [11 / 16 + 5 / 8 * af - 5 / 8 * bf, (15 / 32 + 17 / 16 * af + 15 / 16 * bf) / 2,
         (-3 / 16 + 3 / 8 * af + 13 / 8 * bf) / 2, (1 / 32 - af / 16 + bf / 16) / 2]
    _set(B, n - 4, {n - 4 + k: c[abs(k)] for k in range(-3, 4)})
    return np.linalg.solve(A, B)


def _gauss_matrix(n, wrap):
    g = [float(np.float32(v)) for v in (3565 / 10368, 3091 / 12960, 1997 / 25920, 149 / 12960, 107 / 103680)]
    M = _stencil(n, {k: g[abs(k)] for k in range(-4, 5)}, 1.0, wrap)
    if not wrap:
        for i in range(n - 4, n):
            _set(M, i, {i: 1.0})
    return M


def _along(M, F, d):
    """M applied along direction d (0: x, 1: y, 2: z) of F (..., nx, nz, ny)."""
    M = torch.from_numpy(M).cuda()
    if d == 1:
        return F @ M.T
    if d == 2:
        return M @ F
    return torch.tensordot(M, F, dims=([1], [0]))


def exact(case, seed):
    kind = case["kind"]
    if kind == "solvers":
        return _exact_solvers(case, seed)
    if kind not in ("derivatives", "filters"):
        return None   # whole calls: restating the solver would be a second implementation
    p = _params(case)
    shape, wrap = (p.nx, p.nz, p.ny), case["family"] == "periodic"
    n, length = (p.nx, p.ny, p.nz), (p.x_leng, p.y_leng, p.z_leng)
    if kind == "derivatives":
        F = _smooth(shape, _gen(seed), 3)
        d = torch.stack([_along(_d_matrix(n[k], length[k], 1, False, wrap), F[0], k) for k in range(3)])
        if not case["second"]:
            return {"d": d}
        d2 = torch.stack([_along(_d_matrix(n[k], length[k], 2, False, wrap), F[0], k) for k in range(3)])
        div = -sum(_along(_d_matrix(n[k], length[k], 1, True, wrap), F[k], k) for k in range(3))
        return {"d": d, "d2": d2, "div": div}
    Q = _smooth(shape, _gen(seed), 7)
    out = []
    for q in range(7):
        f = Q[q]
        for k in range(3):
            M = _filter_matrix(n[k], q == k and not wrap, wrap) if q < 5 else _gauss_matrix(n[k], wrap)
            f = _along(M, f, k)
        out.append(f)
    return {"Qf": torch.stack(out[:5]), "Eg": torch.stack(out[5:])}


def _exact_solvers(case, seed):
    """Each line's matrix solved densely, a block of lines at a time."""
    n, lot = case["n"], case["lot"]
    if n * n * lot > 4e9:
        return None
    tri, pen, R = _solver_coefficients(case, seed)
    out = []
    for k, (bands, per) in enumerate(((tri, 0), (tri, 1), (pen, 0), (pen, 1))):
        h = len(bands) // 2
        X = torch.empty_like(R[k])
        block = max(1, int(2e8 / (n * n)))
        i = torch.arange(n, device="cuda")
        for a in range(0, lot, block):
            m = min(block, lot - a)
            M = torch.zeros((m, n, n), dtype=torch.float64, device="cuda")
            for o in range(-h, h + 1):
                j = i + o
                ok = (j >= 0) & (j < n)
                if per:
                    ok, j = torch.ones_like(ok), j % n
                M[:, i[ok], j[ok]] += bands[o + h][i[ok], a:a + m].T
            X[:, a:a + m] = torch.linalg.solve(M, R[k][:, a:a + m].T.unsqueeze(-1)).squeeze(-1).T
        out.append(X)
    return out
