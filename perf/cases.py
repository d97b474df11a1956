"""Performance cases: the work that a user of this framework has it do, through its public entry
points (gbmv.py), from the smallest calls to the largest.

A case names the kind of call (`kind`), its grid and its options; `prepare` makes the inputs and
the handles that a program keeps, `run` makes one pass, `work` counts the bytes and operations
that the call cannot do without, `exact` evaluates the same formulas in plain FP64 torch.
"""
from __future__ import annotations

import math
import os
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sundials-manyvector-demo_gb300")
for _p in (PKG, ROOT):
    if _p not in sys.path:
        sys.path.insert(0, _p)

FP64, MIXED, MIXED_FAST = 0, 1, 2
PERIODIC, NEUMANN, REFLECTING = 0, 1, 3
TIME_UNITS = 1.0e11  # TimeUnits of the chemistry inputs
ENERGY_UNITS = 3.0e70 / 3.0857e30 / 1.0e22  # MassUnits / LengthUnits / TimeUnits^2
DENSITY_UNITS = 3.0e70 / 3.0857e30 ** 3
M_H = 1.67e-24
KB = 1.3806488e-16


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # the Sod tube input: the smallest grid anyone runs; one adaptive step makes five such calls
        dict(name="rhs_sod_tube", kind="rhs", ic="sod", nx=128, ny=3, nz=3, nchem=0,
             precision=FP64, bcx="rr", bcy="pp", bcz="pp"),
        # Rayleigh-Taylor flux divergence with ten tracers, the FP64 parity form
        dict(name="rhs_rt_fp64", kind="rhs", ic="rt", nx=128, ny=128, nz=128, nchem=10,
             precision=FP64, bcx="pp", bcy="pp", bcz="rr"),
        # an ordinary odd-sized local grid with outflow faces, the float-float form
        dict(name="rhs_ragged_mixed", kind="rhs", ic="smooth", nx=61, ny=45, nz=37, nchem=4,
             precision=MIXED, bcx="nn", bcy="pp", bcz="nr"),
        # the largest Rayleigh-Taylor grid of the throughput runs, the fastest form
        dict(name="rhs_rt_256_fast", kind="rhs", ic="rt", nx=256, ny=256, nz=256, nchem=10,
             precision=MIXED_FAST, bcx="pp", bcy="pp", bcz="rr"),
        # one stage of the chemistry-hydrodynamics program: explicit part and one chemistry Newton
        dict(name="chem_hydro_stage", kind="stage", nx=128, ny=128, nz=128, precision=MIXED_FAST,
             lu=MIXED, refine=2, gamma=1e-6),
        # implicit-stage Newton corrections with the FP64 factor on a small local grid
        dict(name="newton_stage_fp64", kind="newton", nx=24, ny=18, nz=14, lu=FP64, refine=0,
             gamma=1e-6),
        # the chemistry source alone: fimpl of an IMEX run, ffast of a multirate one
        dict(name="chem_rhs_64", kind="chem_rhs", nx=64, ny=64, nz=64),
        # the implicit solver's set-up (Jacobian, Newton matrix, block LU) and three solves with it
        dict(name="block_setup_solve", kind="implicit", nx=64, ny=60, nz=50, gamma=1e-6),
        # the matrix-free Jacobian action of Newton-Krylov on the flow
        dict(name="hydro_jvp_96", kind="jvp", nx=96, ny=96, nz=96, nchem=4),
        # the adjoint of the flow right-hand side, as in a gradient through time steps
        dict(name="hydro_vjp_96", kind="vjp", nx=96, ny=96, nz=96, nchem=4),
        # batched adaptive integration of every cell's chemistry, the fast stage
        dict(name="dirk_mixed", kind="dirk", nx=32, ny=32, nz=32, precision=MIXED, tout=1e-6),
        # what an adaptive step takes besides its right-hand sides: error norm, CFL step, totals
        dict(name="step_norms", kind="norms", nx=100, ny=100, nz=100, nchem=10),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, lo, hi, cells):
    while True:
        n = [_log_int(rng, lo, hi) for _ in range(3)]
        if n[0] * n[1] * n[2] <= cells:
            return dict(nx=n[0], ny=n[1], nz=n[2])


def draw(rng):
    kind = rng.choice(["rhs", "rhs", "rhs", "stage", "newton", "chem_rhs", "implicit", "jvp", "vjp",
                       "dirk", "norms"])
    if kind == "rhs":
        precision = rng.choice([FP64, MIXED, MIXED_FAST])
        c = dict(kind=kind, ic=rng.choice(["rt", "smooth"]), nchem=rng.choice([0, 2, 4, 6, 10]),
                 precision=precision, **_shape(rng, 3, 200, 1 << 21))
        for a in "xyz":
            c["bc" + a] = rng.choice(["pp", "rr", "nn", "nr", "rn"])
        return c
    gamma = 10.0 ** rng.uniform(-8, -5)  # h times the diagonal coefficient of an IMEX run
    if kind == "stage":
        return dict(kind=kind, precision=rng.choice([FP64, MIXED, MIXED_FAST]),
                    lu=rng.choice([FP64, MIXED]), refine=rng.choice([2, 3]), gamma=gamma,
                    **_shape(rng, 6, 128, 1 << 20))
    if kind == "newton":
        return dict(kind=kind, lu=rng.choice([FP64, MIXED]), refine=rng.choice([2, 4]),
                    gamma=gamma, **_shape(rng, 4, 100, 1 << 19))
    if kind == "implicit":
        return dict(kind=kind, gamma=gamma, **_shape(rng, 4, 100, 1 << 19))
    if kind == "chem_rhs":
        return dict(kind=kind, **_shape(rng, 4, 100, 1 << 19))
    if kind in ("jvp", "vjp"):
        return dict(kind=kind, nchem=rng.choice([0, 2, 4, 6, 10]), **_shape(rng, 4, 96, 1 << 19))
    if kind == "dirk":
        return dict(kind=kind, precision=rng.choice([FP64, MIXED]),
                    tout=10.0 ** rng.uniform(-7, -6), **_shape(rng, 4, 64, 1 << 15))
    return dict(kind=kind, nchem=rng.choice([0, 2, 4, 6, 10]), **_shape(rng, 4, 128, 1 << 20))


# ------------------------------------------------------------------ inputs

def _bc(case):
    code = {"p": PERIODIC, "n": NEUMANN, "r": REFLECTING}
    return tuple(code[ch] for a in "xyz" for ch in case.get("bc" + a, "pp"))


def _rand(gen, shape, lo, hi):
    return lo + (hi - lo) * torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64)


def _axis(n, dim):
    x = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
    return x.view([n if d == dim else 1 for d in range(3)])


def _flow(case, gen):
    """Fluid (and tracer) fields: the Sod tube with a seeded 1 % perturbation, the
    Rayleigh-Taylor state, or a smooth density wave with random velocities."""
    nx, ny, nz, nchem = case["nx"], case["ny"], case["nz"], case["nchem"]
    shp = (nz, ny, nx)
    one = torch.ones(shp, device="cuda", dtype=torch.float64)
    force = [0.0] * (5 + nchem)
    ic = case.get("ic", "smooth")
    if ic == "sod":
        left = (_axis(nx, 2) < 0.5).expand(shp)
        rho = torch.where(left, 1.0, 0.125).double() * _rand(gen, shp, 0.99, 1.01)
        p = torch.where(left, 1.0, 0.1).double()
        vel = _rand(gen, (3,) + shp, -0.01, 0.01)
    elif ic == "rt":
        z = _axis(nz, 0)
        rho = one * (1.5 + 0.5 * torch.tanh((z - 0.5) / 0.02))

        def lncosh(s):
            return torch.logaddexp(s, -s) - math.log(2.0)

        integral = 1.5 * (1.0 - z) + 0.01 * (
            lncosh(torch.full_like(z, 25.0)) - lncosh((z - 0.5) / 0.02))
        p = one * (2.5 + 0.1 * integral)
        vel = _rand(gen, (3,) + shp, -1e-2, 1e-2)
        force[3] = -0.1
    else:
        ph = 2 * math.pi * (_axis(nx, 2) + _axis(ny, 1) + _axis(nz, 0))
        rho = one * (1.0 + 0.2 * torch.sin(ph))
        p = one.clone()
        vel = _rand(gen, (3,) + shp, -0.1, 0.1)
    m = [(rho * v).contiguous() for v in vel]
    et = p / 0.4 + (m[0] ** 2 + m[1] ** 2 + m[2] ** 2) * 0.5 / rho
    w = [rho.contiguous(), *m, et.contiguous()]
    if nchem:
        w.append((_rand(gen, shp + (nchem,), 0.0, 1.0) * rho[..., None]).contiguous())
    return w, force


_MASS = (2.01588, 2.01588, 1.00794, 1.00794, 1.00794, 4.002602, 4.002602, 4.002602)


def _species(n, gen, dens, temp):
    """Primordial state: log-uniform mass fractions (hydrogen 0.76, helium 0.24), the electron
    density from charge balance, the gas energy of the given temperature."""
    fr = 10.0 ** _rand(gen, (n, 8), -10.0, 0.0)
    fr[:, :5] *= 0.76 / fr[:, :5].sum(1, keepdim=True)
    fr[:, 5:] *= 0.24 / fr[:, 5:].sum(1, keepdim=True)
    num = fr * dens[:, None] / (torch.tensor(_MASS, device="cuda", dtype=torch.float64) * M_H)
    de = (num[:, 3] + num[:, 6] + 2 * num[:, 7] - num[:, 4] + num[:, 1]) * M_H
    de = torch.clamp(de, min=1e-20 * M_H) / 1.66053904e-24
    ge = KB * temp * num.sum(1) / (dens * (5.0 / 3.0 - 1.0))
    return torch.cat([num, de[:, None], ge[:, None]], 1).contiguous()


def _chem_inputs(case, gen, perturb=1e-3):
    """(scale, scaled state ~1, a first guess of the temperature) of the static-chemistry
    inputs: 1e2 m_H, temperatures log-uniform in [10, 1e4] K."""
    n = case["nx"] * case["ny"] * case["nz"]
    temp = 10.0 ** _rand(gen, (n,), 1.0, 4.0)
    dens = torch.full((n,), 1e2 * M_H, device="cuda", dtype=torch.float64)
    scale = _species(n, gen, dens, temp)
    y = _rand(gen, (n, 10), 1.0 - perturb, 1.0 + perturb)
    return scale, y, temp


def _chem_hydro_inputs(case, gen):
    """A planar Sod-like interface along x carrying the primordial species."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    shp, n = (nz, ny, nx), nx * ny * nz
    left = (_axis(nx, 2) < 0.5).expand(shp).reshape(-1)
    dens = torch.where(left, 1e2 * M_H, 0.125e2 * M_H).double()
    temp = torch.where(left, 2000.0, 1600.0).double()
    y = _species(n, gen, dens, temp)
    rho = (dens / DENSITY_UNITS).view(shp)
    eint = (y[:, 9] / ENERGY_UNITS).view(shp)
    g = 5.0 / 3.0
    vel = _rand(gen, (3,) + shp, -0.1, 0.1) * torch.sqrt(g * (g - 1.0) * eint / rho)
    m = [(rho * v).contiguous() for v in vel]
    et = eint + 0.5 / rho * (m[0] ** 2 + m[1] ** 2 + m[2] ** 2)
    chem = _rand(gen, shp + (10,), 0.999, 1.001)
    w = [rho.contiguous(), *m, et.contiguous(), chem]
    return w, y, temp


_TABLES = None


def _tables():
    global _TABLES
    if _TABLES is None:
        import h5tables
        _TABLES = h5tables.load_table_block(
            os.path.join(ROOT, "tests", "golden", "primordial_tables.h5"))
    return _TABLES


_STAGE_BC = (REFLECTING, REFLECTING, PERIODIC, PERIODIC, PERIODIC, PERIODIC)


def _inputs(case, seed):
    """The arrays of a case, from its seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    d = {}
    if kind in ("rhs", "jvp", "vjp", "norms"):
        d["w"], d["force"] = _flow(case, gen)
        if kind != "rhs":
            d["v"] = [_rand(gen, f.shape, -1.0, 1.0) for f in d["w"]]
        if kind == "norms":
            d["v"] = [1e-6 * v for v in d["v"]]
    elif kind == "stage":
        d["w"], d["scale"], d["Ts"] = _chem_hydro_inputs(case, gen)
    else:
        d["scale"], d["y"], d["Ts"] = _chem_inputs(case, gen, 0.0 if kind == "dirk" else 1e-3)
        n = d["y"].shape[0]
        if kind == "newton":
            d["b"] = _rand(gen, (n, 10), -1e-3, 1e-3)
        elif kind == "implicit":
            d["b"] = [_rand(gen, (n, 10), -1.0, 1.0) for _ in range(3)]
    return d


def prepare(case, seed):
    import gbmv
    s = dict(case=case, gbmv=gbmv, **_inputs(case, seed))
    kind, shape = case["kind"], (case["nx"], case["ny"], case["nz"])
    n = shape[0] * shape[1] * shape[2]
    new = lambda *k: torch.empty(*k, device="cuda", dtype=torch.float64)  # noqa: E731
    if kind in ("rhs", "jvp", "vjp", "norms"):
        s["hydro"] = gbmv.Hydro(shape, case["nchem"], _bc(case), 1.4, s["force"])
        s["out"] = [torch.empty_like(f) for f in s["w"]]
        return s
    s["chem"] = gbmv.Chem(n, _tables())
    s["chem"].set_scale(s["scale"].view(-1))
    s["T"] = s["chem"].state("Ts")  # the handle's own memory: read back into buffers of ours
    s["T1"] = new(n)
    # the temperature that a stage carries over from the one before: that of the unperturbed state
    s["T"].copy_(s["Ts"])
    s["f"] = new(10 * n)
    s["chem"].calculate_rhs_cvklu(0.0, torch.ones_like(s["f"]), s["f"])
    s["Ts"] = s["T"].clone()
    if kind == "stage":
        s["hydro"] = gbmv.Hydro(shape, 10, _STAGE_BC, 5.0 / 3.0)
        s["out"] = [torch.empty_like(f) for f in s["w"]]
        s["status"] = torch.zeros(2, dtype=torch.int32, device="cuda")
    if kind in ("stage", "newton"):
        s["x"] = new(10 * n)
    elif kind == "chem_rhs":
        s["dT"], s["dT1"] = s["chem"].state("dTs_ge"), new(n)
    elif kind == "implicit":
        s["A"], s["x"] = new(100 * n), [new(10 * n) for _ in range(3)]
        s["ls"] = gbmv.BlockLinearSolver(n)
        s["chem"].calculate_rhs_cvklu(0.0, s["y"].view(-1), s["f"], TIME_UNITS)
        s["Ts"] = s["T"].clone()
    elif kind == "dirk":
        s["z"] = new(10 * n)
    return s


def run(s):
    g, case = s["gbmv"], s["case"]
    kind = case["kind"]
    if kind == "rhs":
        s["hydro"].fEuler(0.0, s["w"], s["out"], case["precision"])
        return s["out"]
    if kind == "jvp":
        s["hydro"].fEuler_jvp(0.0, s["w"], s["v"], s["out"])
        return s["out"]
    if kind == "vjp":
        s["hydro"].fEuler_vjp(0.0, s["w"], s["v"], s["out"])
        return s["out"]
    if kind == "norms":
        h = s["hydro"]
        return [h.wrms_norm(s["v"], s["w"], 1e-6, 1e-11), h.stability(s["w"], 0.5),
                *h.check_conservation(s["w"])]
    s["T"].copy_(s["Ts"])  # the temperature carried into the call
    if kind == "stage":
        g.fexpl_async(s["hydro"], s["chem"], 0.0, s["w"], s["out"], ENERGY_UNITS, s["status"][0:1],
                      case["precision"])
        g.chem_newton_async(s["chem"], 0.0, s["w"][5].view(-1), s["f"], s["x"], case["gamma"],
                            TIME_UNITS, s["status"][1:2], lu_precision=case["lu"],
                            refine=case["refine"])
        return dict(wdot=s["out"], et=s["w"][4], f=s["f"], x=s["x"], T=s["T1"].copy_(s["T"]))
    y = s["z"] if kind == "dirk" else s["y"].view(-1)
    if kind == "newton":
        s["chem"].newton_stage(0.0, y, s["b"].view(-1), s["f"], s["x"], case["gamma"], TIME_UNITS,
                               case["lu"], case["refine"])
        return dict(f=s["f"], x=s["x"], T=s["T1"].copy_(s["T"]))
    if kind == "chem_rhs":
        s["chem"].calculate_rhs_cvklu(0.0, y, s["f"], TIME_UNITS)
        return dict(f=s["f"], T=s["T1"].copy_(s["T"]), dT=s["dT1"].copy_(s["dT"]))
    if kind == "implicit":
        s["chem"].calculate_jacobian_cvklu(0.0, y, s["A"], TIME_UNITS)
        g.form_newton_matrix(s["A"], case["gamma"])
        s["ls"].setup(s["A"])
        for b, x in zip(s["b"], s["x"]):
            s["ls"].solve(s["A"], x, b.view(-1))
        return s["x"]
    y.fill_(1.0)
    failed = s["chem"].dirk_evolve(0.0, case["tout"], y, TIME_UNITS, rtol=1e-6, atol=1e-10, maxcor=10,
                                   nlscoef=0.01, precision=case["precision"], block=32)
    return dict(y=y, T=s["T1"].copy_(s["T"]), failed=failed)


def work(case):
    """Bytes: each input read once, each output written once.  Operations: of the formulas with
    shared subexpressions (FMA = 2), not of any kernel."""
    n = case["nx"] * case["ny"] * case["nz"]
    kind = case["kind"]
    nv = 5 + case.get("nchem", 10)
    # per face: ~250 for the averages, projections and fluxes, ~60 per reconstruction and side
    face = 3 * (250 + 120 * nv)
    if kind == "rhs":
        return dict(bytes=n * 16 * nv, flops=n * (face + 9 * nv))
    if kind == "jvp":
        return dict(bytes=n * 24 * nv, flops=n * 3 * face)
    if kind == "vjp":
        return dict(bytes=n * 24 * nv, flops=n * 4 * face)
    if kind == "norms":
        return dict(bytes=n * 8 * (2 * nv + 5 + 2), flops=n * (6 * nv + 20))
    rhs, jac, lu = 500, 700, 800
    if kind == "stage":
        return dict(bytes=n * (16 * 15 + 8 * 46), flops=n * (face + rhs + jac + lu + 200))
    if kind == "newton":
        return dict(bytes=n * 8 * 56, flops=n * (rhs + jac + lu + 200))
    if kind == "chem_rhs":
        return dict(bytes=n * 8 * 46, flops=n * rhs)
    if kind == "implicit":
        return dict(bytes=n * 8 * (36 + 60), flops=n * (jac + lu + 3 * 200))
    # a dozen steps of seven stages, two to three iterations each
    return dict(bytes=n * 8 * 50, flops=n * (12 * 20 * (rhs + 250) + 12 * (jac + lu)))


# ------------------------------------------------------------------ plain FP64 evaluation

def _pad(f, dim, bc, normal):
    """Three ghost cells on both sides of `dim`: periodic wrap, else the lower mirror and the
    upper shifted copy, negated for the normal momentum at a reflecting face."""
    n = f.shape[dim]
    if bc[0] == PERIODIC:
        return torch.cat([f.narrow(dim, n - 3, 3), f, f.narrow(dim, 0, 3)], dim)
    lo = f.narrow(dim, 0, 3).flip(dim)
    hi = f.narrow(dim, n - 3, 3)
    if normal and bc[0] == REFLECTING:
        lo = -lo
    if normal and bc[1] == REFLECTING:
        hi = -hi
    return torch.cat([lo, f, hi], dim)


def _weno(f, minus):
    """Fifth-order WENO value at i+1/2 from five points (the mirrored stencil for the minus
    side), Jiang-Shu indicators, eps = 1e-6, squared weights."""
    if minus:
        f = f[::-1]
    a, b, c, d, e = f
    bC = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    bB = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    bA = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    tA, tB, tC = 0.3 / (1e-6 + bA) ** 2, 0.6 / (1e-6 + bB) ** 2, 0.1 / (1e-6 + bC) ** 2
    qA, qB, qC = (2 * c + 5 * d - e) / 6, (-b + 5 * c + 2 * d) / 6, (2 * a - 7 * b + 11 * c) / 6
    return (tA * qA + tB * qB + tC * qC) / (tA + tB + tC)


def _direction(w, d, bc, gamma, h):
    """- d F_d / d x_d of the fluid fields and tracers."""
    dim = 2 - d
    n = w[0].shape[dim]
    order = [0, 1 + d, *[1 + k for k in range(3) if k != d], 4]
    P = [_pad(w[k], dim, bc, k == 1 + d) for k in order]
    W = [[p.narrow(dim, j, n + 1) for p in P] for j in range(6)]
    gm = gamma - 1.0
    p = [gm * (q[4] - (q[1] ** 2 + q[2] ** 2 + q[3] ** 2) * 0.5 / q[0]) for q in W]
    u6 = [q[1] / q[0] for q in W]
    sL, sR = torch.sqrt(W[2][0]), torch.sqrt(W[3][0])
    sb = 0.5 * (sL + sR)
    u, v, ww = (0.5 * (W[2][k] / sL + W[3][k] / sR) / sb for k in (1, 2, 3))
    H = 0.5 * ((p[2] + W[2][4]) / sL + (p[3] + W[3][4]) / sR) / sb
    q2 = u * u + v * v + ww * ww
    c = gm * (H - 0.5 * q2)
    rows = [
        (0.5 / c * (u + 0.5 * gm * q2), -0.5 / c * (gm * u + 1), -0.5 * gm * v / c,
         -0.5 * gm * ww / c, 0.5 * gm / c),
        None, None,
        (-gm / c * (q2 - H), gm * u / c, gm * v / c, gm * ww / c, -gm / c),
        (-0.5 / c * (u - 0.5 * gm * q2), -0.5 / c * (gm * u - 1), -0.5 * gm * v / c,
         -0.5 * gm * ww / c, 0.5 * gm / c)]
    alpha = u6[0].abs() + torch.sqrt(gamma * p[0] / W[0][0])
    for j in range(1, 6):
        alpha = torch.maximum(alpha, u6[j].abs() + torch.sqrt(gamma * p[j] / W[j][0]))
    ff = [None] * 5
    for side in (0, 1):
        pr = []
        for j in range(side, side + 5):
            q, uj, pj = W[j], u6[j], p[j]
            fl = (q[1], uj * q[1] + pj, uj * q[2], uj * q[3], uj * (q[4] + pj))
            s = [0.5 * (x + (alpha if side == 0 else -alpha) * y) for x, y in zip(fl, q)]
            pr.append([sum(r * x for r, x in zip(rows[i], s)) if rows[i] is not None
                       else s[1 + i] - (v if i == 1 else ww) * s[0] for i in range(5)])
        for i in range(5):
            r = _weno([pr[j][i] for j in range(5)], side == 1)
            ff[i] = r if side == 0 else ff[i] + r
    out = [None] * 5
    fo = [ff[0] + ff[3] + ff[4], (u - c) * ff[0] + u * ff[3] + (u + c) * ff[4],
          v * (ff[0] + ff[3] + ff[4]) + ff[1], ww * (ff[0] + ff[3] + ff[4]) + ff[2],
          (H - u * c) * ff[0] + v * ff[1] + ww * ff[2] + 0.5 * q2 * ff[3] + (H + u * c) * ff[4]]
    for k, f in zip(order, fo):
        out[k] = -(f.narrow(dim, 1, n) - f.narrow(dim, 0, n)) / h
    if len(w) > 5:
        cols = []
        for k in range(w[5].shape[3]):
            q = _pad(w[5][..., k], dim, bc, False)
            q = [q.narrow(dim, j, n + 1) for j in range(6)]
            f = (_weno([0.5 * (u6[j] + alpha) * q[j] for j in range(5)], False) +
                 _weno([0.5 * (u6[j] - alpha) * q[j] for j in range(1, 6)], True))
            cols.append(-(f.narrow(dim, 1, n) - f.narrow(dim, 0, n)) / h)
        out.append(torch.stack(cols, -1))
    return out


def _rhs(w, bc, gamma, force):
    shp = w[0].shape
    tot = None
    for d in range(3):
        o = _direction(w, d, bc[2 * d:2 * d + 2], gamma, 1.0 / shp[2 - d])
        tot = o if tot is None else [a + b for a, b in zip(tot, o)]
    return [t + force[k] if k < 5 else t for k, t in enumerate(tot)]


class _Chem:
    """The primordial network in physical units, one row per cell."""

    def __init__(self, y, scale, T0):
        self.tab = torch.tensor(_tables(), device="cuda", dtype=torch.float64)
        self.y = y * scale
        self.scale = scale
        m = (scale[:, :8] * torch.tensor(_MASS, device="cuda", dtype=torch.float64)).sum(1)
        # H2 species count twice the atomic weight 1 in the network's density
        m = (2 * (scale[:, 0] + scale[:, 1]) + 1.00794 * scale[:, 2:5].sum(1) +
             4.002602 * scale[:, 5:8].sum(1)) * 1.67e-24
        self.md = m
        tau = torch.clamp((m / 3.3e-8) ** 2.8, min=1e-5)
        self.cie = torch.clamp((1 - torch.exp(-tau)) / tau, max=1.0)
        self.h2 = torch.clamp((m / 1.34e-14) ** -0.45, max=1.0)
        self._temperature(T0)
        self._rates()

    def _bins(self, T):
        db = math.log(1e5) / 1023
        x = torch.log(T)
        b = torch.clamp((x / db).long(), 0, 1022)
        return b, (x - b.double() * db) / db, db

    def _temperature(self, T):
        y, kb, mh = self.y, 1.3806504e-16, 1.67e-24
        dmh = (2 * (y[:, 0] + y[:, 1]) + 1.00794 * y[:, 2:5].sum(1) +
               4.002602 * y[:, 5:8].sum(1)) * mh
        for _ in range(30):
            b, w, _d = self._bins(T)
            t = [self.tab[r][b] + w * (self.tab[r][b + 1] - self.tab[r][b]) for r in range(46, 50)]
            g1, dg1, g2, dg2 = t
            i1, i2 = 1 / (g1 - 1), 1 / (g2 - 1)
            ns = y[:, 0] * i1 + y[:, 1] * i2 + 1.5 * y[:, 2:9].sum(1)
            dge = T * kb * (-y[:, 0] * i1 * i1 * dg1 - y[:, 1] * i2 * i2 * dg2) / dmh + kb * ns / dmh
            T = T - (T * kb * ns / dmh - y[:, 9]) / dge
        self.T, self.dT = torch.clamp(T, 1.0, 1e5), 1 / dge

    def _rates(self):
        b, w, db = self._bins(self.T)
        self.k, self.dk = {}, {}
        for r in range(46):
            d = self.tab[r][b + 1] - self.tab[r][b]
            self.k[r] = self.tab[r][b] + w * d
            self.dk[r] = d / (db * self.T)

    @staticmethod
    def _sources(k, y):
        """Species sources of the 21 reactions, in the tables' order k01..k19, k21, k22."""
        H2, H2p, H, Hp, Hm, He, Hep, Hepp, e = (y[:, i] for i in range(9))
        r = [k[0] * H * e, k[1] * Hp * e, k[2] * He * e, k[3] * Hep * e, k[4] * Hep * e,
             k[5] * Hepp * e, k[6] * H * e, k[7] * H * Hm, k[8] * H * Hp, k[9] * H2p * H,
             k[10] * H2 * Hp, k[11] * H2 * e, k[12] * H2 * H, k[13] * Hm * e, k[14] * H * Hm,
             k[15] * Hp * Hm, k[16] * Hp * Hm, k[17] * H2p * e, k[18] * H2p * Hm,
             k[19] * H2 * H * H, k[20] * H * H * H]
        return torch.stack([
            r[7] + r[9] - r[10] - r[11] - r[12] + r[18] + r[19] + r[20],
            r[8] - r[9] + r[10] + r[16] - r[17] - r[18],
            -r[0] + r[1] - r[6] - r[7] - r[8] - r[9] + r[10] + 2 * r[11] + 2 * r[12] + r[13] +
            r[14] + 2 * r[15] + 2 * r[17] + r[18] - 2 * r[19] - 2 * r[20],
            r[0] - r[1] - r[8] + r[9] - r[10] - r[15] - r[16],
            r[6] - r[7] - r[13] - r[14] - r[15] - r[16] - r[18],
            -r[2] + r[3], r[2] - r[3] - r[4] + r[5], r[4] - r[5],
            r[0] - r[1] + r[2] - r[3] + r[4] - r[5] - r[6] + r[7] + r[13] + r[14] + r[16] - r[17],
        ], 1)

    # cooling tables after the 21 rates
    BREM, CEHEI, CEHEII, CEHI, CIECO, CIHEI, CIHEII, CIHEIS, CIHI, COMPTON, GAEL, GAH2, GAHE, GAHI, \
        GAHP, LTE, MCOOL, MHEAT, NCRD1, NCRD2, NCRN, RE1, RE2, RE3, REH = range(21, 46)

    def _terms(self):
        k, y = self.k, self.y
        H2, H, Hp, He, e = y[:, 0], y[:, 2], y[:, 3], y[:, 5], y[:, 8]
        G = H2 * k[self.GAH2] + H * k[self.GAHI] + Hp * k[self.GAHP] + He * k[self.GAHE] + \
            e * k[self.GAEL]
        N = H2 * k[self.NCRD2] + H * k[self.NCRD1]
        Hf = -H2 * H * k[self.MCOOL] + H ** 3 * k[self.MHEAT]
        return G, k[self.LTE] / G + 1, N, k[self.NCRN] / N + 1, Hf

    def source(self):
        k, y = self.k, self.y
        H2, _, H, Hp, _, He, Hep, Hepp, e = (y[:, i] for i in range(9))
        G, D, N, F, Hf = self._terms()
        lin = (H * (k[self.CEHI] + k[self.CIHI]) + Hp * k[self.REH] + He * k[self.CIHEI] +
               Hep * (k[self.CEHEII] + k[self.CIHEII] + k[self.RE1] + k[self.RE2]) +
               Hep * e * (k[self.CEHEI] + k[self.CIHEIS]) + Hepp * k[self.RE3] +
               k[self.BREM] * (Hp + Hep + 4 * Hepp))  # Compton term: (1 + z)^4 = 0 at z = -1
        ge = (-2.01588 * H2 * k[self.CIECO] * self.cie * self.md -
              H2 * self.cie * k[self.LTE] * self.h2 / D - self.cie * e * lin + 0.5 * Hf / F)
        f = torch.cat([self._sources(k, y), (ge / self.md)[:, None]], 1)
        return f / self.scale * TIME_UNITS

    def jacobian(self):
        """The network's analytic Jacobian in scaled variables, J[:, row, col]."""
        k, dk, y = self.k, self.dk, self.y
        H2, _, H, Hp, _, He, Hep, Hepp, e = (y[:, i] for i in range(9))
        J = torch.zeros(y.shape[0], 10, 10, device="cuda", dtype=torch.float64)
        for q in range(9):  # species by species: the sources are polynomials
            v = torch.zeros_like(y)
            v[:, q] = 1.0
            J[:, :9, q] = torch.func.jvp(lambda x: self._sources(k, x), (y,), (v,))[1]
        J[:, :9, 9] = self._sources(dk, y) * self.dT[:, None]
        G, D, N, F, Hf = self._terms()
        lte, h2o, md = k[self.LTE], self.h2, self.md
        a = lte ** 2 * h2o / (D * G) ** 2
        b = 0.5 * k[self.NCRN] * Hf / (F * N) ** 2
        g = {}
        g[0] = -H2 * k[self.GAH2] * a - 0.5 * H * k[self.MCOOL] / F - \
            2.01588 * k[self.CIECO] * md - lte * h2o / D + b * k[self.NCRD2]
        g[2] = -H2 * k[self.GAHI] * a - (k[self.CEHI] + k[self.CIHI]) * e + b * k[self.NCRD1] + \
            0.5 * (-H2 * k[self.MCOOL] + 3 * H ** 2 * k[self.MHEAT]) / F
        g[3] = -H2 * k[self.GAHP] * a - (k[self.BREM] + k[self.REH]) * e
        g[5] = -H2 * k[self.GAHE] * a - k[self.CIHEI] * e
        g[6] = -e * (k[self.BREM] + k[self.CEHEII] + k[self.CIHEII] + k[self.RE1] + k[self.RE2]) - \
            e * e * (k[self.CEHEI] + k[self.CIHEIS])
        g[7] = -e * (4 * k[self.BREM] + k[self.RE3])
        g[8] = -H2 * k[self.GAEL] * a - H * (k[self.CEHI] + k[self.CIHI]) - Hp * k[self.REH] - \
            He * k[self.CIHEI] - Hep * (k[self.CEHEII] + k[self.CIHEII] + k[self.RE1] +
                                        k[self.RE2]) - \
            2 * Hep * e * (k[self.CEHEI] + k[self.CIHEIS]) - Hepp * k[self.RE3] - \
            k[self.BREM] * (Hp + Hep + 4 * Hepp)
        for q, v in g.items():
            J[:, 9, q] = v / md
        dG = H2 * dk[self.GAH2] + H * dk[self.GAHI] + Hp * dk[self.GAHP] + He * dk[self.GAHE] + \
            e * dk[self.GAEL]
        dN = H2 * dk[self.NCRD2] + H * dk[self.NCRD1]
        gg = -H2 * lte * h2o * (lte * dG / G ** 2 - dk[self.LTE] / G) / D ** 2 - \
            H2 * h2o * dk[self.LTE] / D + \
            0.5 * Hf / F ** 2 * (k[self.NCRN] * dN / N ** 2 - dk[self.NCRN] / N) + \
            0.5 / F * (-H2 * H * dk[self.MCOOL] + H ** 3 * dk[self.MHEAT])
        J[:, 9, 9] = gg / md * self.dT
        return J * (self.scale[:, None, :] / self.scale[:, :, None]) * TIME_UNITS


def _newton_matrix(C, gamma):
    return torch.eye(10, device="cuda", dtype=torch.float64) - gamma * C.jacobian()


def exact(case, seed):
    kind = case["kind"]
    if kind == "dirk":
        return None  # adaptive: no closed form
    d = _inputs(case, seed)
    if kind == "rhs":
        return _rhs(d["w"], _bc(case), 1.4, d["force"])
    if kind == "jvp":
        fn = lambda *w: tuple(_rhs(list(w), _bc(case), 1.4, d["force"]))  # noqa: E731
        return list(torch.func.jvp(fn, tuple(d["w"]), tuple(d["v"]))[1])
    if kind == "vjp":
        tot = None
        for a in range(3):
            w = [f.clone().requires_grad_(True) for f in d["w"]]
            o = _direction(w, a, _bc(case)[2 * a:2 * a + 2], 1.4, 1.0 / w[0].shape[2 - a])
            g = torch.autograd.grad(o, w, d["v"])
            tot = list(g) if tot is None else [x + y for x, y in zip(tot, g)]
        return tot
    if kind == "norms":
        w, v = d["w"], d["v"]
        num = sum(((a / (1e-6 * b.abs() + 1e-11)) ** 2).sum() for a, b in zip(v, w))
        norm = torch.sqrt(num / sum(a.numel() for a in v))
        p = 0.4 * (w[4] - (w[1] ** 2 + w[2] ** 2 + w[3] ** 2) * 0.5 / w[0])
        speed = ((w[1] / w[0]).abs() + torch.sqrt(1.4 * p / w[0])).max()
        dx = min(1.0 / case["nx"], 1.0 / case["ny"], 1.0 / case["nz"])
        return [float(norm), float(0.5 * dx / speed), float(w[0].sum()), float(w[4].sum())]
    if kind == "stage":
        w = d["w"]
        chem = w[5].reshape(-1, 10)
        C = _Chem(chem, d["scale"], d["Ts"])
        phys = (chem * d["scale"]).view(w[5].shape)
        et = phys[..., 9] / ENERGY_UNITS + 0.5 / w[0] * (w[1] ** 2 + w[2] ** 2 + w[3] ** 2)
        r = _rhs([*w[:4], et, phys], _STAGE_BC, 5.0 / 3.0, [0.0] * 15)
        r[5] = torch.cat([r[5][..., :9], r[4][..., None]], -1)
        r[4] = torch.zeros_like(r[4])
        f = C.source()
        x = torch.linalg.solve(_newton_matrix(C, case["gamma"]), f)
        return dict(wdot=r, et=et, f=f.reshape(-1), x=x.reshape(-1), T=C.T)
    C = _Chem(d["y"], d["scale"], d["Ts"])
    f = C.source()
    if kind == "chem_rhs":
        return dict(f=f.reshape(-1), T=C.T, dT=C.dT)
    A = _newton_matrix(C, case["gamma"])
    if kind == "newton":
        x = torch.linalg.solve(A, d["b"] + case["gamma"] * f)
        return dict(f=f.reshape(-1), x=x.reshape(-1), T=C.T)
    return [torch.linalg.solve(A, b).reshape(-1) for b in d["b"]]
