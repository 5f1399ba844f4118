"""Timing cases of the package: calls that a user's program makes, over the sizes it makes them with.

Every case goes through the Python mirror of the reference's API (``DGModel``,
``LSRK54CarpenterKennedy`` / ``dostep_``, ``Ensemble``,
``ARK2GiraldoKellyConstantinescu`` and the filters).  ``exact`` restates the
same calls in plain FP64 torch: hexahedral grids with curl-invariant metrics,
the dry AtmosModel tendency in weak DG form with its hydrostatic reference
state, SmagorinskyLilly, ConstantDynamicViscosity and DryBiharmonic, LSRK54,
and ARK2 with a dense solve per column.

Initial states are the configurations' own flows plus seeded smooth winds, so
that every term of the equations is active.
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "climatemachine.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import cmdg  # noqa: E402
from cmdg import filters  # noqa: E402

# constants of the planet and of dry air (the package's defaults)
R_D = 8.3144598 / 28.97e-3
CP_D = R_D / (2 / 7)
CV_D = CP_D - R_D
T_0, GRAV, MSLP, RADIUS = 273.16, 9.81, 1.01325e5, 6.371e6
INV_PR, C_SMAG = 3.0, 0.21
RHO_NU = 2.0          # dynamic viscosity of the "constant" closure
BOX = 2500.0          # side of the bubble's box
LID = 30e3            # lid of the GCM shell
WAVE_LID = 10e3       # lid of the acoustic-wave shell


def listed():
    return [
        # one right-hand side of the periodic vortex on 4^3 elements: the smallest
        # call (a driver that has its own time stepper, a convergence study's
        # coarse level); FP64 as the reference runs it
        dict(name="vortex_rhs_fp64", kind="vortex", nx=4, ny=4, nz=4, N=4, precision="fp64"),
        # a step of one small ensemble member run by itself: launches and latency
        dict(name="bubble_small", kind="bubble", nx=9, ny=8, nz=11, N=3, precision="mixed", closure="none"),
        # the rising bubble on 20^3 elements, the package's default workload
        dict(name="bubble", kind="bubble", nx=20, ny=20, nz=20, N=4, precision="mixed", closure="none"),
        # the same in plain FP64, the reference's precision
        dict(name="bubble_fp64", kind="bubble", nx=20, ny=20, nz=20, N=4, precision="fp64", closure="none"),
        # a large box with odd element counts and the highest order
        dict(name="bubble_large", kind="bubble", nx=33, ny=31, nz=29, N=5, precision="mixed", closure="none"),
        # the bubble on a terrain-following mesh handed over as grid arrays
        dict(name="terrain_arrays", kind="terrain", nx=20, ny=18, nz=16, N=4, precision="mixed"),
        # an uneven ensemble of bubbles, orders 3 to 5, in one call
        dict(name="ensemble", kind="ensemble", members=24, sizes=2024),
        # a step of the dry GCM on the cubed shell
        dict(name="gcm", kind="gcm", nhorz=12, nvert=6, N=4, precision="mixed", closure="none"),
        # the GCM with horizontal hyperdiffusion, as climate runs configure it
        dict(name="gcm_hyper", kind="gcm", nhorz=9, nvert=7, N=4, precision="mixed", closure="hyper"),
        # Smagorinsky LES, the diffusive passes
        dict(name="les", kind="les", nx=32, ny=32, nz=16, N=4, precision="mixed", closure="smagorinsky"),
        # a smaller LES in FP64, the check that a production run is compared with
        dict(name="les_fp64", kind="les", nx=15, ny=16, nz=9, N=4, precision="fp64", closure="smagorinsky"),
        # the acoustic wave on the sphere stepped implicitly in the vertical, with its filter
        dict(name="hevi_wave", kind="hevi", nhorz=10, nvert=5, N=5, precision="mixed"),
    ]


def draw(rng: random.Random):
    """One more case of the same kinds and ranges."""
    kind = rng.choice(["vortex", "bubble", "bubble", "bubble", "terrain", "ensemble", "gcm", "gcm", "les", "les", "hevi"])
    if kind == "ensemble":
        return dict(kind=kind, members=rng.randint(2, 24), sizes=rng.randrange(1 << 20))
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind in ("gcm", "hevi"):
        c = dict(kind=kind, nhorz=rng.randint(3, 12 if kind == "gcm" else 10),
                 nvert=rng.randint(2, 8 if kind == "gcm" else 5), N=rng.randint(3, 5), precision=precision)
        if c["N"] == 5:
            c["nhorz"] = min(c["nhorz"], 10)
        if kind == "gcm":
            c["closure"] = rng.choice(["none", "none", "hyper"])
        return c
    closure = {"bubble": rng.choice(["none", "none", "none", "hyper"]),
               "les": rng.choice(["smagorinsky", "smagorinsky", "constant"])}.get(kind)
    # elements in all, log-uniform, and a box of uneven sides
    N = rng.randint(2, 5) if kind != "terrain" else rng.randint(3, 5)
    most = {"vortex": 1e6, "terrain": 8e5, "les": 2e6}.get(kind, 4e6)
    most = min(most, 1e6) if precision == "fp64" else most
    total = math.exp(rng.uniform(math.log(64), math.log(most / (N + 1) ** 3)))
    side = total ** (1 / 3)
    nx, ny = (max(3, round(side * rng.uniform(0.7, 1.4))) for _ in range(2))
    nz = max(3, round(total / (nx * ny)))
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, N=N, precision=precision if kind != "vortex" else "fp64")
    if closure:
        c["closure"] = closure
    return c


# --------------------------------------------------------------------------
# what a user's program has before the call
# --------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] == "ensemble":
        specs = _member_specs(case)
        members, states = [], []
        for n, s in enumerate(specs):
            dg, Q = _model(s), _initial(s, _coordinates(s), seed * 131 + n)
            members.append(dg)
            states.append(dg.to_perturbation(Q))
        regs = [torch.zeros(q.shape, dtype=torch.float64, device=q.device) for q in states]
        return dict(call="ensemble", ens=cmdg.Ensemble(members), Qs=states, dQs=regs, dts=[_dt(s) for s in specs])
    dg = _model(case)
    Q = _initial(case, _coordinates(case), seed)
    if case["kind"] == "vortex":
        return dict(call="rhs", dg=dg, Q=Q, T=torch.zeros_like(Q))
    if case["kind"] == "hevi":
        lin = cmdg.DGModel(cmdg.AtmosAcousticGravityLinearModel(dg.balance_law), dg.grid, direction="vertical",
                           state_auxiliary=dg)
        ark = cmdg.ARK2GiraldoKellyConstantinescu(dg, lin, cmdg.LinearBackwardEulerSolver(cmdg.ManyColumnLU()), Q,
                                                  dt=_dt(case))
        return dict(call="hevi", dg=dg, Q=Q, ark=ark, filt=filters.ExponentialFilter(dg.grid, 0, 18),
                    fdg=_model(dict(case, precision="fp64")) if dg.mixed else dg)
    if dg.mixed:
        Q = dg.to_perturbation(Q)
    return dict(call="step", dg=dg, Q=Q, lsrk=cmdg.LSRK54CarpenterKennedy(dg, Q, dt=_dt(case)))


def run(state):
    call = state["call"]
    if call == "rhs":
        return state["dg"](state["T"], state["Q"], None, 0.0)
    if call == "ensemble":
        state["ens"].lsrk54_step(state["Qs"], state["dQs"], state["dts"])
        return state["Qs"]
    if call == "hevi":
        cmdg.dostep_(state["Q"], state["ark"], None, 0.0)
        return filters.apply_(state["Q"], None, state["fdg"], state["filt"], direction="vertical")
    cmdg.dostep_(state["Q"], state["lsrk"], None, 0.0)
    return state["Q"]


def work(case):
    """A Runge-Kutta stage depends on the whole previous stage, so the state
    is read and written once per stage, the FP64 register as well (not read
    by the first stage nor written by the last), and per-node geometry read."""
    if case["kind"] == "ensemble":
        each = [work(s) for s in _member_specs(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    N, Nq = case["N"], case["N"] + 1
    nodes = _nelem(case) * Nq**3
    b = 4 if case.get("precision") == "mixed" else 8
    geo = {"gcm": 13, "hevi": 13, "terrain": 19}.get(case["kind"], 0) * b
    # volume contraction, pointwise terms, 6 (N+1)^2 face nodes
    rhs = 30 * Nq + 60 + 6 * 70 / Nq
    passes = {"smagorinsky": 30 * Nq + 250, "constant": 24 * Nq + 120, "hyper": 54 * Nq + 150}.get(case.get("closure"), 0)
    if case["kind"] == "vortex":
        return {"bytes": nodes * 80.0, "flops": nodes * rhs}
    if case["kind"] == "hevi":
        n, bw = 5 * Nq * case["nvert"], 5 * Nq - 1
        lines = 6 * case["nhorz"] ** 2 * Nq * Nq
        # two solves read the factors' non-zeros; three tendencies, the filter
        lu = 2 * 0.66 * (2 * bw + 1) * n * lines
        return {"bytes": lu * 8 + nodes * (3 * (80 + geo) + 240.0), "flops": 2 * lu + nodes * 3 * (rhs + 20 * Nq)}
    return {"bytes": nodes * (5 * 10 * b + 8 * 40 + 5 * geo), "flops": nodes * 5.0 * (rhs + passes)}


# --------------------------------------------------------------------------
# the cases' meshes, models and initial states
# --------------------------------------------------------------------------
def _member_specs(case):
    """Members of an ensemble: 8 to 16 elements a side, orders 3 to 5."""
    r = random.Random(case["sizes"])
    return [dict(kind="bubble", nx=r.randint(8, 16), ny=r.randint(8, 16), nz=r.randint(8, 16), N=r.randint(3, 5),
                 precision="mixed", closure="none") for _ in range(case["members"])]


def _is_shell(case):
    return case["kind"] in ("gcm", "hevi")


def _nelem(case):
    return 6 * case["nhorz"] ** 2 * case["nvert"] if _is_shell(case) else case["nx"] * case["ny"] * case["nz"]


def _box(case):
    """Corners of a box: the vortex's periodic cube, the LES's 100 m cells, the bubble's cube."""
    if case["kind"] == "vortex":
        return (-0.05,) * 3, (0.05,) * 3
    if case["kind"] == "les":
        return (0.0,) * 3, (100.0 * case["nx"], 100.0 * case["ny"], 100.0 * case["nz"])
    return (0.0,) * 3, (BOX,) * 3


def _lid(case):
    return LID if case["kind"] == "gcm" else WAVE_LID


def _dt(case):
    """A step at an acoustic Courant number of 0.4 (0.3 horizontally for HEVI)."""
    gap = float(_lgl(case["N"])[0][1] + 1) / 2
    if case["kind"] == "hevi":
        return 0.3 * gap * (math.pi / 2 * RADIUS / case["nhorz"]) / 350.0
    if case["kind"] == "gcm":
        return 0.4 * gap * min(LID / case["nvert"], math.pi / 2 * RADIUS / case["nhorz"]) / 370.0
    lo, hi = _box(case)
    h = min((b - a) / n for a, b, n in zip(lo, hi, (case["nx"], case["ny"], case["nz"])))
    return (0.3 if case["kind"] == "terrain" else 0.4) * gap * h / 350.0


def _model(case):
    N, precision = case["N"], case["precision"]
    closure = case.get("closure", "none")
    if _is_shell(case):
        grid = cmdg.CubedShellGrid(N, case["nhorz"], case["nvert"], RADIUS, RADIUS + _lid(case))
        law = cmdg.AtmosModel(orientation="sphere", gravity=True,
                              ref_state=cmdg.HydrostaticState(cmdg.IsothermalProfile(_profile(case)[1])),
                              hyperdiffusion=cmdg.DryBiharmonic(8 * 3600.0) if closure == "hyper" else None)
        return cmdg.DGModel(law, grid, precision=precision, diffusion_direction="horizontal")
    lo, hi = _box(case)
    ne = (case["nx"], case["ny"], case["nz"])
    if case["kind"] == "vortex":
        return cmdg.DGModel(cmdg.AtmosModel(), cmdg.BrickGrid(N, ne, lo, hi), precision=precision)
    law = cmdg.AtmosModel(orientation="flat", gravity=True,
                          ref_state=cmdg.HydrostaticState(cmdg.DryAdiabaticProfile(300.0, 0.0)),
                          turbulence=closure if closure in ("smagorinsky", "constant") else "none", rho_nu=RHO_NU,
                          C_smag=C_SMAG, hyperdiffusion=cmdg.DryBiharmonic(3600.0) if closure == "hyper" else None)
    if case["kind"] == "terrain":
        g = _Grid(case)
        vgeo = torch.zeros((g.nelem, 16, g.Np), dtype=torch.float64, device=g.X.device)
        for d in range(3):
            for j in range(3):
                vgeo[:, 3 * j + d] = g.xi[d][j]
        vgeo[:, 9] = g.J * g.www
        vgeo[:, 10] = 1 / vgeo[:, 9]
        vgeo[:, 12:15] = g.X.permute(1, 0, 2)
        wall = g.wall.to(torch.int64)
        wall[:, 5] *= 2
        arrays = cmdg.ArraysGrid(N, vgeo.cpu().numpy(), (g.partner + 1).cpu().numpy(), wall.cpu().numpy())
        dg = cmdg.DGModel(law, arrays, precision=precision)
        phi, dphi, rho, rhoe, p = _reference(case, g)
        dg.set_reference(torch.stack([phi, *dphi, rho, rhoe, p], 1).cpu().numpy())
        return dg
    grid = cmdg.BrickGrid(N, ne, lo, hi, periodicity=(True, True, False), boundary=((0, 0), (0, 0), (1, 2)))
    return cmdg.DGModel(law, grid, precision=precision)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _coordinates(case):
    """Node coordinates (3, nelem, Np)."""
    N = case["N"]
    xi = torch.tensor(_lgl(N)[0], device=_device())
    a, b = (1 - xi) / 2, (1 + xi) / 2
    c = _corners(case)  # (8, 3, nelem): lower, upper in xi1, then xi2, then xi3

    def blend(lo, hi, shape):
        return lo * a.view(shape) + hi * b.view(shape)

    c = c.reshape(2, 2, 2, 3, -1, 1, 1, 1)
    x = blend(c[:, :, 0], c[:, :, 1], (1, 1, -1))  # corner axes are (xi3, xi2, xi1)
    x = blend(x[:, 0], x[:, 1], (1, -1, 1))
    x = blend(x[0], x[1], (-1, 1, 1))
    return _warp(case, x.reshape(3, x.shape[1], -1))


def _corners(case):
    dev = _device()
    if _is_shell(case):
        Ne, nv = case["nhorz"], case["nvert"]
        vert, _, _ = _shell_base(Ne)
        flat = torch.tensor((2.0 * vert - Ne) / Ne, device=dev)  # (base, 4, 3) on the cube
        r = RADIUS + _lid(case) * torch.arange(nv + 1, device=dev, dtype=torch.float64) / nv
        c = flat.permute(1, 2, 0)[None, :, :, :, None] * torch.stack([r[:-1], r[1:]])[:, None, None, None, :]
        return c.reshape(8, 3, -1)
    ix = _cells(case)
    lo, hi = _box(case)
    out = []
    for v in range(8):
        out.append(torch.stack([lo[d] + (hi[d] - lo[d]) * (ix[d] + ((v >> d) & 1)).double() / n
                                for d, n in enumerate((case["nx"], case["ny"], case["nz"]))]))
    return torch.stack(out)


def _cells(case):
    """(ix, iy, iz) of every element: columns contiguous on generated bricks,
    ix fastest on the arrays a program hands over."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    e = torch.arange(nx * ny * nz, device=_device())
    if case["kind"] == "terrain":
        return e % nx, (e // nx) % ny, e // (nx * ny)
    return (e // nz) % nx, e // (nz * nx), e % nz


def _warp(case, x):
    if case["kind"] == "terrain":
        k = 2 * math.pi / BOX
        hill = 120.0 * torch.sin(k * x[0]) * torch.cos(k * x[1])
        return torch.stack([x[0], x[1], x[2] + hill * (1 - x[2] / BOX)])
    if not _is_shell(case):
        return x
    # equiangular cubed sphere: the face is the coordinate of largest magnitude
    R = x.abs().amax(0)
    out = torch.zeros_like(x)
    face = x.mean(-1, keepdim=True).abs().argmax(0).expand(x.shape[1:])  # one face per element
    for d in range(3):
        p, q = [c for c in range(3) if c != d]
        X, Y = torch.tan(math.pi / 4 * x[p] / x[d]), torch.tan(math.pi / 4 * x[q] / x[d])
        z = torch.sign(x[d]) * R / torch.sqrt(1 + X * X + Y * Y)
        for c, v in ((d, z), (p, X * z), (q, Y * z)):
            out[c] = torch.where(face == d, v, out[c])
    return out


def _shell_base(Ne):
    """Base elements of the cubed shell: lattice vertices (base, 4, 3) and the
    neighbour element and face across each of the four horizontal faces."""
    h = np.arange(6 * Ne * Ne)
    i, j, blk = h % Ne + 1, (h // Ne) % Ne + 1, h // (Ne * Ne)
    vert = np.empty((h.size, 4, 3))
    for n in range(4):
        a, b, one, top = i + n % 2, j + n // 2, np.ones_like(i), np.full_like(i, Ne + 1)
        nets = [(one, Ne + 2 - a, b), (a, one, b), (top, a, b), (a, b, top), (a, top, Ne + 2 - b), (a, Ne + 2 - b, one)]
        for k, v in enumerate(nets):
            vert[blk == k, n] = np.stack(v, -1)[blk == k]
    vert -= 1
    ids = (vert @ np.array([1, Ne + 1, (Ne + 1) ** 2])).astype(np.int64)
    edges, nb, nf = {}, np.empty((h.size, 4), np.int64), np.empty((h.size, 4), np.int64)
    for f, (a, b) in enumerate(((0, 2), (1, 3), (0, 1), (2, 3))):
        for e in range(h.size):
            key = (min(ids[e, a], ids[e, b]), max(ids[e, a], ids[e, b]))
            if key in edges:
                e2, f2 = edges[key]
                nb[e, f], nf[e, f], nb[e2, f2], nf[e2, f2] = e2, f2, e, f
            else:
                edges[key] = (e, f)
    return vert, nb, nf


def _initial(case, x, seed):
    """FP64 state (nelem, 5, Np) at the nodes x."""
    r = random.Random(seed)
    kind = case["kind"]
    if kind == "vortex":
        # the isentropic vortex of the reference's Euler test with seeded noise
        p_inf, T_inf, speed, Rv = 1e5, 300.0, 50.0, 0.005
        ang = r.uniform(0, 2 * math.pi)
        cx, cy = r.uniform(-0.01, 0.01), r.uniform(-0.01, 0.01)
        X, Y = x[0] - cx, x[1] - cy
        g = torch.exp(-(X * X + Y * Y) / Rv**2 / 2)
        u = torch.stack([150 * math.cos(ang) - speed * Y / Rv * g, 150 * math.sin(ang) + speed * X / Rv * g, 0 * g])
        rho_inf = p_inf / (R_D * T_inf)
        T = T_inf * (1 - R_D / CP_D * speed**2 / 2 * rho_inf / p_inf * g * g)
        rho = p_inf * (T / T_inf) ** (CP_D / R_D) / (R_D * T)
        phi = 0.0
    elif kind in ("gcm", "hevi"):
        rad = x.square().sum(0).sqrt()
        lat, lon = torch.asin(x[2] / rad), torch.atan2(x[1], x[0])
        phi = GRAV * (rad - RADIUS)
        T_ref = _profile(case)[1]
        z = phi / GRAV
        p = MSLP * torch.exp(-z * GRAV / (R_D * T_ref))
        lat0, lon0 = r.uniform(-1, 1), r.uniform(-3, 3)
        dist = torch.arccos((torch.sin(lat) * math.sin(lat0)
                             + torch.cos(lat) * math.cos(lat0) * torch.cos(lon - lon0)).clamp(-1, 1))
        if kind == "gcm":
            T = T_ref + torch.exp(-((RADIUS * dist / 1e6) ** 2) - ((z - LID / 3) / 5e3) ** 2)
            speed = r.uniform(15, 30)
        else:
            beta = (3 * dist).clamp(max=1.0)
            p = p + 100.0 * (1 + torch.cos(math.pi * beta)) / 2 * torch.sin(math.pi * z / WAVE_LID)
            T = torch.full_like(p, T_ref)
            speed = r.uniform(1, 5)
        k, ph = r.randint(1, 3), r.uniform(0, 2 * math.pi)
        u = speed * torch.cos(lat) * (1 + torch.sin(k * lon + ph)) / 2
        u = torch.stack([-torch.sin(lon) * u, torch.cos(lon) * u, 0 * u])
        rho = p / (R_D * T)
    else:
        z = x[2]
        phi = GRAV * z
        lo, hi = _box(case)
        if kind == "les":
            S = 1e-4 / GRAV  # stable stratification, N = 0.01 / s
            th = 300.0 * torch.exp(S * z)
            ex = 1 + GRAV / (CP_D * 300.0 * S) * (torch.exp(-S * z) - 1)
            speed, modes = 1.0, 12
        else:
            amp, rc = r.uniform(0.5, 3), r.uniform(150, 400)
            c = (r.uniform(0.4, 0.6) * BOX, r.uniform(0.4, 0.6) * BOX, 350.0 + (rc if kind == "terrain" else 0))
            d = sum((x[i] - c[i]) ** 2 for i in range(3)).sqrt()
            th = 300.0 + torch.where(d <= rc, amp * torch.cos(math.pi / 2 * d / rc) ** 2, 0 * d)
            ex = 1 - GRAV / (CP_D * th) * z
            speed, modes = 0.5, 3
        rho = MSLP / (R_D * th) * ex ** (CV_D / R_D)
        T = th * ex
        # seeded eddies, periodic in x and y, with no flow through the walls
        u = torch.zeros_like(x)
        for _ in range(modes):
            kx, ky = (2 * math.pi * r.choice([-1, 1]) * r.randint(1, 5) / (hi[i] - lo[i]) for i in range(2))
            kz = math.pi * r.randint(1, 5) / (hi[2] - lo[2])
            ph, size = r.uniform(0, 2 * math.pi), r.gauss(0, 1) / math.sqrt(modes)
            s = kx * x[0] + ky * x[1] + ph
            for i, k in ((0, kx), (1, ky)):
                u[i] += -size * k * kz / (kx * kx + ky * ky) * torch.cos(s) * torch.cos(kz * z)
            u[2] += -size * torch.sin(s) * torch.sin(kz * z)
        u *= speed
    e = CV_D * (T - T_0) + u.square().sum(0) / 2 + phi
    Q = torch.stack([rho, *(rho * u), rho * e], 1)
    if kind == "vortex":
        gen = torch.Generator().manual_seed(seed)
        Q += (1e-6 * (2 * torch.rand(Q.shape, generator=gen, dtype=torch.float64) - 1)).to(Q.device)
    return Q.contiguous()


def _profile(case):
    return ("isothermal", 285.0 if case["kind"] == "gcm" else 300.0) if _is_shell(case) else ("adiabatic", 300.0)


# --------------------------------------------------------------------------
# the same calls in plain FP64
# --------------------------------------------------------------------------
def exact(case, seed):
    with torch.no_grad():
        if case["kind"] == "ensemble":
            return [_exact_step(s, seed * 131 + n) for n, s in enumerate(_member_specs(case))]
        if case["kind"] == "hevi":
            return _exact_hevi(case, seed)
        if case["kind"] == "vortex":
            g = _Grid(case)
            Q = _initial(case, g.X, seed).permute(1, 0, 2).contiguous()
            return _Law(case, g).rhs(Q).permute(1, 0, 2).contiguous()
        return _exact_step(case, seed)


# Carpenter and Kennedy's five-stage fourth-order 2N scheme
_A = (0.0, -567301805773 / 1357537059087, -2404267990393 / 2016746695238, -3550918686646 / 2091501179385,
      -1275806237668 / 842570457699)
_B = (1432997174477 / 9575080441755, 5161836677717 / 13612068292357, 1720146321549 / 2090206949498,
      3134564353537 / 4481467310338, 2277821191437 / 14882151754819)


def _exact_step(case, seed):
    g = _Grid(case)
    law = _Law(case, g)
    Q = _initial(case, g.X, seed).permute(1, 0, 2).contiguous()
    ref = torch.zeros_like(Q)
    mixed = case["precision"] == "mixed"
    if mixed:  # the call's input is the FP32 perturbation
        ref[0], ref[4] = law.rho_ref, law.rhoe_ref
        Q = ref + (Q - ref).float().double()
    dt, dQ = _dt(case), torch.zeros_like(Q)
    for a, b in zip(_A, _B):
        dQ = law.rhs(Q) + a * dQ
        Q = Q + b * dt * dQ
    return (Q - ref if mixed else Q).permute(1, 0, 2).contiguous()


def _lgl(N):
    """Legendre-Gauss-Lobatto nodes and weights."""
    leg = np.polynomial.legendre
    c = np.zeros(N + 1)
    c[N] = 1.0
    x = np.concatenate(([-1.0], np.sort(np.real(leg.legroots(leg.legder(c)))), [1.0]))
    for _ in range(3):  # Newton on P_N'
        d1, d2 = leg.legval(x[1:-1], leg.legder(c)), leg.legval(x[1:-1], leg.legder(c, 2))
        x[1:-1] -= d1 / d2
    x = (x - x[::-1]) / 2
    return x, 2.0 / (N * (N + 1) * leg.legval(x, c) ** 2)


class _Grid:
    """Hexahedral grid: metrics, facing nodes and the DG operators."""

    def __init__(self, case):
        N = case["N"]
        dev = _device()
        self.N, self.Nq = N, N + 1
        self.Np, self.Nfp = self.Nq**3, self.Nq**2
        x, w = _lgl(N)
        bary = np.array([1 / np.prod([x[j] - x[i] for i in range(N + 1) if i != j]) for j in range(N + 1)])
        with np.errstate(divide="ignore"):
            D = bary[None, :] / bary[:, None] / (x[:, None] - x[None, :])
        np.fill_diagonal(D, 0)
        np.fill_diagonal(D, -D.sum(1))
        self.D = torch.tensor(D, device=dev)
        w = torch.tensor(w, device=dev)
        self.w0 = float(w[0])
        self.Dw = (self.D.T * w[None, :] / w[:, None]).contiguous()  # M^-1 D^T M on a line
        self.www = (w[:, None, None] * w[None, :, None] * w[None, None, :]).reshape(-1)
        self.X = X = _coordinates(case)
        self.nelem = X.shape[1]
        dX = [[self.d(X[c], r) for r in range(3)] for c in range(3)]  # dX[c][r] = dx_c / dxi_r
        self.J = (dX[0][0] * (dX[1][1] * dX[2][2] - dX[2][1] * dX[1][2])
                  + dX[1][0] * (dX[2][1] * dX[0][2] - dX[0][1] * dX[2][2])
                  + dX[2][0] * (dX[0][1] * dX[1][2] - dX[1][1] * dX[0][2]))
        # curl-invariant metric terms: J dxi_r/dx_c = curl_r of (x_m grad x_n - x_n grad x_m) / 2
        self.Jxi = [[None] * 3 for _ in range(3)]
        for c in range(3):
            m, n = (c + 1) % 3, (c + 2) % 3
            v = [X[m] * dX[n][r] - X[n] * dX[m][r] for r in range(3)]
            for r in range(3):
                a, b = (r + 1) % 3, (r + 2) % 3
                self.Jxi[r][c] = (self.d(v[b], a) - self.d(v[a], b)) / 2
        self.xi = [[t / self.J for t in row] for row in self.Jxi]
        n = torch.arange(self.Np, device=dev).reshape(self.Nq, self.Nq, self.Nq)
        self.fm = [t.reshape(-1) for t in (n[:, :, 0], n[:, :, N], n[:, 0], n[:, N], n[0], n[N])]
        self._connect(case)
        self.nrm, self.lift = [], []
        for f in range(6):
            v = [(1 if f % 2 else -1) * self.Jxi[f // 2][c][:, self.fm[f]] for c in range(3)]
            s = (v[0] ** 2 + v[1] ** 2 + v[2] ** 2).sqrt()
            self.nrm.append([c / s for c in v])
            self.lift.append(s / (self.J[:, self.fm[f]] * self.w0))

    def _connect(self, case):
        dev = self.X.device
        ne = self.nelem
        e = torch.arange(ne, device=dev)
        nb, nf = torch.empty((ne, 6), dtype=torch.int64, device=dev), [f ^ 1 for f in range(6)]
        self.wall = torch.zeros((ne, 6), dtype=torch.bool, device=dev)
        self.partner = torch.empty((ne, 6, self.Nfp), dtype=torch.int64, device=dev)
        if _is_shell(case):
            nv = case["nvert"]
            _, bn, bf = _shell_base(case["nhorz"])
            bn, bf = torch.tensor(bn, device=dev), torch.tensor(bf, device=dev)
            h, iz = e // nv, e % nv
            nb[:, :4] = bn[h] * nv + iz[:, None]
            nb[:, 4], nb[:, 5] = e - 1, e + 1
            self.wall[:, 4], self.wall[:, 5] = iz == 0, iz == nv - 1
        else:
            ix, n = torch.stack(_cells(case)), (case["nx"], case["ny"], case["nz"])
            where = torch.empty(n, dtype=torch.int64, device=dev)
            where[ix[0], ix[1], ix[2]] = e
            for f in range(6):
                j = ix.clone()
                j[f // 2] += 1 if f % 2 else -1
                if case["kind"] != "vortex" and f // 2 == 2:
                    self.wall[:, f] = (j[2] < 0) | (j[2] >= n[2])
                j[f // 2] %= n[f // 2]
                nb[:, f] = where[j[0], j[1], j[2]]
        for f in range(6):
            self.partner[:, f] = nb[:, f, None] * self.Np + self.fm[nf[f]]
            if f < 4 and _is_shell(case):  # the face node of the neighbour at the same place
                cand = torch.stack(self.fm)[bf[h, f]]  # (nelem, Nfp)
                mine = self.X[:, :, self.fm[f]].permute(1, 2, 0)
                other = self.X[:, nb[:, f, None], cand].permute(1, 2, 0)
                near = (mine[:, :, None] - other[:, None]).square().sum(-1).argmin(-1)
                self.partner[:, f] = nb[:, f, None] * self.Np + cand.gather(1, near)
            self.partner[:, f] = torch.where(self.wall[:, f, None], e[:, None] * self.Np + self.fm[f], self.partner[:, f])

    def line(self, A, q, r):
        """A applied along xi_r to q (..., nelem, Np)."""
        v = q.reshape(*q.shape[:-1], self.Nq, self.Nq, self.Nq)
        v = torch.einsum(("...kjn,in->...kji", "...kni,jn->...kji", "...nji,kn->...kji")[r], v, A)
        return v.reshape(q.shape)

    def d(self, q, r):
        return self.line(self.D, q, r)

    def grad(self, q, dirs=(0, 1, 2)):
        """Element-local gradient, a list over x_c."""
        dq = {r: self.d(q, r) for r in dirs}
        return [sum(self.xi[r][c] * dq[r] for r in dirs) for c in range(3)]

    def weak(self, F, dirs=(0, 1, 2)):
        """M^-1 D^T M (xi . F) of a flux F[c] (..., nelem, Np)."""
        return sum(self.line(self.Dw, sum(self.Jxi[r][c] * F[c] for c in range(3)), r) for r in dirs) / self.J

    def plus(self, q, f):
        return q.reshape(*q.shape[:-2], -1)[..., self.partner[:, f].reshape(-1)].reshape(*q.shape[:-1], self.Nfp)

    def add_face(self, out, f, v):
        """out += lift v at the nodes of face f."""
        out[..., self.fm[f]] += self.lift[f] * v


def _reference(case, g):
    """Geopotential, its gradient and the hydrostatic state in discrete balance."""
    if case["kind"] == "vortex":
        return None
    phi = GRAV * ((g.X.square().sum(0).sqrt() - RADIUS) if _is_shell(case) else g.X[2])
    dphi = g.grad(phi)
    name, T = _profile(case)
    z = phi / GRAV
    if name == "isothermal":
        p = MSLP * torch.exp(-z * GRAV / (R_D * T))
    else:
        p = MSLP * ((T - GRAV / CP_D * z) / T) ** (CP_D / R_D)
    zero = torch.zeros_like(p)
    dp = torch.stack([g.weak([-p if c == s else zero for c in range(3)]) for s in range(3)])
    for f in range(6):
        mean = (p[:, g.fm[f]] + g.plus(p, f)) / 2
        for s in range(3):
            g.add_face(dp[s], f, mean * g.nrm[f][s])
    rho = -sum(a * b for a, b in zip(dphi, dp)) / sum(a * a for a in dphi)
    return phi, dphi, rho, rho * (phi + CV_D * (p / (R_D * rho) - T_0)), p


class _Law:
    """The dry AtmosModel on a grid; states are (5, nelem, Np)."""

    def __init__(self, case, g):
        self.g, self.closure = g, case.get("closure", "none")
        ref = _reference(case, g)
        self.gravity = ref is not None
        if ref is None:
            zero = torch.zeros_like(g.J)
            ref = (zero, [zero] * 3, zero, zero, zero)
        self.phi, self.dphi, self.rho_ref, self.rhoe_ref, self.p_ref = ref
        self.horizontal = _is_shell(case)
        self.tau = 8 * 3600.0 if self.horizontal else 3600.0

    def pressure(self, q, phi):
        return R_D / CV_D * (q[4] - (q[1] ** 2 + q[2] ** 2 + q[3] ** 2) / (2 * q[0]) - q[0] * phi) + R_D * T_0 * q[0]

    def flux(self, q, phi, p_ref):
        """First-order flux F[c] (5, ...), pressure and velocity."""
        p, u = self.pressure(q, phi), q[1:4] / q[0]
        F = []
        for c in range(3):
            f = torch.stack([q[1 + c], *(q[1:4] * u[c]), u[c] * (q[4] + p)])
            f[1 + c] += p - p_ref
            F.append(f)
        return F, p, u

    def rhs(self, Q):
        g = self.g
        F, p, u = self.flux(Q, self.phi, self.p_ref)
        second = self.second_order(Q, p, u)
        total = F if second is None else [a + b for a, b in zip(F, second)]
        out = g.weak(total)
        if self.gravity:
            for c in range(3):
                out[1 + c] -= (Q[0] - self.rho_ref) * self.dphi[c]
        for f in range(6):
            n, wall = g.nrm[f], g.wall[:, f, None]
            qm, qp = Q[..., g.fm[f]], g.plus(Q, f)
            mirror = qm.clone()
            un = sum(qm[1 + c] * n[c] for c in range(3))
            for c in range(3):
                mirror[1 + c] -= 2 * un * n[c]
            qp = torch.where(wall, mirror, qp)
            Fm, pm, um = self.flux(qm, self.phi[:, g.fm[f]], self.p_ref[:, g.fm[f]])
            Fp, pp, up = self.flux(qp, g.plus(self.phi, f), g.plus(self.p_ref, f))
            speed = [sum(v[c] * n[c] for c in range(3)).abs() + (CP_D / CV_D * a / q[0]).sqrt()
                     for v, a, q in ((um, pm, qm), (up, pp, qp))]
            num = sum((a + b) * (c / 2) for a, b, c in zip(Fm, Fp, n)) + torch.maximum(*speed) * (qm - qp) / 2
            if second is not None:
                both = sum((s[..., g.fm[f]] + g.plus(s, f)) * (c / 2) for s, c in zip(second, n))
                num = num + torch.where(wall, torch.zeros_like(both), both)
            g.add_face(out, f, -num)
        return out

    def arguments(self, Q, p):
        """Velocity, total specific enthalpy and, for the LES, potential temperature."""
        G = [*(Q[1:4] / Q[0]), (Q[4] + p) / Q[0]]
        if self.closure == "smagorinsky":
            G.append(p / (R_D * Q[0]) / (p / MSLP) ** (R_D / CP_D))
        return torch.stack(G)

    def dg_gradient(self, G, wall_value, dirs=(0, 1, 2)):
        """Strong gradient with central corrections; G (s, nelem, Np)."""
        g = self.g
        out = torch.stack(g.grad(G, dirs))
        for f in range(2 * len(dirs)):
            Gm = G[..., g.fm[f]]
            star = torch.where(g.wall[:, f, None], wall_value(f, Gm), (g.plus(G, f) + Gm) / 2)
            for c in range(3):
                g.add_face(out[c], f, g.nrm[f][c] * (star - Gm))
        return out

    def second_order(self, Q, p, u):
        if self.closure == "none":
            return None
        g = self.g

        def slip(f, Gm):  # the wall state without its normal velocity
            G, n = Gm.clone(), g.nrm[f]
            un = sum(Gm[c] * n[c] for c in range(3))
            for c in range(3):
                G[c] -= un * n[c]
            # h_tot and theta_v of the state that has lost that kinetic energy
            rho, pw = Q[0][:, g.fm[f]], p[:, g.fm[f]] + R_D / CV_D * Q[0][:, g.fm[f]] * un * un / 2
            G[3] = (Q[4][:, g.fm[f]] + pw) / rho
            if G.shape[0] > 4:
                G[4] = pw / (R_D * rho) / (pw / MSLP) ** (R_D / CP_D)
            return G

        G = self.arguments(Q, p)
        rho = Q[0]
        khat = [d / GRAV for d in self.dphi]
        if self.closure == "hyper":
            dirs = (0, 1) if self.horizontal else (0, 1, 2)

            def project(v):
                dot = sum(v[c] * k for c, k in enumerate(khat))
                return torch.stack([*(v[c] - khat[c] * dot for c in range(3)), v[3]])

            def wall_args(f, Hm):
                k = [c[:, g.fm[f]] for c in khat]
                v = slip(f, G[..., g.fm[f]])
                dot = sum(v[c] * k[c] for c in range(3))
                return torch.stack([*(v[c] - k[c] * dot for c in range(3)), v[3]])

            grad = self.dg_gradient(project(G), wall_args, dirs)
            lap = -g.weak(list(grad), dirs)
            for f in range(2 * len(dirs)):
                g.add_face(lap, f, sum((grad[c][..., g.fm[f]] + g.plus(grad[c], f)) * g.nrm[f][c] / 2 for c in range(3)))
            cof = [[self._cofactor(r, c) for c in range(3)] for r in range(2)]
            size = sum(sum(c * c for c in row).sqrt() for row in cof) / g.N
            nu4 = (size / 2) ** 4 / 2 / self.tau
            g3 = nu4 * self.dg_gradient(lap, lambda f, Lm: Lm, dirs)
            return [torch.stack([0 * rho, *(rho * g3[c][:3]), (g3[c][:3] * Q[1:4]).sum(0) + rho * g3[c][3]])
                    for c in range(3)]
        grad = self.dg_gradient(G, slip)  # (3, s, nelem, Np)
        S = [[(grad[a][b] + grad[b][a]) / 2 for b in range(3)] for a in range(3)]
        if self.closure == "constant":
            nu = [RHO_NU / rho] * 3
        else:
            norm = (2 * sum(S[a][b] ** 2 for a in range(3) for b in range(3))).sqrt()
            N2 = sum(grad[c][4] * self.dphi[c] for c in range(3)) / G[4]
            tiny = torch.nextafter(norm, torch.full_like(norm, math.inf)) - norm
            fb = (1 - N2 / (norm * norm + tiny) * INV_PR).clamp(0, 1).sqrt()
            det = 1 / g.J
            delta = 2 / (det ** (1 / 3) * g.N)
            nu0 = norm * (C_SMAG * delta) ** 2 + 1e-5
            along = sum(nu0 * k for k in khat)
            nu = [nu0 - k * along + k * along * fb for k in khat]
        F = []
        for d in range(3):
            tau = [-2 * nu[d] * S[d][c] for c in range(3)]
            heat = sum(t * Q[1 + c] for c, t in enumerate(tau)) - nu[d] * INV_PR * grad[d][3] * rho
            F.append(torch.stack([0 * rho, *(t * rho for t in tau), heat]))
        return F

    def _cofactor(self, r, c):
        """dx_c / dxi_r from the inverse of the metric terms."""
        x, m, n = self.g.xi, (r + 1) % 3, (r + 2) % 3
        a, b = (c + 1) % 3, (c + 2) % 3
        return (x[m][a] * x[n][b] - x[m][b] * x[n][a]) * self.g.J


class _Linear:
    """Acoustic-gravity model linearized about the reference state, vertical only."""

    def __init__(self, law):
        self.law, g = law, law.g
        self.h = (law.rhoe_ref + law.p_ref) / law.rho_ref
        self.c = (CP_D / CV_D * law.p_ref / law.rho_ref).sqrt()

    def rhs(self, Q):
        law, g = self.law, self.law.g

        def flux(q, phi, h):
            p = q[0] * R_D * T_0 + R_D / CV_D * (q[4] - q[0] * phi)
            zero = torch.zeros_like(p)
            return [torch.stack([q[1 + c], *(p if s == c else zero for s in range(3)), h * q[1 + c]]) for c in range(3)]

        out = g.weak(flux(Q, law.phi, self.h), (2,))
        for c in range(3):
            out[1 + c] -= Q[0] * law.dphi[c]
        for f in (4, 5):
            n = g.nrm[f]
            at = lambda v: v[..., g.fm[f]]  # noqa: E731
            qm, qp = at(Q), g.plus(Q, f)
            mirror = qm.clone()
            un = sum(qm[1 + c] * n[c] for c in range(3))
            for c in range(3):
                mirror[1 + c] -= 2 * un * n[c]
            qp = torch.where(g.wall[:, f, None], mirror, qp)
            Fm, Fp = flux(qm, at(law.phi), at(self.h)), flux(qp, g.plus(law.phi, f), g.plus(self.h, f))
            num = sum((a + b) * (c / 2) for a, b, c in zip(Fm, Fp, n))
            num = num + torch.maximum(at(self.c), g.plus(self.c, f)) * (qm - qp) / 2
            g.add_face(out, f, -num)
        return out


def _exact_hevi(case, seed):
    """An ARK2 step (low-storage form) and the vertical exponential filter."""
    g = _Grid(case)
    law = _Law(case, g)
    lin = _Linear(law)
    nv, Nq, Nfp = case["nvert"], g.Nq, g.Nfp
    n = 5 * Nq * nv

    def to_lines(q):  # (5, nelem, Np) -> (columns Nfp, n)
        return q.reshape(5, -1, nv, Nq, Nfp).permute(1, 4, 2, 3, 0).reshape(-1, n)

    def from_lines(b):
        return b.reshape(-1, Nfp, nv, Nq, 5).permute(4, 0, 2, 3, 1).reshape(5, g.nelem, g.Np)

    dt, s2, a32 = _dt(case), math.sqrt(2.0), 0.5
    al = dt * (1 - 1 / s2)
    lines = g.nelem // nv * Nfp
    A = torch.empty((lines, n, n), dtype=torch.float64, device=g.X.device)
    unit = torch.zeros((lines, n), dtype=torch.float64, device=g.X.device)
    for c in range(n):
        unit[:, c] = 1
        A[:, :, c] = unit - al * to_lines(lin.rhs(from_lines(unit)))
        unit[:, c] = 0
    # elimination by blocks of one element, which couple only to the next
    m = 5 * Nq
    blk = lambda r, c: A[:, r * m:(r + 1) * m, c * m:(c + 1) * m]  # noqa: E731
    for v in range(1, nv):
        W = torch.linalg.solve(blk(v - 1, v - 1), blk(v, v - 1), left=False)
        blk(v, v).sub_(W @ blk(v - 1, v))
        blk(v, v - 1).copy_(W)

    def solve(q):
        b = to_lines(q).clone()
        part = lambda v: b[:, v * m:(v + 1) * m]  # noqa: E731
        for v in range(1, nv):
            part(v).sub_((blk(v, v - 1) @ part(v - 1)[..., None])[..., 0])
        for v in reversed(range(nv)):
            if v + 1 < nv:
                part(v).sub_((blk(v, v + 1) @ part(v + 1)[..., None])[..., 0])
            part(v).copy_(torch.linalg.solve(blk(v, v), part(v)))
        return from_lines(b)

    Ae = ((), (2 - s2,), (1 - a32, a32))
    Ai = ((), (1 - 1 / s2,), (1 / (2 * s2), 1 / (2 * s2)))
    Bc = (1 / (2 * s2), 1 / (2 * s2), 1 - 1 / s2)
    aii = 1 - 1 / s2
    Q = _initial(case, g.X, seed).permute(1, 0, 2).contiguous()
    S, R = [Q], [law.rhs(Q)]
    for i in (1, 2):
        rk = [(Ai[i][j] - Ae[i][j]) / aii for j in range(i)]
        common = sum(rk[j] * S[j] for j in range(i))
        S.append(solve(Q + common + dt * sum(Ae[i][j] * R[j] for j in range(i))) - common)
        R.append(law.rhs(S[i]))
    Q = Q + dt * sum(b * r for b, r in zip(Bc, R))
    x = _lgl(g.N)[0]
    V = np.polynomial.legendre.legvander(x, g.N)
    sig = np.exp(math.log(np.finfo(np.float64).eps) * (np.arange(g.N + 1) / g.N) ** 18)
    W = torch.tensor(V @ np.diag(sig) @ np.linalg.inv(V), device=Q.device)
    return g.line(W, Q, 2).permute(1, 0, 2).contiguous()
