"""The work that programs built on this framework have it do, as cases that can be timed and checked.

A case is a dict of plain values. `prepare` makes what a program holds before the call (the mesh's
context, the state, the time step), `run` is one call of the public entry points, `work` what that
call cannot do without, and `exact` the same result in 64 bits from plain torch.

Fields of a case:
  do         "step"      SSP-RK3 steps of the device-resident state
             "field"     the same, then the field in single precision: what a program takes out of a
                         mixed-precision solve (whose fluxes are FP32) for output or coupling
             "adaptive"  the drivers' loop body: CFL time step from the state's wave speed, then the step
             "monitored" one step, then the conservation sums (the kinetic energy history of a flow)
             "residual"  the operator on device buffers, as another solver's time loop calls it
             "host"      the operator on host arrays, the drop-in for ExplicitConvection::eval
  order, qv, qf, flux, precision, schedule, limiter, mu: the context's options (qv, qf: -1 = Auto rules)
  steps      steps of one call
  graph      replay the step as a CUDA graph
  problem    "vortex", "dwave" (density wave), "thin" (a density wave near vacuum), "tgv" (Taylor-Green)
  n          cubes per side (6 n^3 tetrahedra); "sizes" instead lists the instances of an ensemble
  jitter     displacement of the interior vertices over the cell size
  walls      "" periodic, "z" Pseudo3DZ faces across z, "box" Dirichlet data on the whole boundary
  part       of a residual: 0 all, 1 volume, 2 interior faces, 3 boundary faces
"""
import functools
import math
import random

import numpy as np
import torch

from fve_dg_b200 import Ensemble, ExplicitConvection, box_mesh, problems
from fve_dg_b200 import _lib as abi

GAMMA = 1.4
PRANDTL = 0.71
CFL = 0.3
SIDE = {"vortex": 10.0, "dwave": 1.0, "thin": 1.0, "tgv": 2.0 * math.pi}
CONFIG_RULES = {1: (0, 1), 2: (1, 2), 3: (3, 3), 4: (5, 3)}
F64 = torch.float64


def _case(name, do, order, problem, n, **more):
    qv, qf = CONFIG_RULES[order] if more.pop("rules", "config") == "config" else (-1, -1)
    c = dict(name=name, do=do, order=order, qv=qv, qf=qf, flux="LF", precision="fp64", schedule="two-launch",
             limiter="none", mu=0.0, steps=1, graph=True, problem=problem, n=n, sizes="", jitter=0.0, walls="", part=0)
    c.update(more)
    return c


def listed():
    return [
        # The smallest solve: 3,072 tets, where a step is six short launches and their latency.
        _case("vortex_p1_step", "step", 1, "vortex", 8),
        # A single evaluation on a small ragged mesh with walls, inside another program's time loop.
        _case("walls_p2_residual", "residual", 2, "dwave", 13, rules="auto", flux="Roe", jitter=0.1, walls="z"),
        # The drop-in for a CPU driver: host state in, host residual out, Dirichlet data all round.
        _case("box_p3_host", "host", 3, "dwave", 15, rules="auto", jitter=0.1, walls="box"),
        # The smooth density wave run, mixed precision.
        _case("dwave_p2_field_mixed", "field", 2, "dwave", 32, precision="mixed", steps=4, jitter=0.1),
        # The headline flow and size: Taylor-Green at Mach 0.1, P3, Roe, 663,552 tets, mixed precision.
        _case("tgv_p3_field_mixed", "field", 3, "tgv", 48, precision="mixed", flux="Roe", steps=4),
        # The same flow in FP64 with the time step from the wave speed of every state.
        _case("tgv_p3_adaptive", "adaptive", 3, "tgv", 36, flux="Roe", graph=False),
        # High order, mixed precision.
        _case("dwave_p4_field_mixed", "field", 4, "dwave", 25, precision="mixed", steps=4, jitter=0.1),
        # High order, FP64, with the Auto rules (the largest of both kinds up to P4).
        _case("dwave_p4_step", "step", 4, "dwave", 20, rules="auto", jitter=0.1),
        # An ensemble of vortices on uneven meshes, one persistent launch per stage.
        _case("vortex_p2_ensemble", "field", 2, "vortex", 0, sizes="8,9,11,12,14,15,17,20,22,24",
              precision="mixed", schedule="persistent", steps=4),
        # Navier-Stokes: Taylor-Green at Re 1600 with its kinetic energy followed.
        _case("tgv_p3_navier_stokes", "monitored", 3, "tgv", 24, flux="Roe", mu=0.000625),
        # A flow near vacuum, limited after every stage.
        _case("thin_p2_limited", "step", 2, "thin", 26, limiter="positive", jitter=0.1),
        # The highest order the operator has.
        _case("wave_p5_residual", "residual", 5, "dwave", 11, rules="auto", jitter=0.1),
    ]


# The most cubes per side that a drawn case of an order takes, by what it does.
_MOST = {0: 40, 1: 48, 2: 44, 3: 40, 4: 26, 5: 11}


def draw(rng):
    def size(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(["step", "field", "field", "adaptive", "residual", "residual", "host", "ensemble", "viscous", "limited"])
    jitter = rng.choice([0.0, 0.05, 0.1])
    flux = rng.choice(["LF", "Roe"])
    if kind in ("residual", "host"):
        order = rng.choice([0, 1, 2, 2, 3, 3, 4, 5])
        rules = "config" if order in CONFIG_RULES and rng.random() < 0.5 else "auto"
        top = _MOST[order] if kind == "residual" else min(_MOST[order], 18)
        walls = rng.choice(["", "z", "box"])
        problem = "dwave" if walls == "box" else rng.choice(["vortex", "dwave"])
        c = _case("", kind, order, problem, size(5, top), rules=rules, flux=flux, jitter=jitter, walls=walls,
                  part=rng.choice([0, 0, 0, 1, 2]) if kind == "residual" else 0)
    elif kind == "ensemble":
        c = _case("", "field", 2, "vortex", 0, flux=flux, precision="mixed", schedule="persistent", steps=rng.choice([2, 4]),
                  sizes=",".join(str(rng.randint(8, 24)) for _ in range(rng.randint(3, 10))))
    elif kind == "viscous":
        order = rng.choice([1, 2, 3, 3])
        c = _case("", "monitored", order, "tgv", size(6, 24), flux=flux, jitter=jitter,
                  mu=10.0 ** rng.uniform(-4.0, -2.0))
    elif kind == "limited":
        order = rng.choice([1, 2, 3])
        c = _case("", "step", order, "thin", size(8, 28), flux=flux, jitter=jitter,
                  limiter=rng.choice(["positive", "positive-avg"]))
    else:
        order = rng.choice([1, 2, 3, 3, 4])
        mixed = kind == "field"
        c = _case("", kind, order, rng.choice(["dwave", "tgv"]), size(6, _MOST[order]), flux=flux,
                  rules=rng.choice(["config", "auto"]), precision="mixed" if mixed else "fp64",
                  jitter=jitter, steps=rng.choice([2, 4]) if mixed else 1,
                  graph=kind != "adaptive" and rng.random() < 0.7)
    del c["name"]
    return c


# ---- what a program holds before the call ---------------------------------------------------------

@functools.lru_cache(maxsize=4)
def _mesh(n, side, jitter, walls):
    periodic = {"": (1, 1, 1), "z": (1, 1, 0), "box": (0, 0, 0)}[walls]
    return box_mesh(n, hi=(side,) * 3, jitter=jitter, seed=20261203 + n, periodic=periodic,
                    bc="Dirichlet" if walls == "box" else "Pseudo3DZ")


def _sizes(case):
    return [int(s) for s in case["sizes"].split(",")] if case["sizes"] else [case["n"]]


def _meshes(case):
    return [_mesh(n, SIDE[case["problem"]], case["jitter"], case["walls"]) for n in _sizes(case)]


def _conserved(rho, u, v, w, p):
    return torch.stack([rho, rho * u, rho * v, rho * w, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v + w * w)], dim=-1)


def _flow(case, seed, instance):
    """The initial flow as a function of points (..., 3): the case's problem with the seed's parameters."""
    r = random.Random(1000003 * int(seed) + instance)
    name = case["problem"]
    if name == "vortex":
        side = SIDE[name]
        beta = r.uniform(1.0, 5.0)
        centre = torch.tensor([r.uniform(0.0, side) for _ in range(3)], dtype=F64)
        axis = torch.tensor([r.gauss(0.0, 1.0) for _ in range(3)], dtype=F64)
        axis = axis / axis.norm()

        def f(X):
            c, a = centre.to(X.device), axis.to(X.device)
            d = X - c
            d = d - side * torch.round(d / side)
            d = d - (d @ a)[..., None] * a
            r2 = (d * d).sum(-1)
            vel = torch.cross(a.expand_as(d), d, dim=-1) * (beta / (2.0 * math.pi) * torch.exp(0.5 * (1.0 - r2)))[..., None]
            T = 1.0 - (GAMMA - 1.0) * beta * beta / (8.0 * GAMMA * math.pi ** 2) * torch.exp(1.0 - r2)
            rho = T ** (1.0 / (GAMMA - 1.0))
            return _conserved(rho, 1.0 + vel[..., 0], 1.0 + vel[..., 1], vel[..., 2], rho ** GAMMA)
        return f
    if name in ("dwave", "thin"):
        thin = name == "thin"
        amp = r.uniform(0.75, 0.85) if thin else r.uniform(0.1, 0.3)
        phase = r.uniform(0.0, 2.0 * math.pi)
        vel = (2.0, 1.0, 0.5) if thin else (1.0, 0.5, 0.25)
        p = 0.01 if thin else 1.0

        def f(X):
            rho = 1.0 + amp * torch.sin(2.0 * math.pi * X.sum(-1) + phase)
            one = torch.ones_like(rho)
            return _conserved(rho, vel[0] * one, vel[1] * one, vel[2] * one, p * one)
        return f
    shift = [r.uniform(0.0, 2.0 * math.pi) for _ in range(3)]
    p0 = 1.0 / (GAMMA * 0.1 ** 2)

    def f(X):
        x, y, z = X[..., 0] + shift[0], X[..., 1] + shift[1], X[..., 2] + shift[2]
        u = torch.sin(x) * torch.cos(y) * torch.cos(z)
        v = -torch.cos(x) * torch.sin(y) * torch.cos(z)
        p = p0 + (torch.cos(2 * x) + torch.cos(2 * y)) * (torch.cos(2 * z) + 2.0) / 16.0
        return _conserved(torch.ones_like(u), u, v, torch.zeros_like(u), p)
    return f


def _rules(case):
    auto = problems.auto_rules(case["order"])
    return (auto[0] if case["qv"] < 0 else case["qv"], auto[1] if case["qf"] < 0 else case["qf"])


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _project(case, m, f):
    """L2 projection of the flow onto the basis at the volume rule's points, on the GPU."""
    pts, w = (torch.from_numpy(a).to(_device()) for a in problems.quad_rule(0, _rules(case)[0]))
    phi = _basis(case["order"], pts)[0]
    P = torch.from_numpy(m.points).to(_device())[torch.from_numpy(m.cells).to(_device())]
    lam = torch.cat([1.0 - pts.sum(1, keepdim=True), pts], dim=1)
    to = phi * w[:, None] / (phi * phi * w[:, None]).sum(0)
    return torch.cat([torch.einsum("egk,gb->ebk", f(torch.einsum("ga,ead->egd", lam, part)), to).reshape(part.shape[0], -1)
                      for part in P.split(100_000)])


def _boundary_data(case, m, f):
    """U_D at every face point, (nface, nqf, 5)."""
    uv, _ = problems.quad_rule(1, _rules(case)[1])
    uv = torch.from_numpy(uv).to(_device())
    X = torch.from_numpy(m.points).to(_device())[torch.from_numpy(m.faces).to(_device())]
    return f(torch.einsum("ga,fad->fgd", torch.cat([1.0 - uv.sum(1, keepdim=True), uv], dim=1), X))


def _wave_speed(case, U):
    """Largest |u| + c over the volume points, the time step's lambda."""
    pts, _ = problems.quad_rule(0, _rules(case)[0])
    V = torch.einsum("gb,ebk->egk", _basis(case["order"], torch.from_numpy(pts).to(U.device))[0],
                     U.view(U.shape[0], -1, 5))
    u = V[..., 1:4] / V[..., :1]
    p = (GAMMA - 1.0) * (V[..., 4] - 0.5 * V[..., 0] * (u * u).sum(-1))
    return float(((u * u).sum(-1).sqrt() + (GAMMA * p / V[..., 0]).sqrt()).max())


def _dt(case, n, lam):
    return problems.cfl_dt(CFL, SIDE[case["problem"]] / n, case["order"], lam)


class _Buffer:
    """The context's device-resident state for torch; keeps the context alive as long as a view of it is."""

    def __init__(self, conv):
        self.conv = conv
        ptr = abi.lib().dg_state_device(conv._ctx, 0)
        self.__cuda_array_interface__ = {"shape": conv.shape, "typestr": "<f8", "data": (ptr, False), "version": 3}


def prepare(case, seed):
    meshes = _meshes(case)
    flows = [_flow(case, seed, i) for i in range(len(meshes))]
    U = [_project(case, m, f) for m, f in zip(meshes, flows)]
    kw = dict(order=case["order"], flux=case["flux"], quad_vol=case["qv"], quad_face=case["qf"], gamma=GAMMA,
              precision=case["precision"], schedule=case["schedule"], limiter=case["limiter"], mu=case["mu"],
              prandtl=PRANDTL)
    conv = Ensemble(meshes, **kw) if case["sizes"] else ExplicitConvection(meshes[0], **kw)
    if case["walls"] == "box":
        conv.set_dirichlet(_boundary_data(case, meshes[0], flows[0]).cpu().numpy())
    state = dict(case=case, conv=conv)
    if case["do"] == "residual":
        state["U"] = U[0]
        state["R"] = torch.empty_like(U[0])
    elif case["do"] == "host":
        state["U"] = U[0].cpu().numpy()
    else:
        dt = [_dt(case, n, _wave_speed(case, u)) for n, u in zip(_sizes(case), U)]
        state["dt"] = np.array(dt) if case["sizes"] else dt[0]
        conv.set_state(torch.cat(U).cpu().numpy())
        state["out"] = torch.as_tensor(_Buffer(conv), device="cuda")
    return state


def run(state):
    case, conv = state["case"], state["conv"]
    if case["do"] == "residual":
        conv.eval_device(state["U"].data_ptr(), state["R"].data_ptr(), part=case["part"],
                         stream=torch.cuda.current_stream().cuda_stream)
        return state["R"]
    if case["do"] == "host":
        return conv.eval(state["U"])
    if case["do"] == "adaptive":
        dt = _dt(case, case["n"], conv.max_wave_speed())
        conv.ssprk3(dt, 1, graph=case["graph"])
        return state["out"], dt
    conv.ssprk3(state["dt"], case["steps"], graph=case["graph"])
    if case["do"] == "field":
        return state["out"].to(torch.float32)
    if case["do"] == "monitored":
        return state["out"], conv.conservation()
    return state["out"]


def work(case):
    order = case["order"]
    nb = problems.num_basis(order)
    qv, qf = _rules(case)
    nqv, nqf = problems.quad_rule(0, qv)[1].size, problems.quad_rule(1, qf)[1].size
    cells = sum(6 * n ** 3 for n in _sizes(case))
    sides = 4 * cells  # a face is shared by two cells
    faces = sides // 2
    volume = cells * (2 * 5 * nqv * nb * 4 + 100 * nqv)        # values, flux, integral against three gradients
    surface = sides * (2 * 5 * nqf * nb * 2) + faces * 150 * nqf  # traces, numerical flux, integral
    if case["do"] == "residual":
        volume *= case["part"] in (0, 1)
        surface *= case["part"] in (0, 2)
    flops = volume + surface
    if case["mu"] > 0.0:  # values and gradients, the viscous flux, both integrals
        flops += cells * (2 * 5 * nqv * nb * 7 + 250 * nqv) + sides * (2 * 5 * nqf * nb * 5) + faces * 300 * nqf
    if case["limiter"] != "none":
        flops += cells * 2 * 5 * nqv * nb
    moved = 2 * 8 * 5 * nb * cells + 80 * cells + 42 * faces
    if case["do"] in ("residual", "host"):
        return {"bytes": moved, "flops": flops}
    field = 4 * 5 * nb * cells if case["do"] == "field" else 0
    return {"bytes": case["steps"] * moved + field, "flops": 3 * case["steps"] * flops}


# ---- the same results in 64 bits, from plain torch ------------------------------------------------

def _jacobi(n, a, y, s):
    """s^n P_n^(a,0)(2 y / s - 1) by the sum over powers of y - s and y."""
    return sum((math.comb(n + a, n - m) * math.comb(n, m)) * (y - s) ** m * y ** (n - m) for m in range(n + 1))


def _basis(order, pts):
    """Values (npts, nb) and reference gradients (npts, nb, 3) of the modal basis on the unit tetrahedron."""
    X = pts.detach().clone().requires_grad_(True)
    phi, grad = [], []
    with torch.enable_grad():
        x, y, z = X[:, 0], X[:, 1], X[:, 2]
        for d in range(order + 1):
            for r in range(d + 1):
                for q in range(d - r + 1):
                    v = (_jacobi(d - q - r, 2 * (q + r) + 2, x, torch.ones_like(x))
                         * _jacobi(q, 2 * r + 1, y, 1.0 - x) * _jacobi(r, 0, z, 1.0 - x - y))
                    v = v + 0.0 * X.sum(1)
                    grad.append(torch.autograd.grad(v.sum(), X, retain_graph=True)[0])
                    phi.append(v.detach())
    return torch.stack(phi, 1), torch.stack(grad, 1)


def _flux(U):
    """Physical flux (..., 5, 3) with pressure (...)."""
    rho = U[..., 0].clamp_min(1e-16)
    u = U[..., 1:4] / rho[..., None]
    p = (GAMMA - 1.0) * (U[..., 4] - 0.5 * rho * (u * u).sum(-1))
    F = torch.empty(U.shape + (3,), dtype=U.dtype, device=U.device)
    F[..., 0, :] = rho[..., None] * u
    F[..., 1:4, :] = rho[..., None, None] * u[..., :, None] * u[..., None, :]
    for i in range(3):
        F[..., 1 + i, i] += p
    F[..., 4, :] = u * (U[..., 4] + p)[..., None]
    return F, rho, u, p


def _lax_friedrichs(UL, UR, n):
    FL, rL, uL, pL = _flux(UL)
    FR, rR, uR, pR = _flux(UR)
    sL = (uL * uL).sum(-1).sqrt() + (GAMMA * (pL / rL).clamp_min(1e-16)).sqrt()
    sR = (uR * uR).sum(-1).sqrt() + (GAMMA * (pR / rR).clamp_min(1e-16)).sqrt()
    lam = torch.maximum(sL, sR)[..., None]
    return 0.5 * (((FL + FR) * n[..., None, :]).sum(-1) + lam * (UL - UR))


def _roe(UL, UR, n):
    """Roe's flux: the five waves of the averaged state, Harten's fix with 0.1 c on the acoustic ones."""
    FL, rL, uL, pL = _flux(UL)
    FR, rR, uR, pR = _flux(UR)
    sL, sR = rL.sqrt(), rR.sqrt()
    u = (sL[..., None] * uL + sR[..., None] * uR) / (sL + sR)[..., None]
    H = (sL * (UL[..., 4] + pL) / rL + sR * (UR[..., 4] + pR) / rR) / (sL + sR)
    q2 = (u * u).sum(-1)
    c2 = ((GAMMA - 1.0) * (H - 0.5 * q2)).clamp_min(1e-16)
    c = c2.sqrt()
    un = (u * n).sum(-1)
    du, dr, dp, r = uR - uL, rR - rL, pR - pL, sL * sR
    dun = (du * n).sum(-1)

    def fixed(lam):
        lam, d = lam.abs(), 0.1 * c
        return torch.where(lam < d, (lam * lam + d * d) / (2.0 * d), lam)

    w1 = fixed(un - c) * (dp - r * c * dun) / (2.0 * c2)
    w5 = fixed(un + c) * (dp + r * c * dun) / (2.0 * c2)
    w2 = un.abs() * (dr - dp / c2)
    shear = (un.abs() * r)[..., None] * (du - dun[..., None] * n)
    D = torch.empty_like(UL)
    D[..., 0] = w1 + w5 + w2
    D[..., 1:4] = (w1[..., None] * (u - c[..., None] * n) + w5[..., None] * (u + c[..., None] * n)
                   + w2[..., None] * u + shear)
    D[..., 4] = w1 * (H - c * un) + w5 * (H + c * un) + 0.5 * w2 * q2 + (u * shear).sum(-1)
    return 0.5 * (((FL + FR) * n[..., None, :]).sum(-1) - D)


class _Operator:
    """The discontinuous Galerkin operators of one mesh, order and pair of rules."""

    def __init__(self, case, m, f):
        dev = _device()
        self.case, self.m = case, m
        order = case["order"]
        qv, qf = _rules(case)
        pts, self.wv = (torch.from_numpy(a).to(dev) for a in problems.quad_rule(0, qv))
        uv, self.wf = (torch.from_numpy(a).to(dev) for a in problems.quad_rule(1, qf))
        self.phi, self.dphi = _basis(order, pts)
        self.nb = self.phi.shape[1]
        P = torch.from_numpy(m.points).to(dev)
        cells, faces = (torch.from_numpy(a).to(dev) for a in (m.cells, m.faces))
        fc = torch.from_numpy(m.face_cells).to(dev)
        self.c0, self.c1 = fc[:, 0], fc[:, 1]
        self.inner = self.c1 >= 0
        X = P[cells]
        E = X[:, 1:] - X[:, :1]              # rows: edges from vertex 0
        self.detj = torch.linalg.det(E).abs()
        self.J = torch.linalg.inv(E)         # physical = J times reference gradients
        T = P[faces]
        cr = torch.cross(T[:, 1] - T[:, 0], T[:, 2] - T[:, 0], dim=-1)
        out = T.mean(1) - X[self.c0].mean(1)  # away from the first cell
        cr = torch.where(((cr * out).sum(-1) < 0)[:, None], -cr, cr)
        self.twice = cr.norm(dim=-1)
        self.n = cr / self.twice[:, None]
        fn1 = faces if m.face_nodes1 is None else torch.from_numpy(m.face_nodes1).to(dev)
        lam = torch.cat([1.0 - uv.sum(1, keepdim=True), uv], dim=1)
        corner = torch.cat([torch.zeros(1, 3, dtype=F64, device=dev), torch.eye(3, dtype=F64, device=dev)])
        self.sides = []                      # per side: (faces, their cells, phi, dphi) of each face map
        for side, (cell, nodes) in enumerate(((self.c0, faces), (self.c1, fn1))):
            slot = (cells[cell.clamp_min(0)][:, None, :] == nodes[:, :, None]).to(torch.int64).argmax(-1)
            code = slot[:, 0] * 16 + slot[:, 1] * 4 + slot[:, 2]
            code = torch.where(cell >= 0, code, torch.full_like(code, -1))
            maps = []
            for k in torch.unique(code).tolist():
                if k < 0:
                    continue
                at = torch.nonzero(code == k).ravel()
                ref = lam @ corner[torch.tensor([k // 16, k // 4 % 4, k % 4], device=dev)]
                maps.append((at, cell[at]) + _basis(order, ref))
            self.sides.append(maps)
        bc = torch.from_numpy(m.bc).to(dev)
        self.dirichlet = ~self.inner & (bc == 0)
        self.mirror = ~self.inner & (bc == 5)
        self.UD = _boundary_data(case, m, f) if case["walls"] == "box" else None
        self.mass = (self.detj[:, None] * ((self.phi ** 2 * self.wv[:, None]).sum(0)))[:, :, None]
        area = torch.zeros_like(self.detj)
        area.index_add_(0, self.c0, 0.5 * self.twice)
        area.index_add_(0, self.c1[self.inner], 0.5 * self.twice[self.inner])
        self.h = self.detj / 6.0 / area
        other = torch.where(self.inner, self.c1, self.c0)
        self.pairs = (torch.cat([self.c0, other]), torch.cat([other, self.c0]))

    def _trace(self, C, side):
        V = torch.zeros(self.n.shape[0], self.wf.numel(), 5, dtype=F64, device=C.device)
        for at, cell, phi, _ in self.sides[side]:
            V[at] = torch.einsum("gb,fbk->fgk", phi, C[cell])
        return V

    def _grad_trace(self, C, side):
        G = torch.zeros(self.n.shape[0], self.wf.numel(), 5, 3, dtype=F64, device=C.device)
        for at, cell, _, dphi in self.sides[side]:
            G[at] = torch.einsum("gbd,fbk,fmd->fgkm", dphi, C[cell], self.J[cell])
        return G

    def _ghost(self, UL, UR):
        if self.UD is not None:
            UR[self.dirichlet] = 2.0 * self.UD[self.dirichlet] - UL[self.dirichlet]
        flip = torch.tensor([1.0, 1.0, 1.0, -1.0, 1.0], dtype=F64, device=UL.device)
        UR[self.mirror] = flip * UL[self.mirror]
        return UR

    def _scatter(self, R, F, scale=1.0):
        """R += sum over the face points of F (already weighted) times the basis, out of the first cell."""
        for side, sign in ((0, scale), (1, -scale)):
            for at, cell, phi, _ in self.sides[side]:
                R.index_add_(0, cell, sign * torch.einsum("gb,fgk->fbk", phi, F[at]))
        return R

    def convection(self, C, part=0):
        R = torch.zeros_like(C)
        if part in (0, 1):
            V = torch.einsum("gb,ebk->egk", self.phi, C)
            F = _flux(V)[0]
            F = torch.einsum("egkm,emd,e->egkd", F, self.J, self.detj)
            R -= torch.einsum("gbd,g,egkd->ebk", self.dphi, self.wv, F)
            del F, V
        if part != 1:
            UL = self._trace(C, 0)
            UR = self._ghost(UL, self._trace(C, 1))
            flux = _roe if self.case["flux"] == "Roe" else _lax_friedrichs
            n = self.n[:, None, :]
            on = {0: self.inner | self.dirichlet | self.mirror, 2: self.inner, 3: self.dirichlet | self.mirror}[part]
            F = torch.zeros_like(UL)
            F[on] = flux(UL[on], UR[on], n.expand(-1, UL.shape[1], -1)[on]) * self.wf[None, :, None] * self.twice[on][:, None, None]
            self._scatter(R, F)
        return R

    def _homogeneity(self, U, X):
        """sum_m K_mn X_m by its columns n, for gradients X (..., 5, 3) at the state U."""
        mu, k = self.case["mu"], self.case["mu"] * GAMMA / PRANDTL
        rho = U[..., 0, None, None]
        u = U[..., 1:4] / U[..., :1]
        e = (U[..., 4] / U[..., 0])[..., None]
        Y = (X[..., 1:4, :] - u[..., :, None] * X[..., 0:1, :]) / rho
        Ye = (X[..., 4, :] - e * X[..., 0, :]) / rho[..., 0]
        tr = Y.diagonal(dim1=-2, dim2=-1).sum(-1)
        eye = torch.eye(3, dtype=F64, device=U.device)
        H = torch.zeros_like(X)
        H[..., 1:4, :] = mu * (Y + tr[..., None, None] * eye - (2.0 / 3.0) * Y.transpose(-1, -2))
        H[..., 4, :] = (u[..., :, None] * H[..., 1:4, :]).sum(-2) + k * (Ye - (u[..., :, None] * Y).sum(-2))
        return H

    def viscous(self, C):
        """The interior-penalty viscous residual."""
        R = torch.zeros_like(C)
        V = torch.einsum("gb,ebk->egk", self.phi, C)
        G = torch.einsum("gbd,ebk,emd->egkm", self.dphi, C, self.J)
        H = torch.einsum("egkm,emd,e,g->egkd", self._homogeneity(V, G), self.J, self.detj, self.wv)
        R -= torch.einsum("gbd,egkd->ebk", self.dphi, H)
        UL = self._trace(C, 0)
        UR = self._ghost(UL, self._trace(C, 1))
        GL, GR = self._grad_trace(C, 0), self._grad_trace(C, 1)
        inner = self.inner[:, None, None]
        X = torch.where(inner[..., None], 0.5 * (GL + GR), GL)
        Um = 0.5 * (UL + UR)
        n = self.n[:, None, None, :]
        dU = torch.where(inner, UL - UR, UL)
        beta = ((self.case["order"] + 1) ** 2 / self.h[self.c0])[:, None, None]
        F = (self._homogeneity(Um, X) * n).sum(-1) - beta * (self._homogeneity(Um, dU[..., None] * n) * n).sum(-1)
        on = (self.inner | self.dirichlet | self.mirror)[:, None, None]
        jw = (self.wf[None, :] * self.twice[:, None])[..., None]
        self._scatter(R, torch.where(on, F * jw, torch.zeros_like(F)))
        s = (torch.where(self.inner, 0.5, 1.0)[:, None] * self.case["mu"] * GAMMA / PRANDTL / Um[..., 0]
             * (UR[..., 4] - UL[..., 4]) * jw[..., 0])
        s = torch.where(on[..., 0], s, torch.zeros_like(s))
        S = torch.zeros(self.n.shape[0], self.nb, dtype=F64, device=C.device)
        for side in (0, 1):
            for at, cell, _, dphi in self.sides[side]:
                S[at] += torch.einsum("fg,gbd,fmd,fm->fb", s[at], dphi, self.J[cell], self.n[at])
        R[..., 4].index_add_(0, self.c0, S)
        R[..., 4].index_add_(0, self.c1[self.inner], -S[self.inner])
        return R

    def limited(self, C, before):
        """Bounds from the neighbourhood's values before, then density and pressure kept positive."""
        W = torch.einsum("gb,ebk->egk", self.phi, before)
        if self.case["limiter"] == "positive-avg":
            top = low = before[:, 0]
        else:
            top, low = W.amax(1), W[:, -1]
        index = self.pairs[0][:, None].expand(-1, 5)
        bmax = top.scatter_reduce(0, index, top[self.pairs[1]], "amax")
        bmin = low.scatter_reduce(0, index, low[self.pairs[1]], "amin")
        avg = C[:, 0]
        V = torch.einsum("gb,ebk->egk", self.phi, C)
        vmin, vmax = V.amin(1), V.amax(1)
        zero, one = torch.zeros_like(avg), torch.ones_like(avg)
        tmin = torch.where(avg != vmin, (avg - bmin) / (avg - vmin + 1e-32), zero)
        tmax = torch.where(avg != vmax, (bmax - avg) / (vmax - avg + 1e-32), zero)
        theta = torch.where((vmin < bmin) | (vmax > bmax), torch.minimum(torch.minimum(tmin, tmax), one), one)
        V = avg[:, None] + theta[:, None] * (V - avg[:, None])
        eps = 1e-16
        rmin = V[..., 0].amin(1)
        eff = avg[:, 0].clamp_min(eps)
        tr = torch.where(eff - rmin < 1e-32, zero[:, 0], torch.minimum((eff - eps) / (eff - rmin), one[:, 0]))
        tr = torch.where(rmin < eps, tr, one[:, 0])
        V[..., 0] = avg[:, None, 0] + tr[:, None] * (V[..., 0] - avg[:, None, 0])

        def pressure(S):
            p = (GAMMA - 1.0) * (S[..., 4] - (S[..., 1:4] ** 2).sum(-1) / (2.0 * S[..., 0]))
            return torch.where(S[..., 0] <= 1e-16, -torch.ones_like(p), p)

        bad = pressure(V) < 0
        lo = torch.zeros_like(V[..., 0])
        hi = torch.ones_like(lo)
        for _ in range(100):
            mid = 0.5 * (lo + hi)
            neg = pressure((1.0 - mid)[..., None] * avg[:, None] + mid[..., None] * V) < 0
            hi, lo = torch.where(neg, mid, hi), torch.where(neg, lo, mid)
        tp = torch.where(bad, mid, torch.ones_like(mid)).amin(1)
        scale = theta * tp[:, None]
        scale[:, 0] *= tr
        D = C.clone()
        D[:, 1:] *= scale[:, None, :]
        return D

    def step(self, C, dt):
        def rate(U):
            R = -self.convection(U)
            if self.case["mu"] > 0.0:
                R += self.viscous(U)
            return R / self.mass

        keep = self.limited if self.case["limiter"] != "none" else (lambda now, before: now)
        U1 = keep(C + dt * rate(C), C)
        U2 = keep(0.75 * C + 0.25 * (U1 + dt * rate(U1)), U1)
        return keep(C / 3.0 + (2.0 / 3.0) * (U2 + dt * rate(U2)), U2)

    def sums(self, C):
        V = torch.einsum("gb,ebk->egk", self.phi, C)
        kinetic = 0.5 * (V[..., 1:4] ** 2).sum(-1) / V[..., 0]
        total = (C[:, 0] * self.detj[:, None] / 6.0).sum(0)
        return np.append(total.cpu().numpy(), float((kinetic * self.wv * self.detj[:, None]).sum()))


def exact(case, seed):
    out = []
    for i, (n, m) in enumerate(zip(_sizes(case), _meshes(case))):
        f = _flow(case, seed, i)
        U = _project(case, m, f)
        op = _Operator(case, m, f)
        C = U.view(U.shape[0], -1, 5)
        if case["do"] in ("residual", "host"):
            R = op.convection(C, case["part"]).reshape(U.shape)
            return R.cpu().numpy() if case["do"] == "host" else R
        dt = _dt(case, n, _wave_speed(case, U))
        for _ in range(case["steps"]):
            C = op.step(C, dt)
        out.append(C.reshape(U.shape))
    if case["do"] == "adaptive":
        return out[0], dt
    if case["do"] == "monitored":
        return out[0], op.sums(out[0].view(U.shape[0], -1, 5))
    return torch.cat(out)
