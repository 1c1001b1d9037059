"""Workloads of the implicit hot path that its performance is followed on.

Three families, each through the entry points that a program calls:

solve     one ``Solver.solve(acoef, ss, sp, res, phi, n)``, the boundary that the host model calls three times per
          outer iteration: on device tensors, or on host arrays as a host model hands them over;
grad      the same solve inside torch's autograd (``adjoint.solve_fn``), forward and backward;
flow      a short simulation: cold start, a few implicit time steps, the water pressure and velocities read back.
          ``members`` > 1 steps that many basins together (``EnsembleModel``).

The linear systems are those of the solver sweep (face coefficients U[0.1, 1], diagonal 1.02 times their sum,
right-hand side N(0,1)) on telescoping and Cartesian grids; velocity systems have a larger diagonal, under-relaxation
and a non-zero start.  Grids and solver handles are kept from one call to the next, as a program keeps them.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from cms2d_b200 import adjoint, cases as flow_cases, grid as grids
from cms2d_b200.ensemble import EnsembleModel
from cms2d_b200.flow import FlowModel
from cms2d_b200.solver import RELAX_DEFAULT, Solver

GMRES, BICGSTAB = 4, 3


def _solve(name, grid, nx, ny, **kw):
    """A solve case.  grid: "telescoping" with about nx * ny cells, or "cartesian" nx x ny.  nswp 0: the default of
    the variable n.  tol and norm: the stopping test (1e-3 of the L1 or GMRES residual is the solver's default)."""
    c = {"name": name, "family": "solve", "grid": grid, "nx": nx, "ny": ny, "n": 1, "nsolv": GMRES,
         "precision": "fp64", "dtype": "float64", "tol": 1e-3, "norm": 1, "nswp": 0, "host": False}
    c.update(kw)
    return c


def listed():
    return [
        # a velocity system of the tidal basin with every option at its default (GMRES, FP64): the shortest call that
        # a model makes, twice per outer iteration
        _solve("uv_gmres_20k", "cartesian", 200, 100, n=2),
        # a pressure-correction system of the 1M-cell grid with every option at its default
        _solve("pp_gmres_1m", "telescoping", 1000, 1000),
        # the default solver called on host arrays, as the drop-in for a host model's solve(); ragged Cartesian grid
        _solve("pp_gmres_host_100k", "cartesian", 333, 301, host=True),
        # the solver sweep's systems to 1e-6 with the FP64 BiCGStab
        _solve("pp_bicg64_1m", "telescoping", 1000, 1000, nsolv=BICGSTAB, tol=1e-6, norm=2, nswp=200),
        # the same solver in single precision, as a build with 4-byte reals calls it
        _solve("pp_bicg32_1m", "telescoping", 1000, 1000, nsolv=BICGSTAB, dtype="float32", tol=1e-5, norm=2, nswp=200),
        # FP32 inner solves inside FP64 refinement, to the accuracy of an FP64 solution, over the sweep's sizes
        _solve("pp_refine_250k", "telescoping", 500, 500, nsolv=BICGSTAB, precision="fp32_refine", tol=1e-11, norm=2,
               nswp=600),
        _solve("pp_refine_1m", "telescoping", 1000, 1000, nsolv=BICGSTAB, precision="fp32_refine", tol=1e-11, norm=2,
               nswp=600),
        _solve("pp_refine_4m", "telescoping", 2000, 2000, nsolv=BICGSTAB, precision="fp32_refine", tol=1e-11, norm=2,
               nswp=600),
        # a solve and its adjoint: gradients of a loss on the solution for every coefficient
        {"name": "grad_100k", "family": "grad", "grid": "telescoping", "nx": 317, "ny": 317, "tol": 1e-10,
         "adjoint_tol": 1e-9},
        # simulations: the tidal basin with every option at its default (GMRES, FP64), the telescoping inlet with
        # FP32 + refinement at converged solves, and a small ensemble of uneven inlets stepped together
        {"name": "flow_basin_20k", "family": "flow", "case": "basin", "nx": 200, "ny": 100, "members": 1, "steps": 3,
         "nsolv": GMRES, "precision": "fp64", "tol": 1e-3, "norm": 1, "nswp": 0},
        {"name": "flow_inlet_30k", "family": "flow", "case": "inlet", "nx": 171, "ny": 180, "members": 1, "steps": 2,
         "nsolv": BICGSTAB, "precision": "fp32_refine", "tol": 1e-10, "norm": 2, "nswp": 600},
        {"name": "ensemble_6x10k", "family": "flow", "case": "inlet", "nx": 110, "ny": 100, "members": 6, "steps": 1,
         "nsolv": BICGSTAB, "precision": "fp32_refine", "tol": 1e-10, "norm": 2, "nswp": 600},
    ]


def _sides(rng, lo, hi):
    """nx, ny with nx * ny log-uniform in [lo, hi], aspect ratio up to 4, any parity."""
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a = math.exp(rng.uniform(-math.log(4.0), math.log(4.0)) / 2)
    return max(8, round(math.sqrt(cells) * a)), max(8, round(math.sqrt(cells) / a))


def draw(rng):
    kind = rng.choice(["gmres", "gmres_host", "bicg64", "bicg32", "refine", "refine", "grad", "flow", "flow", "ensemble"])
    grid = rng.choice(["telescoping", "cartesian"])
    if kind in ("grad", "flow", "ensemble"):
        if kind == "grad":
            nx, ny = _sides(rng, 20_000, 500_000)
            return {"family": "grad", "grid": grid, "nx": nx, "ny": ny, "tol": 1e-10, "adjoint_tol": 1e-9}
        refine = kind == "ensemble" or rng.random() < 0.5
        nx, ny = _sides(rng, 4_000, 11_000 if kind == "ensemble" else 30_000 if refine else 40_000)
        c = {"family": "flow", "case": "inlet" if refine else rng.choice(["basin", "inlet"]), "nx": nx, "ny": ny,
             "members": 1 if kind == "flow" else rng.randint(2, 6), "steps": 1 if kind == "ensemble" else rng.randint(1, 2)}
        if refine:
            return dict(c, nsolv=BICGSTAB, precision="fp32_refine", tol=1e-10, norm=2, nswp=600)
        return dict(c, nsolv=GMRES, precision="fp64", tol=1e-3, norm=1, nswp=0)
    top = {"gmres": 1_200_000, "gmres_host": 300_000, "bicg64": 1_200_000, "bicg32": 2_000_000, "refine": 4_000_000}[kind]
    nx, ny = _sides(rng, 1_000, top)
    kw = {"gmres": {"n": rng.choice([1, 2, 3])}, "gmres_host": {"n": rng.choice([1, 2]), "host": True},
          "bicg64": {"nsolv": BICGSTAB, "tol": 1e-6, "norm": 2, "nswp": 200},
          "bicg32": {"nsolv": BICGSTAB, "dtype": "float32", "tol": 1e-5, "norm": 2, "nswp": 200},
          "refine": {"nsolv": BICGSTAB, "precision": "fp32_refine", "tol": 1e-11, "norm": 2, "nswp": 600}}[kind]
    c = _solve("", grid, nx, ny, **kw)
    del c["name"]
    return c


@functools.lru_cache(maxsize=4)
def _grid(kind, nx, ny):
    return grids.cartesian_grid(nx, ny) if kind == "cartesian" else grids.solver_test_grid(nx * ny)


@functools.lru_cache(maxsize=2)
def _solver(kind, nx, ny, **options):
    return Solver(_grid(kind, nx, ny), **options)


def _links(g, device):
    """Per cell and face slot: whether the face exists, and the neighbour's 0-based number (the cell itself elsewhere)."""
    n = g.ncells
    has = torch.as_tensor(np.arange(g.nmaxfaces)[None, :] < g.ncface[:n, None], device=device)
    nb = torch.as_tensor(g.cell2cell[:n].astype(np.int64) - 1, device=device)
    return has, torch.where(has, nb, torch.arange(n, device=device)[:, None])


def _system(case, seed):
    """acoef, ss, sp, phi of a system in the solve() layout (float64 values of the case's type, on the GPU), relax(n)."""
    g = _grid(case["grid"], case["nx"], case["ny"])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case.get("n", 1)
    real = getattr(torch, case.get("dtype", "float64"))
    has, _ = _links(g, "cuda")
    acoef = torch.zeros(g.ncellsD, g.nmaxfaces, dtype=torch.float64, device="cuda")
    acoef[: g.ncells] = (0.1 + 0.9 * torch.rand(has.shape, dtype=torch.float64, device="cuda", generator=gen)) * has
    sp = -(0.02 if n == 1 else 0.5) * acoef.sum(1)
    ss = torch.zeros_like(sp)
    ss[: g.ncells] = torch.randn(g.ncells, dtype=torch.float64, device="cuda", generator=gen)
    phi = torch.zeros_like(sp)
    if n != 1:
        phi[: g.ncells] = 0.3 * torch.randn(g.ncells, dtype=torch.float64, device="cuda", generator=gen)
    return g, [t.to(real).contiguous() for t in (acoef, ss, sp, phi)], RELAX_DEFAULT[n]


def _flow_case(case, seed, k=0):
    """The case of a simulation (member k of an ensemble).  It starts in the running tide, a quarter of an M2 period
    after high water: slack water, with hardly any current, is what a simulation sees least of."""
    if case["members"] == 1:
        share, tide = 1.0, 1.0
    else:  # uneven members: half to full size, a tide and a bed of their own
        share = np.random.default_rng(k).uniform(0.5, 1.0)
        tide = np.random.default_rng([seed, k]).uniform(0.5, 1.5)
    if case["case"] == "inlet":
        c = flow_cases.tidal_inlet(round(case["nx"] * case["ny"] * share), seed=seed + k)
    else:
        c = flow_cases.tidal_basin(case["nx"], round(case["ny"] * share), seed=seed + k)
    c.tide = [(tide * a, period) for a, period in c.tide]
    c.t0 = 0.25 * flow_cases.M2_HOURS * 3600.0
    return c


def prepare(case, seed):
    if case["family"] == "flow":
        kw = {k: case[k] for k in ("nsolv", "precision", "tol", "norm")}
        if case["nswp"]:
            kw.update(nswp_pp=case["nswp"], nswp_uv=case["nswp"])
        if case["members"] == 1:
            model = FlowModel(_flow_case(case, seed), **kw)
        else:
            model = EnsembleModel([_flow_case(case, seed, k) for k in range(case["members"])], **kw)
        return {"case": case, "model": model}
    g, system, relax = _system(case, seed)
    key = (case["grid"], case["nx"], case["ny"])
    if case["family"] == "grad":
        solver = _solver(*key, tol=case["tol"], norm=2, max_iters=4000, verify=False, nsolv=BICGSTAB)
        gen = torch.Generator(device="cuda").manual_seed(seed + 1)
        w = torch.zeros_like(system[1])
        w[: g.ncells] = torch.randn(g.ncells, dtype=torch.float64, device="cuda", generator=gen)
        return {"case": case, "solver": solver, "system": system, "weights": w}
    solver = _solver(*key, precision=case["precision"], tol=case["tol"], norm=case["norm"], nsolv=case["nsolv"])
    if case["host"]:
        system = [t.cpu().numpy() for t in system]
        work = [np.empty_like(system[1]), np.zeros_like(system[1]), np.empty_like(system[3])]
    else:
        work = [torch.empty_like(system[1]), torch.zeros_like(system[1]), torch.empty_like(system[3])]
    return {"case": case, "solver": solver, "system": system, "work": work, "relax": relax}


def run(state):
    case = state["case"]
    if case["family"] == "flow":
        model = state["model"]
        model.init()
        for _ in range(case["steps"]):
            model.step()
        return [[m.get(f) for f in ("p", "u", "v")] for m in getattr(model, "members", [model])]
    if case["family"] == "grad":
        acoef, ss, sp, phi = state["system"]
        leaf = [t.detach().requires_grad_() for t in (acoef, ss, sp)]
        x = adjoint.solve_fn(state["solver"], *leaf, phi, relax=1.0, nswp=4000, tol=case["adjoint_tol"])
        x.backward(state["weights"])
        return [x.detach()] + [t.grad for t in leaf]
    acoef, ss0, sp, phi0 = state["system"]
    ss, res, phi = state["work"]  # solve() updates ss and phi: each call gets its own
    if case["host"]:
        np.copyto(ss, ss0)
        np.copyto(phi, phi0)
    else:
        ss.copy_(ss0)
        phi.copy_(phi0)
    state["solver"].solve(acoef, ss, sp, res, phi, n=case["n"], nswp=case["nswp"] or None)
    return [phi, res, ss]


def work(case):
    """Bytes: the call's arrays, each input read once and each output written once (the systems' coefficients, sources
    and solution; a simulation's fields per step).  Flops: one product with the matrix (per solve of one outer iteration)."""
    cells = case["nx"] * case["ny"]
    if case["family"] == "flow":
        cells = round(cells * (1.0 if case["members"] == 1 else 0.75)) * case["members"]
        return {"bytes": case["steps"] * cells * 8 * (3 * 2 + 3 * 4), "flops": case["steps"] * cells * 3 * 10}
    faces = 6 if case["grid"] == "telescoping" else 4
    real = 4 if case.get("dtype") == "float32" else 8
    if case["family"] == "grad":
        return {"bytes": cells * real * (2 * faces + 7), "flops": 4 * cells * 10}
    return {"bytes": cells * real * (faces + 6), "flops": cells * 10}


def _jacobi(rhs, ap, step):
    """x = (rhs + O x) / ap to the rounding of 64 bits (diagonally dominant: the error shrinks by the dominance per step)."""
    x = rhs / ap
    for _ in range(80):
        for _ in range(50):
            x, old = (rhs + step(x)) / ap, x
        if float((x - old).norm()) <= 1e-15 * float(x.norm()):
            break
    return x


def exact(case, seed):
    if case["family"] == "flow":
        return None
    g, system, relax = _system(case, seed)
    acoef, ss, sp, phi = [t.double() for t in system]
    if case["family"] == "grad":
        relax = 1.0
    n = g.ncells
    has, nb = _links(g, "cuda")
    a = acoef[:n]
    inner = has & (nb < n)
    ghost = (a * phi[nb] * (has & ~inner)).sum(1)
    to, ai = torch.where(inner, nb, 0), a * inner

    def forward(x):
        y = ai[:, 0] * x[to[:, 0]]
        for k in range(1, g.nmaxfaces):
            y += ai[:, k] * x[to[:, k]]
        return y

    ap = (a.sum(1) - sp[:n]) / relax
    ss2, res, x = ss.clone(), torch.zeros_like(ss), phi.clone()
    ss2[:n] += (1.0 - relax) * phi[:n] * ap
    res[:n] = (forward(phi[:n]) + ghost + ss2[:n] - ap * phi[:n]) / ap
    x[:n] = _jacobi(ss2[:n] + ghost, ap, forward)
    if case["family"] == "solve":
        return [x, res, ss2]
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    w = torch.randn(n, dtype=torch.float64, device="cuda", generator=gen)
    flat, coef = to.reshape(-1), ai
    lam = _jacobi(w, ap, lambda v: torch.zeros_like(v).index_add_(0, flat, (coef * v[:, None]).reshape(-1)))
    gss, gsp, gac = torch.zeros_like(ss), torch.zeros_like(sp), torch.zeros_like(acoef)
    gss[:n] = lam
    gsp[:n] = lam * x[:n]
    gac[:n] = lam[:, None] * (x[nb] - x[:n, None]) * has
    return [x, gac, gss, gsp]
