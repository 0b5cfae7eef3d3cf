"""Performance cases of pic_b200: what a user's program has the library do.

Seven kinds of call, each through the public classes:

  step      PICSimulation.step, the fused PIC step (the library's main path):
            the small, collisional and large workloads of pic_b200.workloads,
            and the axisymmetric r-z step
  ensemble  Ensemble.step, several simulations stepped as one graph
  dropin    simulation.reference_step on Particles2D / Grid2D / Solver, the
            operators called one by one in the reference's order
  mcc       MccOperator.apply and take_births, the collision operator alone
  poisson   MultigridSolver.solve, one Poisson solve from a given guess
  solver    Solver.solve and Grid2D.update_E ('direct', 'cg', 'multigrid')
  adjoint   ElectrodeLoss forward and backward, the differentiable step

Sizes come from pic_b200/workloads.py, pic_b200/ensemble.py, pic_b200/adjoint.py
and the tests; node counts are c * 2^k + 1, as the multigrid needs them.

A case is a dict of plain values.  prepare() makes its inputs on the GPU from
a seed, run() is one pass, work() the bytes and operations the pass cannot do
without, exact() the same outputs in FP64 with torch alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pic_b200 import Consts, adjoint, workloads
from pic_b200.Boundaries import Boundaries, walls_box
from pic_b200.ensemble import Ensemble
from pic_b200.Grid import Grid2D
from pic_b200.MCC import MccOperator
from pic_b200.multigrid import MultigridSolver
from pic_b200.Particles import Particles2D
from pic_b200.simulation import PICSimulation, reference_init_step, reference_step
from pic_b200.Solvers import Solver

DX, DT, N0 = 1e-4, 1e-11, 1e14
TE, TI = 2.0, 0.03
TILE, SORT_INTERVAL = 16, 80
MASS = (Consts.me, workloads.ION_MASS)
CHARGE = (-Consts.qe, Consts.qe)
F8, F4 = torch.float64, torch.float32


def listed():
    return [
        # the smallest run of the reference's configurations: launches and latency count
        _step("step_small", 129, 129, 100_000, 100_000, steps=20),
        # the headline workload: 8M particles with collisions
        _step("step_mcc", 513, 513, 4_000_000, 4_000_000, left=100.0, mcc=True, steps=10),
        # the largest stated workload, half the electrons in a blob, tight field solves
        _step("step_large", 2049, 2049, 64_000_000, 64_000_000, tol=1e-10, blob=True, steps=3),
        # an axisymmetric discharge on a rectangular grid, uneven counts
        _step("step_rz", 257, 129, 1_234_567, 987_654, rz=True, left=50.0, steps=10),
        # a parameter scan: members of different grids stepped together
        {"name": "ensemble_8", "kind": "ensemble", "members": 8, "n_min": 100_000, "n_max": 2_000_000, "steps": 10},
        # the operators one call at a time, particles in the order they were loaded in
        {"name": "dropin_step", "kind": "dropin", "nx": 257, "ny": 257, "n": 1_000_003, "left": 20.0, "tol": 1e-8},
        # collisions on their own, as null_collision_method makes them
        {"name": "mcc_operator", "kind": "mcc", "nx": 513, "ny": 513, "n": 4_000_001},
        # one large potential, mixed precision, to a tight residual
        _poisson("poisson_2049", 2049, 2049, "mixed", 1e-10),
        # a rectangular domain with an electrode inside, FP64 throughout
        _poisson("poisson_fp64_ragged", 385, 193, "fp64", 1e-9, electrode=True),
        # the exact solve of the 'direct' and 'inverse' branches on the headline grid
        {"name": "solver_direct", "kind": "solver", "solver": "direct", "nx": 513, "ny": 513, "left": 100.0,
         "tol": 1e-8},
        # the Krylov branch on a rectangular grid
        {"name": "solver_cg", "kind": "solver", "solver": "cg", "nx": 385, "ny": 257, "left": 25.0, "tol": 1e-9},
        # the differentiable workload with fewer steps: the forward and the backward pass
        {"name": "adjoint", "kind": "adjoint", "nodes": 257, "n": 1_000_000, "steps": 40, "every": 20},
    ]


def _step(name, nx, ny, n_e, n_i, tol=1e-8, left=0.0, mcc=False, rz=False, blob=False, solver="graph", steps=10):
    return {"name": name, "kind": "step", "nx": nx, "ny": ny, "n_e": n_e, "n_i": n_i, "tol": tol, "left": left,
            "mcc": mcc, "rz": rz, "blob": blob, "solver": solver, "steps": steps}


def _poisson(name, nx, ny, precision, tol, electrode=False):
    return {"name": name, "kind": "poisson", "nx": nx, "ny": ny, "precision": precision, "tol": tol,
            "electrode": electrode}


def draw(rng):
    """One more case of the listed ranges."""
    kind = rng.choice(["step", "step", "step", "ensemble", "dropin", "mcc", "poisson", "poisson", "solver", "solver",
                       "adjoint"])
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731

    def nodes(qmin, qmax):
        # c * 2^q + 1 in both directions, c in 4..8: from 65 nodes for q = 4 to 2049 for q = 8
        q = rng.randint(qmin, qmax)
        return rng.randint(4, 8) * 2 ** q + 1, rng.randint(4, 8) * 2 ** q + 1

    def powers(qmin, qmax):
        # 2^q + 1 in both directions, as the sine-transform solve takes them, at most 4 : 1
        q = rng.randint(qmin, qmax)
        return 2 ** q + 1, 2 ** min(qmax, max(qmin, q + rng.randint(-2, 2))) + 1

    if kind == "step":
        rz, dst = rng.random() < 0.25, rng.random() < 0.2
        nx, ny = powers(6, 11) if dst and not rz else nodes(4, 8)
        c = _step("", nx, ny, log(20_000, 16_000_000), log(20_000, 16_000_000), tol=rng.choice([1e-6, 1e-8, 1e-10]),
                  left=rng.choice([0.0, 20.0, 100.0]), mcc=rng.random() < 0.4, rz=rz, blob=rng.random() < 0.3,
                  solver="dst" if dst and not rz else "graph", steps=rng.randint(4, 20))
    elif kind == "ensemble":
        lo = log(20_000, 200_000)
        c = {"kind": "ensemble", "members": rng.randint(2, 8), "n_min": lo, "n_max": lo * rng.randint(2, 10),
             "steps": rng.randint(4, 10)}
    elif kind == "dropin":
        nx, ny = nodes(4, 6)
        c = {"kind": "dropin", "nx": nx, "ny": ny, "n": log(20_000, 1_000_000), "left": rng.choice([0.0, 20.0, 100.0]),
             "tol": rng.choice([1e-6, 1e-8])}
    elif kind == "mcc":
        nx, ny = nodes(4, 7)
        c = {"kind": "mcc", "nx": nx, "ny": ny, "n": log(20_000, 4_000_000)}
    elif kind == "poisson":
        nx, ny = nodes(3, 8)
        c = _poisson("", nx, ny, rng.choice(["mixed", "fp64"]), rng.choice([1e-6, 1e-8, 1e-9]), rng.random() < 0.3)
    elif kind == "solver":
        solver = rng.choice(["direct", "cg", "multigrid"])
        nx, ny = powers(5, 11) if solver == "direct" else nodes(3, 7)
        c = {"kind": "solver", "solver": solver, "nx": nx, "ny": ny, "left": rng.choice([0.0, 25.0, 100.0]),
             "tol": rng.choice([1e-6, 1e-8, 1e-9])}
    else:
        steps = rng.randint(6, 40)
        c = {"kind": "adjoint", "nodes": rng.choice([65, 129, 257]), "n": log(10_000, 1_000_000), "steps": steps,
             "every": rng.randint(3, 20)}
    c.pop("name", None)
    return c


# ---- inputs ----------------------------------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, n, lo, hi):
    return torch.rand(n, generator=g, device="cuda", dtype=F4).mul_(hi - lo).add_(lo)


def _inside(x, top):
    return x.clamp_(0.0, float(np.nextafter(np.float32(top), np.float32(0))))


def _positions(g, n, nx, ny, rz=False, blob=False):
    """Grid-unit positions: uniform (r-z: uniform in volume), or half of them in a Gaussian blob."""
    x, y = _rand(g, n, 0.0, nx - 1.0), _rand(g, n, 0.0, 1.0)
    y = (y.sqrt_() if rz else y).mul_(ny - 1.0)
    if blob and not rz:
        for a, top in ((x, nx - 1.0), (y, ny - 1.0)):
            b = torch.randn(n // 2, generator=g, device="cuda", dtype=F4).mul_(0.2 * top).add_(0.5 * top)
            a[: n // 2] = torch.where((b >= 0) & (b < top), b, a[: n // 2])
    return _inside(x, nx - 1.0), _inside(y, ny - 1.0)


def _species(g, s, n, nx, ny, rz=False, blob=False):
    vth = math.sqrt((TE, TI)[s] * Consts.qe / MASS[s])
    x, y = _positions(g, n, nx, ny, rz, blob and s == 0)
    v = [torch.randn(n, generator=g, device="cuda", dtype=F4).mul_(vth) for _ in range(3)]
    return [x, y, *v]


def _np2c(nx, ny, n, rz=False):
    X, Y = DX * (nx - 1), DX * (ny - 1)
    return N0 * X * (math.pi * Y * Y if rz else Y) / n


def _walls(nx, ny, left, rz=False):
    """Dirichlet mask and values: every edge (r-z: not the axis), the left wall at `left` volts."""
    mask, phi = np.zeros((ny, nx), np.uint8), np.zeros((ny, nx))
    mask[-1, :] = mask[:, 0] = mask[:, -1] = 1
    if not rz:
        mask[0, :] = 1
    phi[0 if rz else 1:-1, 0] = left
    return mask, phi


def _simulation(c, seed, s_interval=SORT_INTERVAL):
    nx, ny, rz = c["nx"], c["ny"], c["rz"]
    g = _gen(seed)
    mask, phi = _walls(nx, ny, c["left"], rz)
    counts = (c["n_e"], c["n_i"])
    species = [dict(name="ei"[s], charge=CHARGE[s], mass=MASS[s], np2c=_np2c(nx, ny, counts[s], rz),
                    capacity=counts[s] + (counts[s] // 8 + 4096 if c["mcc"] else 64)) for s in (0, 1)]
    mcc = workloads.mcc_tables(workloads.MCC) if c["mcc"] else None
    sim = PICSimulation(nx, ny, DX, DX, DT, species, mask.reshape(-1), phi.reshape(-1), tol=c["tol"],
                        sort_interval=s_interval, tile=TILE, mcc=mcc, seed=int(seed), use_graph=True,
                        mg_launch=c["solver"], geometry="rz" if rz else "cartesian")
    for s in (0, 1):
        sim.load(s, *_species(g, s, counts[s], nx, ny, rz, c["blob"]))
    sim.init()
    return sim, counts


def _member_cases(c, seed):
    """The members of an ensemble: grids and particle counts drawn from the case alone."""
    rng = np.random.default_rng(c["members"] * 1009 + c["n_min"])
    out = []
    for i in range(c["members"]):
        side = int(rng.choice((129, 257, 513)))
        n = rng.integers(c["n_min"], c["n_max"] + 1, 2)
        out.append(_step("", side, side, int(n[0]), int(n[1]), left=float(rng.uniform(0.0, 200.0))))
    return [(m, int(seed) * 64 + i) for i, m in enumerate(out)]


def _rhs(g, nx, ny):
    """Space charge over eps0: smooth modes and the noise of a particle load."""
    i = torch.arange(nx, device="cuda", dtype=F8) / (nx - 1)
    j = torch.arange(ny, device="cuda", dtype=F8)[:, None] / (ny - 1)
    a = torch.rand(6, generator=g, device="cuda", dtype=F8).tolist()
    f = torch.zeros(ny, nx, device="cuda", dtype=F8)
    for k in range(3):
        f += (a[k] - 0.5) * torch.sin(math.pi * (k + 1) * i) * torch.sin(math.pi * (3 - k) * j + a[3 + k])
    f += 0.1 * torch.randn(ny, nx, generator=g, device="cuda", dtype=F8)
    return f * (N0 * Consts.qe / Consts.eps0)


def _electrode(nx, ny, mask, phi):
    i = (nx - 1) // 4
    a, b = (ny - 1) // 4, (ny - 1) // 2
    mask[a:b + 1, i] = 1
    phi[a:b + 1, i] = -30.0


def _poisson_inputs(c, seed):
    nx, ny = c["nx"], c["ny"]
    mask, phi = _walls(nx, ny, 100.0)
    if c["electrode"]:
        _electrode(nx, ny, mask, phi)
    f = _rhs(_gen(seed), nx, ny)
    f[torch.as_tensor(mask, device="cuda").bool()] = 0.0
    return mask, torch.as_tensor(phi, device="cuda"), f


def _solver_grid(c):
    grid = Grid2D(c["nx"], c["ny"], DX * (c["nx"] - 1), DX * (c["ny"] - 1))
    return grid, Boundaries(walls_box(grid, left=c["left"]), grid)


def _adjoint_inputs(c, seed):
    """Initial particles (FP64, grid units), the perturbation direction, potentials and the target density."""
    m, n, g = c["nodes"], c["n"], _gen(seed)
    sp = [[a.to(F8) for a in _species(g, s, n, m, m)[:4]] for s in (0, 1)]
    dvx = torch.sin(2 * math.pi * sp[0][0] / (m - 1))
    V = (torch.rand(4, generator=g, device="cuda", dtype=F8) * 50.0).cpu()
    target = torch.as_tensor(adjoint.target_density(m, m, N0, int(seed) + 1), device="cuda")
    return sp, dvx, V, torch.tensor(1e4, dtype=F8), target


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        sim, counts = _simulation(case, seed)
        return {"kind": kind, "sim": sim, "counts": counts, "steps": case["steps"]}
    if kind == "ensemble":
        sims = [_simulation(m, s) for m, s in _member_cases(case, seed)]
        return {"kind": kind, "ens": Ensemble([s for s, _ in sims]), "members": sims, "steps": case["steps"]}
    if kind == "dropin":
        grid, bnd = _solver_grid(case)
        parts = Particles2D(case["n"])
        parts.grid = grid
        g = _gen(seed)
        parts.np2c = _np2c(case["nx"], case["ny"], case["n"])
        for s, name in enumerate(("electrons", "ions")):
            parts.add_species(name, MASS[s], CHARGE[s], s)
            x, y, *v = _species(g, s, case["n"], case["nx"], case["ny"])
            parts.load_species_arrays(s + 1, x.to(F8) * grid.dx, y.to(F8) * grid.dy, *v)
        solver = Solver("multigrid", grid, boundaries=bnd, tol=case["tol"])
        reference_init_step(parts, grid, solver, DT)
        return {"kind": kind, "parts": parts, "grid": grid, "solver": solver}
    if kind == "mcc":
        op = MccOperator(workloads.mcc_tables(workloads.MCC), list(MASS), DT, seed=int(seed))
        return {"kind": kind, "op": op, "e": _species(_gen(seed), 0, case["n"], case["nx"], case["ny"])}
    if kind == "poisson":
        mask, phi, f = _poisson_inputs(case, seed)
        mg = MultigridSolver(mask.reshape(-1), case["nx"], case["ny"], DX, precision=case["precision"])
        return {"kind": kind, "mg": mg, "guess": phi.reshape(-1), "phi": phi.reshape(-1).clone(), "f": f.reshape(-1),
                "tol": case["tol"]}
    if kind == "solver":
        grid, bnd = _solver_grid(case)
        grid.rho = (_rhs(_gen(seed), case["nx"], case["ny"]) * -Consts.eps0).to(F4).reshape(-1)
        solver = Solver(case["solver"], grid, boundaries=bnd, tol=case["tol"])
        return {"kind": kind, "grid": grid, "solver": solver, "guess": grid.phi.clone()}
    sp, dvx, V, A, target = _adjoint_inputs(case, seed)
    m, n = case["nodes"], case["n"]
    mask, seg = adjoint.wall_segments(m, m)
    species = [dict(n=n, charge=CHARGE[s], mass=MASS[s], np2c=_np2c(m, m, n)) for s in (0, 1)]
    prob = adjoint.AdjointProblem(m, m, DX, DX, DT, species, mask, seg, 4, case["steps"], case["every"], tol=1e-11,
                                  max_cycles=60)
    prob.set_particles(0, *sp[0], dvx, torch.zeros_like(dvx))
    prob.set_particles(1, *sp[1])
    prob.set_target(target)
    return {"kind": kind, "prob": prob, "V": V, "A": A}


# ---- one pass --------------------------------------------------------------------------------------------------------


def _fields_of(sim):
    """The fields, as views of the simulation's own buffers that keep it alive."""
    out = dict(zip(("phi", "rho", "Ex", "Ey"), sim.fields()))
    for t in out.values():
        t.owner = sim
    return out


def _state_of(sim, counts):
    """Fields and particles after a step.  Slots of particles born since the load follow the loaded ones in no
    fixed order and are left out."""
    out = _fields_of(sim)
    for s in (0, 1):
        for name, a in zip(("x", "y", "vx", "vy", "vz"), sim.species_arrays(s)):
            t = out[f"{name}{s}"] = a[: counts[s]]
            t.owner = sim
    return out


def run(state):
    kind = state["kind"]
    if kind == "step":
        state["sim"].step(state["steps"])
        return _state_of(state["sim"], state["counts"])
    if kind == "ensemble":
        state["ens"].step(state["steps"])
        return [_fields_of(sim) for sim, _ in state["members"]]
    if kind == "dropin":
        parts, grid = state["parts"], state["grid"]
        reference_step(parts, grid, DT, state["solver"])
        out = {"phi": grid.phi, "rho": grid.rho, "E": grid.E}
        for s, sp in enumerate(parts.species):
            out.update({f"{name}{s}": a[: sp.n] for name, a in zip(("x", "y", "vx", "vy"), sp.arrays())})
        return out
    if kind == "mcc":
        op, e = state["op"], state["e"]
        op.apply(0, *e, e[0].numel())
        births = op.take_births()
        return {"vx": e[2], "vy": e[3], "vz": e[4], "counters": op.counters, "born": births[0].numel()}
    if kind == "poisson":
        phi = state["phi"].copy_(state["guess"])
        phi, _ = state["mg"].solve(phi, state["f"], tol=state["tol"])
        return phi
    if kind == "solver":
        grid = state["grid"]
        grid.phi.copy_(state["guess"])
        state["solver"].solve(grid)
        grid.update_E()
        return {"phi": grid.phi, "E": grid.E}
    V = state["V"].clone().requires_grad_()
    A = state["A"].clone().requires_grad_()
    loss = adjoint.ElectrodeLoss.apply(V, A, state["prob"])
    loss.backward()
    return {"loss": loss.detach(), "dV": V.grad, "dA": A.grad}


# ---- what a pass cannot do without -----------------------------------------------------------------------------------

# per particle and step: x, y, vx, vy read and written in FP32 (r-z: vz too); per node and step: phi read and
# written, its last value read, E written and read, rho written and read
STEP_NODE_BYTES = 8 * 3 + 8 * 2 + 4 * 2
PUSH_FLOPS, SOLVE_FLOPS = 60, 60


def work(case):
    kind = case["kind"]
    if kind == "step":
        n, G = case["n_e"] + case["n_i"], case["nx"] * case["ny"]
        return {"bytes": case["steps"] * (n * (40 if case["rz"] else 32) + G * STEP_NODE_BYTES),
                "flops": case["steps"] * (n * PUSH_FLOPS + G * SOLVE_FLOPS)}
    if kind == "ensemble":
        parts = [work(dict(m, steps=case["steps"])) for m, _ in _member_cases(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if kind == "dropin":
        n, G = 2 * case["n"], case["nx"] * case["ny"]
        return {"bytes": n * 32 + G * STEP_NODE_BYTES, "flops": n * PUSH_FLOPS + G * SOLVE_FLOPS}
    if kind == "mcc":
        # only the candidates' state is touched: about 0.24 % of the electrons, 28 bytes read and 12 written each
        return {"bytes": case["n"] * 0.0024 * 40, "flops": case["n"] * 0.0024 * 200}
    if kind in ("poisson", "solver"):
        G = case["nx"] * case["ny"]
        return {"bytes": G * (25 if kind == "poisson" else 29), "flops": G * SOLVE_FLOPS}
    # forward: x, y, ux, uy read and written; backward: they are recomputed, and the adjoint state is read and written
    n = 2 * case["n"]
    return {"bytes": case["steps"] * n * (64 + 64 + 64), "flops": case["steps"] * n * 4 * PUSH_FLOPS}


# ---- the same in FP64 with torch alone -------------------------------------------------------------------------------


def _dst(a, dim):
    """DST-I along dim (length M - 1) through the FFT of the odd extension."""
    a = a.movedim(dim, -1)
    z = torch.zeros_like(a[..., :1])
    y = torch.fft.rfft(torch.cat([z, a, z, -a.flip(-1)], -1), dim=-1)
    return (-0.5 * y.imag[..., 1:a.shape[-1] + 1]).movedim(-1, dim)


def _lam(m):
    k = torch.arange(1, m - 1, device="cuda", dtype=F8)
    return 4.0 / (DX * DX) * torch.sin(math.pi * k / (2.0 * (m - 1))) ** 2


def _solve_box(phi, f):
    """lap(phi) = f inside, phi given on the four edges."""
    ny, nx = phi.shape
    c = 1.0 / (DX * DX)
    b = f[1:-1, 1:-1].clone()
    b[:, 0] -= c * phi[1:-1, 0]
    b[:, -1] -= c * phi[1:-1, -1]
    b[0] -= c * phi[0, 1:-1]
    b[-1] -= c * phi[-1, 1:-1]
    u = _dst(_dst(b, 0), 1) / -(_lam(nx)[None] + _lam(ny)[:, None])
    u = _dst(_dst(u, 0), 1) * (4.0 / ((nx - 1) * (ny - 1)))
    pad = torch.nn.functional.pad(u, (1, 1, 1, 1))
    edge = torch.zeros_like(phi)
    edge[0], edge[-1], edge[:, 0], edge[:, -1] = phi[0], phi[-1], phi[:, 0], phi[:, -1]
    return pad + edge


def _solve_rz(phi, f):
    """The axisymmetric operator: rows are radii, row 0 the free axis; sine modes along z, tridiagonal in r."""
    ny, nx = phi.shape
    c = 1.0 / (DX * DX)
    j = torch.arange(ny - 1, device="cuda", dtype=F8)
    up = c * (1.0 + 0.5 / j.clamp(min=1.0))
    dn = c * (1.0 - 0.5 / j.clamp(min=1.0))
    up[0], dn[0] = 4.0 * c, 0.0
    b = f[:-1, 1:-1].clone()
    b[:, 0] -= c * phi[:-1, 0]
    b[:, -1] -= c * phi[:-1, -1]
    b[-1] -= up[-1] * phi[-1, 1:-1]
    b = _dst(b, 1)
    diag = -(up + dn)[:, None] - _lam(nx)[None]
    cp, dp = torch.empty_like(b), torch.empty_like(b)
    cp[0], dp[0] = up[0] / diag[0], b[0] / diag[0]
    for r in range(1, ny - 1):
        den = diag[r] - dn[r] * cp[r - 1]
        cp[r], dp[r] = up[r] / den, (b[r] - dn[r] * dp[r - 1]) / den
    for r in range(ny - 3, -1, -1):
        dp[r] -= cp[r] * dp[r + 1]
    out = phi.clone()
    out[:-1, 1:-1] = _dst(dp, 1) * (2.0 / (nx - 1))
    return out


def _solve_masked(mask, phi, f):
    """lap(phi) = f on the free nodes of any mask: block elimination over columns."""
    ny, nx = phi.shape
    free = ~torch.as_tensor(mask, device="cuda").bool()
    c = 1.0 / (DX * DX)
    eye = torch.eye(ny, device="cuda", dtype=F8)
    off = c * (torch.diag(torch.ones(ny - 1, device="cuda", dtype=F8), 1) +
               torch.diag(torch.ones(ny - 1, device="cuda", dtype=F8), -1))
    inv, rhs = [], []
    for i in range(nx):
        fr = free[:, i:i + 1]
        D = torch.where(fr, off - 4.0 * c * eye, eye)
        r = torch.where(fr[:, 0], f[:, i], phi[:, i])
        w = fr[:, 0].to(F8) * c  # coupling to the columns beside it
        if i:
            P = inv[-1] * (free[:, i - 1].to(F8) * c)[None]
            D = D - w[:, None] * P
            r = r - w * (inv[-1] @ rhs[-1])
        inv.append(torch.linalg.inv(D))
        rhs.append(r)
    u = torch.empty_like(phi)
    u[:, -1] = inv[-1] @ rhs[-1]
    for i in range(nx - 2, -1, -1):
        u[:, i] = inv[i] @ (rhs[i] - free[:, i].to(F8) * c * u[:, i + 1])
    return u


def _grad(phi, rz=False):
    ex, ey = torch.empty_like(phi), torch.empty_like(phi)
    ex[:, 1:-1] = -(phi[:, 2:] - phi[:, :-2]) / (2 * DX)
    ex[:, 0], ex[:, -1] = -(phi[:, 1] - phi[:, 0]) / DX, -(phi[:, -1] - phi[:, -2]) / DX
    ey[1:-1] = -(phi[2:] - phi[:-2]) / (2 * DX)
    ey[0], ey[-1] = -(phi[1] - phi[0]) / DX, -(phi[-1] - phi[-2]) / DX
    if rz:
        ey[0] = 0.0
    return ex, ey


def _cell(x, y, nx, ny):
    i = x.detach().nan_to_num(0.0).clamp(0, nx - 2).floor().long()
    j = y.detach().nan_to_num(0.0).clamp(0, ny - 2).floor().long()
    return j * nx + i, x - i, y - j


def _corners(x, y, nx, ny):
    k, fx, fy = _cell(x, y, nx, ny)
    return [(k, (1 - fx) * (1 - fy)), (k + 1, fx * (1 - fy)), (k + nx, (1 - fx) * fy), (k + nx + 1, fx * fy)]


def _deposit(parts, nx, ny, scale):
    rho = torch.zeros(ny * nx, device="cuda", dtype=F8)
    for s, (x, y, *_) in enumerate(parts):
        live = ~torch.isnan(x.detach())
        for k, w in _corners(x, y, nx, ny):
            rho = rho.index_add(0, k, torch.where(live, w * scale[s], 0.0))
    return rho.reshape(ny, nx)


def _gather(e, x, y, nx, ny):
    return sum(w * e.reshape(-1)[k] for k, w in _corners(x, y, nx, ny))


def _absorb(p, nx, ny):
    out = ~((p[0] >= 0) & (p[0] <= nx - 1) & (p[1] >= 0) & (p[1] <= ny - 1))
    p[0][out] = p[1][out] = float("nan")


def _kick(parts, ex, ey, factor, nx, ny):
    for s, p in enumerate(parts):
        k = factor * CHARGE[s] / MASS[s] * DT
        live = ~torch.isnan(p[0])
        p[2] += torch.where(live, k * _gather(ex, p[0], p[1], nx, ny), 0.0)
        p[3] += torch.where(live, k * _gather(ey, p[0], p[1], nx, ny), 0.0)


def _drift(p, rz):
    h = DT / DX
    p[0] += p[2] * h
    if not rz:
        p[1] += p[3] * h
        return
    yr, yt = p[1] + p[3] * h, p[4] * h
    r = torch.sqrt(yr * yr + yt * yt)
    cs, sn = torch.where(r > 0, yr / r, 1.0), torch.where(r > 0, yt / r, 0.0)
    p[3], p[4], p[1] = cs * p[3] + sn * p[4], cs * p[4] - sn * p[3], r


def _tile_order(x, y, nx, ny):
    """The stable order of the tile-major cell sort."""
    cx, cy = x.long().clamp(max=nx - 2), y.long().clamp(max=ny - 2)
    tiles = (nx - 1 + TILE - 1) // TILE
    tx, ty = cx // TILE, cy // TILE
    return torch.argsort((ty * tiles + tx) * TILE * TILE + (cy - ty * TILE) * TILE + cx - tx * TILE, stable=True)


def _exact_step(c, seed, sort=True, particles=True, steps=None):
    nx, ny, rz = c["nx"], c["ny"], c["rz"]
    g = _gen(seed)
    counts = (c["n_e"], c["n_i"])
    parts = []
    for s in (0, 1):
        p = _species(g, s, counts[s], nx, ny, rz, c["blob"])
        if sort:
            order = _tile_order(p[0], p[1], nx, ny)
            p = [a[order] for a in p]
        parts.append([a.to(F8) for a in p])
    scale = [CHARGE[s] * _np2c(nx, ny, counts[s], rz) / (DX * DX) for s in (0, 1)]
    _, bc = _walls(nx, ny, c["left"], rz)
    phi = torch.as_tensor(bc, device="cuda")
    vol = torch.ones(ny, device="cuda", dtype=F8)
    if rz:
        j = torch.arange(ny, device="cuda", dtype=F8)
        vol = 2 * math.pi * j * DX
        vol[0], vol[-1] = math.pi * DX / 3, math.pi * ((ny - 1) * DX - DX / 3)

    def fields():
        rho = _deposit(parts, nx, ny, scale) / vol[:, None]
        u = (_solve_rz if rz else _solve_box)(phi, -rho / Consts.eps0)
        return rho, u, _grad(u, rz)

    rho, u, e = fields()
    _kick(parts, *e, -0.5, nx, ny)
    for k in range(c["steps"] if steps is None else steps):
        if k:
            _kick(parts, *e, 1.0, nx, ny)
        for p in parts:
            _drift(p, rz)
            _absorb(p, nx, ny)
        rho, u, e = fields()
    out = {"phi": u, "rho": rho, "Ex": e[0], "Ey": e[1]}
    out = {k: v.reshape(-1) for k, v in out.items()}
    if particles:
        out.update({f"{name}{s}": parts[s][i] for s in (0, 1) for i, name in enumerate(("x", "y", "vx", "vy", "vz"))})
    return out, parts, e


def _exact_adjoint(case, seed):
    sp, dvx, V, A, target = _adjoint_inputs(case, seed)
    m, n = case["nodes"], case["n"]
    V = V.cuda().requires_grad_()
    A = A.cuda().requires_grad_()
    w = _np2c(m, m, n) / (DX * DX)
    scale = [CHARGE[s] * w for s in (0, 1)]
    _, seg = adjoint.wall_segments(m, m)
    seg = torch.as_tensor(seg, device="cuda").long().reshape(m, m)
    parts = [[p[0], p[1], p[2], p[3]] for p in sp]
    parts[0][2] = parts[0][2] + A * dvx

    def field():
        edge = torch.where(seg >= 0, V[seg.clamp(min=0)], 0.0)
        u = _solve_box(edge, -_deposit(parts, m, m, scale) / Consts.eps0)
        return _grad(u)

    def kick(e, factor):
        for s, p in enumerate(parts):
            k = factor * CHARGE[s] / MASS[s] * DT
            live = ~torch.isnan(p[0].detach())
            for a in (0, 1):
                v = _gather(e[a], torch.where(live, p[0], 1.0), torch.where(live, p[1], 1.0), m, m)
                p[2 + a] = p[2 + a] + torch.where(live, k * v, 0.0)

    def step():
        for p in parts:
            x, y = p[0] + p[2] * (DT / DX), p[1] + p[3] * (DT / DX)
            with torch.no_grad():
                out = ~((x >= 0) & (x <= m - 1) & (y >= 0) & (y <= m - 1))
            p[0], p[1] = (torch.where(out, float("nan"), a) for a in (x, y))
        kick(field(), 1.0)

    kick(field(), -0.5)
    for _ in range(case["steps"]):
        step()
    dens = _deposit(parts[:1], m, m, [w])
    loss = ((dens.reshape(-1) - target) ** 2).mean()
    loss.backward()
    return {"loss": loss.detach(), "dV": V.grad, "dA": A.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        # collisions are random draws: no value without the library's stream
        return None if case["mcc"] else _exact_step(case, seed)[0]
    if kind == "ensemble":
        return [_exact_step(m, s, particles=False, steps=case["steps"])[0] for m, s in _member_cases(case, seed)]
    if kind == "dropin":
        c = _step("", case["nx"], case["ny"], case["n"], case["n"], left=case["left"], steps=1)
        out, parts, e = _exact_step(c, seed, sort=False)
        _kick(parts, *e, 1.0, case["nx"], case["ny"])
        res = {"phi": out["phi"], "rho": out["rho"], "E": torch.stack([out["Ex"], out["Ey"]])}
        res.update({f"{name}{s}": parts[s][i] for s in (0, 1) for i, name in enumerate(("x", "y", "vx", "vy"))})
        return res
    if kind == "mcc":
        return None
    if kind == "poisson":
        mask, phi, f = _poisson_inputs(case, seed)
        u = _solve_masked(mask, phi, f) if case["electrode"] else _solve_box(phi, f)
        return u.reshape(-1)
    if kind == "solver":
        nx, ny = case["nx"], case["ny"]
        rho = (_rhs(_gen(seed), nx, ny) * -Consts.eps0).to(F4).to(F8)
        _, bc = _walls(nx, ny, case["left"])
        u = _solve_box(torch.as_tensor(bc, device="cuda"), -rho / Consts.eps0)
        return {"phi": u.reshape(-1), "E": torch.stack([a.reshape(-1) for a in _grad(u)])}
    return _exact_adjoint(case, seed)
