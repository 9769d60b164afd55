"""Performance cases of the DG Euler solver: whole runs and resident marches over
the problem sizes it is used at, its single operators, the adjoint, and batches.

A case is a dict of plain values; ``prepare`` builds what a program holds before the
call (mesh, solver, initial state, all seeded), ``run`` makes one pass through the
public entry points, and ``exact`` evaluates the same pass in 64 bits with plain
torch, from the published scheme (degree-4 nodal DG on warp-and-blend nodes,
Cockburn-Shu troubled-cell limiter, Zhang-Shu positivity limiter, SSP-RK3).

Kinds:
  run        EulerSolver.run from a host state to a final time (the drop-in call)
  march      a resident state advanced by a number of CFL steps (begin_run + advance)
  operators  rhs, limit, time_step, cell_averages, integrate and step, called once each
             on a host state, as tests and diagnostics do
  adjoint    differentiable_run and its backward pass over a fixed schedule
  batch      BatchedEulerSolver.run over Riemann problems of uneven sizes
"""

from __future__ import annotations

import math

import numpy as np
import torch

GAMMA = 1.4
STRIP = ((0.0, 1.0), (0.0, 0.1))  # the shock-tube domain
UNIT = ((0.0, 1.0), (0.0, 1.0))
MESH_SEED = 20261203
FLUXES = ("rusanov", "roe", "hllc")
LIMITERS = ("minmod", "mc", "van_leer", "superbee", "unlimited")


def listed() -> list[dict]:
    def tube(name, kind, nx, ny, flux, limiter, precision, steps, **more):
        return dict(name=name, kind=kind, problem="tube", nx=nx, ny=ny, flux=flux, limiter=limiter,
                    precision=precision, steps=steps, **more)

    def fourier(name, nx, precision, steps, **more):
        return dict(name=name, kind="march", problem="fourier", nx=nx, ny=nx, flux="roe", limiter="unlimited",
                    precision=precision, steps=steps, tuned=False, **more)

    return [
        # a smoke-test sized shock tube, run as the README does: launches and latency only
        tube("run_tube_20x2_f64", "run", 20, 2, "rusanov", "minmod", "fp64", 40),
        # the verification shock tube (2,000 elements)
        tube("run_tube_100x10_f64", "run", 100, 10, "hllc", "van_leer", "fp64", 60),
        # every single operator once on the verification mesh, host arrays in and out
        tube("operators_100x10_f64", "operators", 100, 10, "roe", "mc", "fp64", 1),
        # the refined verification tube in the mixed form, advanced between outputs
        tube("march_tube_200x20_f32", "march", 200, 20, "roe", "superbee", "fp32_mixed", 64),
        # the sensitivity study's mesh (32,000 elements), a chunk of the run loop
        tube("march_tube_400x40_f32", "march", 400, 40, "hllc", "van_leer", "fp32_mixed", 32),
        # a sheared channel with exact far-field states (40,000 elements), supersonic
        dict(name="march_channel_200x100_f64", kind="march", problem="channel", nx=200, ny=100, flux="rusanov",
             limiter="minmod", precision="fp64", steps=32),
        # gradient of a schedule on the sensitivity mesh
        tube("adjoint_tube_400x40_f64", "adjoint", 400, 40, "rusanov", "minmod", "fp64", 10, checkpoint=5),
        # a family of Riemann problems of uneven sizes marched together, default form
        dict(name="batch_16_f32", kind="batch", problem="riemann", count=16, nx=50, ny=200, flux="hllc",
             limiter="superbee", precision="fp32_mixed", steps=40),
        # a mesh of odd size, ragged against every tile width (65,522 elements)
        fourier("march_fourier_181_f32", 181, "fp32_mixed", 24),
        # the precision study's mesh (800,000 elements)
        tube("march_tube_2000x200_f64", "march", 2000, 200, "hllc", "van_leer", "fp64", 6),
        # the 1M-triangle microbenchmark in both forms, stage shape tuned outside the march as the benchmark does
        dict(fourier("march_fourier_724_f32", 724, "fp32_mixed", 12), tuned=True),
        dict(fourier("march_fourier_724_f64", 724, "fp64", 8), tuned=True),
    ]


def draw(rng) -> dict:
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("run", "march", "march", "march", "operators", "adjoint", "batch"))
    case = dict(kind=kind, flux=rng.choice(FLUXES), limiter=rng.choice(LIMITERS),
                precision=rng.choice(("fp64", "fp32_mixed")))
    if kind == "batch":
        lo = logint(17, 80)
        return dict(case, problem="riemann", count=logint(3, 20), nx=lo, ny=lo + logint(20, 150),
                    precision="fp32_mixed", steps=logint(10, 40))
    if kind == "march":
        case["problem"] = rng.choice(("tube", "fourier", "channel"))
        nx = logint(15, 1800) if case["problem"] == "tube" else logint(9, 600 if case["problem"] == "fourier" else 260)
        ny = {"tube": max(1, nx // 10), "fourier": max(3, nx - rng.randrange(0, 1 + nx // 3)),
              "channel": max(2, nx // 2 + rng.randrange(0, 3))}[case["problem"]]
        case["limiter"] = "unlimited" if case["problem"] == "fourier" and rng.random() < 0.5 else case["limiter"]
        case.update(tuned=False)
    else:
        nx = logint(12, 260 if kind != "adjoint" else 400)
        ny = max(1, nx // 10 + rng.randrange(0, 2))
        case.update(problem="tube", precision="fp64")
    case.update(nx=nx, ny=ny)
    top = {"run": 60, "march": 64, "operators": 1, "adjoint": 10}[kind]
    case["steps"] = max(1, min(top, int(4.0e6 / (2 * nx * ny)), logint(1, top)))
    if kind == "adjoint":
        case["checkpoint"] = rng.randrange(1, case["steps"] + 1)
    return case


# ---------------------------------------------------------------- problems ---
def conserved(rho, u, v, p, xp=np):
    return xp.stack([rho, rho * u, rho * v, p / (GAMMA - 1.0) + 0.5 * rho * (u * u + v * v)], -1)


def fourier_mode_sum(x, y, rng, lo, hi, modes=8):
    """A seeded sum of Fourier modes of the coordinates, within [lo, hi]."""
    f, total = torch.zeros_like(x), 0.0
    for _ in range(modes):
        kx, ky = rng.integers(1, 5, size=2)
        amp = rng.uniform(0.3, 1.0)
        f += amp * torch.cos(2 * math.pi * (float(kx) * x + float(ky) * y) + rng.uniform(0.0, 2 * math.pi))
        total += amp
    return 0.5 * (lo + hi) + 0.5 * (hi - lo) / total * f


def channel_flow(x, y):
    """Supersonic flow with a smooth wave, the channel's far field (numpy)."""
    w = 0.05 * np.sin(3.0 * x + 5.0 * y)
    return conserved(1.0 + w, 2.0 + 0.0 * w, 0.3 + w, 1.0 / GAMMA + w)


def tube_states(case, seed):
    """Left and right primitive states near Sod's, each seed its own."""
    u = np.random.default_rng((seed, 11)).uniform(0.9, 1.1, size=4)
    return (float(u[0]), 0.0, 0.0, float(u[1])), (0.125 * float(u[2]), 0.0, 0.0, 0.1 * float(u[3]))


def riemann_problems(case, seed):
    """(nx, ny, left, right) of each problem of a batch; the sizes belong to the case."""
    sizes = np.random.default_rng((MESH_SEED, case["count"], case["nx"], case["ny"]))
    values = np.random.default_rng((seed, 12))
    out = []
    for _ in range(case["count"]):
        nx = int(sizes.integers(case["nx"], case["ny"] + 1))
        rl, rr, pl, pr = (float(a) for a in values.uniform(0.4, 1.0, size=4))
        out.append((nx, max(1, nx // 10), (rl, 0.0, 0.0, pl), (rr, 0.0, 0.0, pr)))
    return out


def final_time(case):
    """About `steps` CFL steps of a shock tube of nx cells (of the finest one of a batch)."""
    nx = case["ny"] if case["kind"] == "batch" else case["nx"]
    return 5.0e-3 * case["steps"] / nx


def box(case):
    return {"tube": STRIP, "channel": ((0.0, 1.0), (0.0, 0.5)), "fourier": UNIT}[case["problem"]]


def split_state(corners, left, right):
    """(15, K, 4): the left state where the element's centroid has x < 0.5, else the right one."""
    sides = np.stack([conserved(*(np.float64(a) for a in s)) for s in (left, right)])
    e = sides[(corners[:, :, 0].mean(axis=1) >= 0.5).astype(int)]
    return np.broadcast_to(e[None], (15,) + e.shape).copy()


def initial_state(case, seed, corners):
    """(15, K, 4) float64 state on the elements with these corners (K, 3, 2): a CUDA tensor, or a
    NumPy array for the kinds that take host data."""
    if case["problem"] == "tube" and case["kind"] != "operators":
        left, right = tube_states(case, seed)
        q = split_state(corners, left, right)
        return q if case["kind"] == "run" else torch.from_numpy(q).cuda()
    ref = reference()
    c = torch.as_tensor(np.ascontiguousarray(corners), device="cuda")
    w = torch.tensor(np.stack([-(ref["r"] + ref["s"]) / 2, (1 + ref["r"]) / 2, (1 + ref["s"]) / 2], -1), device="cuda")
    x, y = (torch.einsum("nv,kv->nk", w, c[:, :, d]) for d in range(2))
    rng = np.random.default_rng((seed, 13))
    if case["problem"] == "channel":
        q = torch.from_numpy(channel_flow(x.cpu().numpy(), y.cpu().numpy())).cuda()
        return q * (1.0 + fourier_mode_sum(x, y, rng, -0.02, 0.02))[..., None]
    ranges = ((0.5, 1.5), (-0.5, 0.5), (-0.5, 0.5), (0.5, 1.5))
    rho, u, v, p = (fourier_mode_sum(x, y, rng, lo, hi) for lo, hi in ranges)
    if case["kind"] == "operators":  # a developed flow: a jump across the tube on top of the waves
        rho, p = (torch.where(x < 0.5, f, 0.3 * f) for f in (rho, p))
        return conserved(rho, u, v, p, torch).cpu().numpy()
    return conserved(rho, u, v, p, torch).contiguous()


def boundaries(case, seed):
    """tag -> ("wall",), ("fixed", conserved state) or ("exact", function)."""
    if case["problem"] == "tube":
        left, right = (conserved(*(np.float64(a) for a in s)) for s in tube_states(case, seed))
        return {"left": ("fixed", left), "right": ("fixed", right), "bottom": ("wall",), "top": ("wall",)}
    if case["problem"] == "channel":
        inflow = conserved(*(np.float64(a) for a in (1.0, 2.0, 0.3, 1.0 / GAMMA)))
        return {"left": ("fixed", inflow), "bottom": ("wall",), "top": ("exact", channel_flow),
                "right": ("exact", channel_flow)}
    mean = conserved(*(np.float64(a) for a in (1.0, 0.0, 0.0, 1.0)))
    return {t: ("fixed", mean) for t in ("left", "right", "bottom", "top")}


# ------------------------------------------------------- the measured calls ---
def prepare(case: dict, seed: int) -> dict:
    from cfd_demo_b200 import (EulerSolver, ExactState, FixedState, SlipWall, SolverConfig, rectangle_mesh,
                               sheared_rectangle_mesh)
    from cfd_demo_b200.mesh import jittered_rectangle_mesh

    config = SolverConfig(flux=case["flux"], limiter=case["limiter"], gamma=GAMMA, precision=case["precision"])
    if case["kind"] == "batch":
        from cfd_demo_b200.batch import BatchCase, BatchedEulerSolver

        parts = []
        for nx, ny, left, right in riemann_problems(case, seed):
            mesh = rectangle_mesh(nx, ny, *STRIP)
            bcs = {"left": FixedState.from_primitive(*left, GAMMA), "right": FixedState.from_primitive(*right, GAMMA),
                   "bottom": SlipWall(), "top": SlipWall()}
            parts.append(BatchCase(mesh, bcs, split_state(mesh.vertices[mesh.elements], left, right)))
        return {"case": case, "batch": BatchedEulerSolver(parts, config), "time": final_time(case)}

    if case["problem"] == "channel":
        mesh = sheared_rectangle_mesh(case["nx"], case["ny"], 0.15, *box(case))
    elif case["problem"] == "fourier":
        mesh = jittered_rectangle_mesh(case["nx"], case["ny"], 0.2, MESH_SEED)
    else:
        mesh = rectangle_mesh(case["nx"], case["ny"], *box(case))
    make = {"wall": lambda: SlipWall(), "fixed": lambda q: FixedState(tuple(float(a) for a in q)),
            "exact": lambda f: ExactState(f)}
    bcs = {tag: make[b[0]](*b[1:]) for tag, b in boundaries(case, seed).items()}
    solver = EulerSolver(mesh, bcs, config)
    state = {"case": case, "solver": solver, "q": initial_state(case, seed, mesh.vertices[mesh.elements])}
    if case["kind"] == "run":
        state["time"] = final_time(case)
    if case["kind"] == "operators":
        state["dt"] = 0.02 / (case["nx"] * 25)
    if case["kind"] == "adjoint":
        from cfd_demo_b200.adjoint import AdjointRun, cfl_schedule

        dts = cfl_schedule(solver, state["q"].cpu().numpy(), steps=case["steps"])
        state["runner"] = AdjointRun(solver, dts, checkpoint_every=case["checkpoint"])
        state["bc"] = solver.operators.bc_states.clone().requires_grad_(True)
        x = torch.as_tensor(mesh.vertices[mesh.elements].mean(axis=1)[:, 0], device="cuda")
        state["weight"] = torch.exp(-(((x - 0.5) / 0.1) ** 2))
        state["q"].requires_grad_(True)
    if case.get("tuned"):
        from cfd_demo_b200.autotune import autotune

        autotune(solver, state["q"])
    return state


def run(state: dict):
    kind = state["case"]["kind"]
    if kind == "batch":
        return [{"state": r.state.astype(np.float32), "steps": r.steps} for r in state["batch"].run(final_time=state["time"])]
    solver, q = state["solver"], state["q"]
    if kind == "run":
        r = solver.run(q, state["time"])
        return {"state": r.state, "steps": r.steps, "rejected": r.rejected_steps, "flux": r.boundary_flux_integral,
                "minima": np.array([r.min_density, r.min_pressure]), "troubled": r.max_troubled_cells}
    if kind == "march":
        solver.begin_run(q, math.inf)
        c = solver.advance(state["case"]["steps"])
        x = solver.state_tensor()
        return {"state": x, "steps": int(c.steps), "rejected": int(c.rejected),
                "times": torch.tensor([c.time, c.dt], dtype=x.dtype),
                "flux": torch.tensor(c.flux_integral[:], dtype=x.dtype),
                "minima": torch.tensor([c.min_density, c.min_pressure], dtype=x.dtype)}
    if kind == "operators":
        rhs, bflux = solver.rhs(q)
        new, report = solver.step(q, state["dt"])
        return {"rhs": rhs, "bflux": bflux, "limited": solver.limit(q), "dt": solver.time_step(q),
                "averages": solver.cell_averages(q), "integral": solver.integrate(q), "new": new,
                "flux": report.boundary_flux, "minima": np.array([report.min_density, report.min_pressure]),
                "troubled": report.troubled_cells}
    from cfd_demo_b200.adjoint import differentiable_run

    state["q"].grad = state["bc"].grad = None
    final = differentiable_run(state["runner"], state["q"], state["bc"])
    (final[..., 0] * state["weight"]).sum().backward()
    return {"final": final.detach(), "grad": state["q"].grad, "bc_grad": state["bc"].grad}


def work(case: dict) -> dict:
    """Per step an element's state is read and written once and its geometry read once (13 reals,
    4 indices); a stage is about 8,000 operations an element (two 15x15 contractions of 4 variables,
    their fluxes, 15 face fluxes, LIFT, the combine, averages and limiter tests)."""
    size = 4 if case["precision"] == "fp32_mixed" else 8
    per_step = 2 * 60 * size + 13 * size + 16
    steps = case["steps"]
    if case["kind"] == "batch":
        parts = riemann_problems(case, 0)
        per = [(2 * nx * ny, max(1.0, steps * nx / case["ny"])) for nx, ny, _, _ in parts]
    else:
        per = [(2 * case["nx"] * case["ny"], steps)]
    element_steps = sum(k * n for k, n in per)
    if case["kind"] == "adjoint":  # forward, forward again with the tape, reverse
        return {"bytes": 3.0 * element_steps * per_step, "flops": 5.0 * element_steps * 24000}
    if case["kind"] == "operators":
        k = per[0][0]
        return {"bytes": float(k * (9 * 480 + 32 + 6 * 120)), "flops": float(k * (4 * 8000 + 2000))}
    return {"bytes": float(element_steps * per_step), "flops": float(element_steps * 24000)}


# --------------------------------------- the same scheme in 64 bits, in torch ---
_REFERENCE: dict = {}


def reference() -> dict:
    """Nodes and operators of the degree-4 reference triangle (-1,-1), (1,-1), (-1,1) on
    warp-and-blend nodes (Hesthaven & Warburton 2008, section 6.1), rows in s, increasing r."""
    if _REFERENCE:
        return _REFERENCE
    n = 4
    gll = np.array([-1.0, -math.sqrt(3.0 / 7.0), 0.0, math.sqrt(3.0 / 7.0), 1.0])
    even = np.linspace(-1.0, 1.0, n + 1)
    shift = np.linalg.solve(np.vander(even), gll - even)

    def warp(t):
        inner = (np.abs(t) < 1.0 - 1e-10).astype(float)
        w = np.polyval(shift, t)
        return w / (1.0 - (inner * t) ** 2) + w * (inner - 1.0)

    b1 = np.array([i / n for i in range(n + 1) for _ in range(n + 1 - i)])
    b3 = np.array([m / n for i in range(n + 1) for m in range(n + 1 - i)])
    b2 = 1.0 - b1 - b3
    x, y = b3 - b2, (2 * b1 - b2 - b3) / math.sqrt(3.0)
    for k, (p, q, o) in enumerate(((b2, b3, b1), (b3, b1, b2), (b1, b2, b3))):
        w = 4 * p * q * warp(q - p) * (1 + (0.1001 * o) ** 2)
        x, y = x + math.cos(2 * math.pi * k / 3) * w, y + math.sin(2 * math.pi * k / 3) * w
    l1 = (math.sqrt(3.0) * y + 1) / 3
    l2, l3 = ((-3 * x - math.sqrt(3.0) * y + 2) / 6, (3 * x - math.sqrt(3.0) * y + 2) / 6)
    r, s = l3 - l2 - l1, l1 - l2 - l3
    # products of Legendre polynomials; integrals by Gauss quadrature, on the triangle folded from a square
    leg, eye = np.polynomial.legendre, np.eye(n + 1)
    powers = [(i, j) for i in range(n + 1) for j in range(n + 1 - i)]
    table = lambda t, d=0: leg.legval(t, leg.legder(eye, d) if d else eye)  # (degree, points)  # noqa: E731
    product = lambda p, q: np.stack([p[i] * q[j] for i, j in powers], -1)  # noqa: E731
    inv = np.linalg.inv(product(table(r), table(s)))
    va, vb = product(table(r, 1), table(s)), product(table(r), table(s, 1))
    gx, gw = leg.leggauss(8)
    ga, gb = (m.ravel() for m in np.meshgrid(gx, gx))
    fold = product(table((1 + ga) * (1 - gb) / 2 - 1), table(gb)) @ inv
    mass = fold.T @ ((np.outer(gw, gw).ravel() * (1 - gb) / 2)[:, None] * fold)
    line = table(gx).T @ np.linalg.inv(table(gll).T)
    edge = line.T @ (gw[:, None] * line)
    faces = np.stack([np.flatnonzero(np.abs(m) < 1e-9) for m in (s + 1, r + s, r + 1)])
    lifted = np.zeros((15, 15))
    for f in range(3):
        lifted[faces[f], 5 * f:5 * f + 5] = edge
    plane = np.stack([np.ones(15), r, s], -1)
    project = plane @ np.linalg.solve(plane.T @ mass @ plane, plane.T @ mass)
    _REFERENCE.update(r=r, s=s, dr=va @ inv, ds=vb @ inv, lift=np.linalg.solve(mass, lifted), faces=faces,
                      weights=mass.sum(0), edge_weights=edge.sum(1), mids=faces[:, 2], project=project[faces[:, 2]],
                      linear=np.stack([-s, 1 + r + s, -r], -1))
    return _REFERENCE


def plain_mesh(case, nx, ny):
    """Corners (K, 3, 2) and elements (K, 3) of the case's mesh: nx x ny cells cut along the diagonal
    from the lower left, jittered or sheared as the case's problem has it."""
    (x0, x1), (y0, y1) = STRIP if case["kind"] == "batch" else box(case)
    gx, gy = np.meshgrid(x0 + (x1 - x0) * (np.arange(nx + 1) / nx), y0 + (y1 - y0) * (np.arange(ny + 1) / ny))
    v = np.stack([gx.ravel(), gy.ravel()], -1)
    if case["problem"] == "fourier":
        d = np.random.default_rng(MESH_SEED).uniform(-1.0, 1.0, size=v.shape)
        inside = (np.abs(v - 0.5) < 0.5 - 1e-12).all(axis=1)
        v[inside] += 0.2 * d[inside] * np.array([1.0 / nx, 1.0 / ny])
    if case["problem"] == "channel":
        v[:, 1] += v[:, 0] * np.tan(0.15)
    ci, cj = (m.ravel() for m in np.meshgrid(np.arange(nx), np.arange(ny)))
    a = cj * (nx + 1) + ci
    e = np.stack([np.stack([a, a + 1, a + nx + 2], -1), np.stack([a, a + nx + 2, a + nx + 1], -1)], 1).reshape(-1, 3)
    return v[e], e, v


class Plain:
    """The scheme on one mesh, float64 torch tensors (15, K, 4)."""

    def __init__(self, case, nx, ny, bounds):
        dev, ref = "cuda", reference()
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)  # noqa: E731
        self.flux, self.limiter = case["flux"], case["limiter"]
        corners, elems, verts = plain_mesh(case, nx, ny)
        k = len(elems)
        self.ref = {n: t(a) for n, a in ref.items()}
        nxt = np.roll(corners, -1, 1)
        d = nxt - corners
        length = np.hypot(d[..., 0], d[..., 1])
        (xr, yr), (xs, ys) = (0.5 * (corners[:, i] - corners[:, 0]).T for i in (1, 2))
        jac = xr * ys - xs * yr
        normal = np.stack([d[..., 1], -d[..., 0]], -1) / length[..., None]
        self.metric = [t(m)[None, :, None] for m in (ys / jac, -xs / jac, -yr / jac, xr / jac)]
        self.jac = t(jac)
        self.dt_geometry = t((4.0 * jac[:, None] / (25.0 * length)).min(1))
        # faces matched by their vertex pairs
        ends = np.sort(np.stack([elems, np.roll(elems, -1, 1)], -1).reshape(-1, 2), 1)
        code = ends[:, 0] * len(verts) + ends[:, 1]
        order = np.argsort(code, kind="stable")
        same = np.flatnonzero(code[order][1:] == code[order][:-1])
        other = np.full(3 * k, -1)
        other[order[same]], other[order[same + 1]] = order[same + 1], order[same]
        other = other.reshape(k, 3)
        nb, nf = np.where(other >= 0, other // 3, np.arange(k)[:, None]), np.where(other >= 0, other % 3, 0)
        # boundary tags by position in the unjittered, unsheared box
        gi, gj = np.arange(len(verts)) % (nx + 1), np.arange(len(verts)) // (nx + 1)
        at = {"left": gi == 0, "right": gi == nx, "bottom": gj == 0, "top": gj == ny}
        wall, fixed = np.zeros((k, 3), bool), np.zeros((k, 3), bool)
        outside, ghost = np.zeros((k, 3, 5, 4)), np.zeros((k, 3, 4))
        w = np.stack([-(ref["r"] + ref["s"]) / 2, (1 + ref["r"]) / 2, (1 + ref["s"]) / 2], -1)
        for tag, b in bounds.items():
            m = (other < 0) & at[tag][elems] & at[tag][np.roll(elems, -1, 1)]
            if b[0] == "wall":
                wall |= m
                continue
            fixed |= m
            if b[0] == "fixed":
                outside[m], ghost[m] = b[1], b[1]
                continue
            es, fs = np.nonzero(m)
            pts = np.einsum("nkv,nvd->nkd", w[ref["faces"][fs]], corners[es])
            outside[es, fs] = b[1](pts[..., 0], pts[..., 1])
            ghost[es, fs] = self.reflected_average(b[1], corners[es], corners[es, fs], normal[es, fs])
        kk = np.where(((np.arange(3) == 2) != (nf == 2))[..., None], np.arange(5), 4 - np.arange(5))  # (K, 3, 5)
        partner = ref["faces"][nf[..., None], kk]
        per_node = lambda a: t(np.repeat(np.moveaxis(a, 1, 0), 5, 0))  # (K, 3, ...) -> (15, K, ...)  # noqa: E731
        self.face_nodes = t(ref["faces"].ravel())
        self.partner = t((partner * k + nb[..., None]).transpose(1, 2, 0).reshape(15, k))
        self.nx, self.ny = per_node(normal[..., 0]), per_node(normal[..., 1])
        self.fscale = per_node(0.5 * length / jac[:, None])[..., None]
        self.wall, self.fixed = per_node(wall)[..., None], per_node(fixed)[..., None]
        self.outside = t(outside.transpose(1, 2, 0, 3).reshape(15, k, 4))
        self.bweight = per_node(0.5 * length * (other < 0)) * t(np.tile(ref["edge_weights"], 3))[:, None]
        # limiter: neighbours, ghosts, Cockburn-Shu coefficients
        cen, mid = corners.mean(1), 0.5 * (corners + nxt)
        reflect = cen[:, None] + 2.0 * ((mid - cen[:, None]) * normal).sum(-1, keepdims=True) * normal
        to, half = np.where((other >= 0)[..., None], cen[nb], reflect) - cen[:, None], mid - cen[:, None]
        alpha, beta, pair = np.zeros((k, 3)), np.zeros((k, 3)), np.full((k, 3), -1)
        for f in range(3):
            for o in ((f + 1) % 3, (f + 2) % 3):
                det = to[:, f, 0] * to[:, o, 1] - to[:, f, 1] * to[:, o, 0]
                safe = np.where(det == 0.0, 1.0, det)
                ca = (half[:, f, 0] * to[:, o, 1] - half[:, f, 1] * to[:, o, 0]) / safe
                cb = (to[:, f, 0] * half[:, f, 1] - to[:, f, 1] * half[:, f, 0]) / safe
                ok = (det != 0.0) & (ca >= -1e-12) & (cb >= -1e-12) & (pair[:, f] < 0)
                alpha[ok, f], beta[ok, f], pair[ok, f] = np.maximum(ca[ok], 0), np.maximum(cb[ok], 0), o
        self.nb3, self.alpha, self.beta, self.pair = (t(a.T) for a in (nb, alpha, beta, pair))
        self.wall3, self.fixed3, self.ghost3 = t(wall.T)[..., None], t(fixed.T)[..., None], t(np.moveaxis(ghost, 1, 0))
        self.nx3, self.ny3 = t(normal[..., 0].T), t(normal[..., 1].T)

    @staticmethod
    def reflected_average(function, corners, on, normal, cuts=32):
        """Mean of the function over the centroids of cuts**2 parts of each triangle reflected across its face."""
        tri = corners - 2.0 * np.einsum("nvd,nd->nv", corners - on[:, None], normal)[..., None] * normal[:, None]
        i, j = (m.ravel() for m in np.meshgrid(np.arange(cuts), np.arange(cuts)))
        lam = np.concatenate([np.stack([i, j], -1)[i + j < cuts] + 1 / 3, np.stack([i, j], -1)[i + j < cuts - 1] + 2 / 3]) / cuts
        p = tri[:, None, 0] + lam[None, :, :1] * (tri[:, 1] - tri[:, 0])[:, None] + lam[None, :, 1:] * (tri[:, 2] - tri[:, 0])[:, None]
        return function(p[..., 0], p[..., 1]).mean(1)

    @staticmethod
    def primitive(q):
        u, v = q[..., 1] / q[..., 0], q[..., 2] / q[..., 0]
        return q[..., 0], u, v, (GAMMA - 1.0) * (q[..., 3] - 0.5 * (q[..., 1] * u + q[..., 2] * v))

    @staticmethod
    def along(q, w, nx, ny):
        _, u, v, p = w
        un = u * nx + v * ny
        return torch.stack([q[..., 0] * un, q[..., 1] * un + p * nx, q[..., 2] * un + p * ny, (q[..., 3] + p) * un], -1)

    @staticmethod
    def mirror(q, nx, ny):
        m = 2.0 * (q[..., 1] * nx + q[..., 2] * ny)
        return q - torch.stack([torch.zeros_like(m), m * nx, m * ny, torch.zeros_like(m)], -1)

    def interface(self, qm, qp):
        nx, ny = self.nx, self.ny
        wm, wp = self.primitive(qm), self.primitive(qp)
        (rm, um, vm, pm), (rp, up, vp, pp) = wm, wp
        fm, fp = self.along(qm, wm, nx, ny), self.along(qp, wp, nx, ny)
        unm, unp = um * nx + vm * ny, up * nx + vp * ny
        cm, cp = (GAMMA * pm / rm).sqrt(), (GAMMA * pp / rp).sqrt()
        if self.flux == "rusanov":
            return 0.5 * (fm + fp) - 0.5 * torch.maximum(unm.abs() + cm, unp.abs() + cp)[..., None] * (qp - qm)
        sm, sp = rm.sqrt(), rp.sqrt()
        mean = lambda a, b: (sm * a + sp * b) / (sm + sp)  # noqa: E731
        u, v, h = mean(um, up), mean(vm, vp), mean((qm[..., 3] + pm) / rm, (qp[..., 3] + pp) / rp)
        c = ((GAMMA - 1.0) * (h - 0.5 * (u * u + v * v))).sqrt()
        un, ut = u * nx + v * ny, v * nx - u * ny
        if self.flux == "roe":
            dp, dun, rho = pp - pm, unp - unm, sm * sp
            delta = 0.1 * (un.abs() + c)
            fixed = lambda s: torch.where(s.abs() < delta, (s * s + delta * delta) / (2.0 * delta), s.abs())  # noqa: E731
            back = fixed(un - c) * (dp - rho * c * dun) / (2.0 * c * c)
            ahead = fixed(un + c) * (dp + rho * c * dun) / (2.0 * c * c)
            entropy = un.abs() * (rp - rm - dp / (c * c))
            shear = un.abs() * rho * ((vp - vm) * nx - (up - um) * ny)
            diss = torch.stack([back + entropy + ahead,
                                back * (u - c * nx) + entropy * u - shear * ny + ahead * (u + c * nx),
                                back * (v - c * ny) + entropy * v + shear * nx + ahead * (v + c * ny),
                                back * (h - c * un) + entropy * 0.5 * (u * u + v * v) + shear * ut + ahead * (h + c * un)], -1)
            return 0.5 * (fm + fp) - 0.5 * diss
        s_m, s_p = torch.minimum(unm - cm, un - c), torch.maximum(unp + cp, un + c)
        mm, mp = rm * (s_m - unm), rp * (s_p - unp)
        safe = lambda a: torch.where(a == 0.0, torch.full_like(a, np.finfo(float).tiny), a)  # noqa: E731
        star = (pp - pm + mm * unm - mp * unp) / safe(mm - mp)

        def inside(q, f, w, unk, sk, mk):
            rk, uk, vk, pk = w
            sh, fac = star - unk, mk / safe(sk - star)
            st = torch.stack([torch.ones_like(rk), uk + sh * nx, vk + sh * ny, q[..., 3] / rk + sh * (star + pk / safe(mk))], -1)
            return f + sk[..., None] * (fac[..., None] * st - q)

        f_m, f_p = inside(qm, fm, wm, unm, s_m, mm), inside(qp, fp, wp, unp, s_p, mp)
        return torch.where((s_m >= 0)[..., None], fm,
                           torch.where((star >= 0)[..., None], f_m, torch.where((s_p > 0)[..., None], f_p, fp)))

    def rhs(self, q):
        rho, u, v, p = self.primitive(q)
        e = q[..., 3] + p
        f = torch.stack([q[..., 1], q[..., 1] * u + p, q[..., 2] * u, e * u], -1)
        g = torch.stack([q[..., 2], q[..., 1] * v, q[..., 2] * v + p, e * v], -1)
        rx, ry, sx, sy = self.metric
        out = -torch.einsum("ij,jkc->ikc", self.ref["dr"], rx * f + ry * g)
        out -= torch.einsum("ij,jkc->ikc", self.ref["ds"], sx * f + sy * g)
        qm = q[self.face_nodes]
        qp = torch.where(self.wall, self.mirror(qm, self.nx, self.ny),
                         torch.where(self.fixed, self.outside, q.reshape(-1, 4)[self.partner]))
        hat = self.interface(qm, qp)
        jump = self.fscale * (self.along(qm, self.primitive(qm), self.nx, self.ny) - hat)
        return out + torch.einsum("ij,jkc->ikc", self.ref["lift"], jump), torch.einsum("jk,jkc->c", self.bweight, hat)

    def averages(self, q):
        return torch.einsum("i,ikc->kc", self.ref["weights"] / 2.0, q)

    def phi(self, r):
        one, zero = torch.ones_like(r), torch.zeros_like(r)
        if self.limiter == "minmod":
            return torch.maximum(zero, torch.minimum(one, r))
        if self.limiter == "mc":
            return torch.maximum(zero, torch.minimum(torch.minimum(2 * r, 0.5 * (1 + r)), 2 * one))
        if self.limiter == "van_leer":
            return (r + r.abs()) / (1 + r.abs())
        return torch.maximum(zero, torch.maximum(torch.minimum(2 * r, one), torch.minimum(r, 2 * one)))

    def limit(self, q):
        """(limited state, number of troubled cells)."""
        avg, count = self.averages(q), 0
        if self.limiter != "unlimited":
            near = torch.where(self.wall3, self.mirror(avg.expand(3, -1, -1), self.nx3, self.ny3),
                               torch.where(self.fixed3, self.ghost3, avg[self.nb3]))
            diff = near - avg
            paired = torch.gather(diff, 0, self.pair[..., None].expand(-1, -1, 4))
            scaled = 1.5 * (self.alpha[..., None] * diff + self.beta[..., None] * paired)
            trace = q[self.ref["mids"]] - avg
            bounded = torch.where(trace * scaled > 0, trace.sign() * torch.minimum(trace.abs(), scaled.abs()), 0.0)
            troubled = ((bounded - trace).abs()[..., [0, 3]] > 1e-10 * avg[:, [0, 3]].abs()).any(2).any(0)
            count = int(troubled.sum())
            e = torch.nonzero(troubled).reshape(-1)
            if len(e):
                a, sc = avg[e], scaled[:, e]
                pr = torch.einsum("fi,ikc->fkc", self.ref["project"], q[:, e]) - a
                d = torch.where(pr != 0, pr * self.phi(sc / torch.where(pr != 0, pr, 1.0)).clamp(max=1.0), 0.0)
                up, down = d.clamp(min=0).sum(0), (-d).clamp(min=0).sum(0)
                tu = torch.where(up > 0, (down / torch.where(up > 0, up, 1.0)).clamp(max=1.0), 0.0)
                td = torch.where(down > 0, (up / torch.where(down > 0, down, 1.0)).clamp(max=1.0), 0.0)
                d = tu * d.clamp(min=0) - td * (-d).clamp(min=0)
                q = q.clone()
                q[:, e] = a + torch.einsum("if,fkc->ikc", self.ref["linear"], d)
        return self.positive(q, avg), count

    def positive(self, q, avg):
        low = torch.minimum(torch.minimum(avg[:, 0], self.primitive(avg)[3]), torch.full_like(avg[:, 0], 1e-13))
        thin = q[..., 0].amin(0)
        e = torch.nonzero(thin < low).reshape(-1)
        if len(e):
            q = q.clone()
            theta = ((avg[e, 0] - low[e]) / (avg[e, 0] - thin[e])).clamp(0.0, 1.0)
            q[:, e] = avg[e] + theta[None, :, None] * (q[:, e] - avg[e])
        bad = self.primitive(q)[3] < low
        e = torch.nonzero(bad.any(0)).reshape(-1)
        if len(e):
            q, a, need = q.clone(), avg[e], bad[:, e]
            dev = q[:, e] - a
            lo, hi = torch.zeros_like(dev[..., 0]), torch.ones_like(dev[..., 0])
            for _ in range(60):
                mid = 0.5 * (lo + hi)
                ok = self.primitive(a + mid[..., None] * dev)[3] >= low[e]
                lo, hi = torch.where(ok, mid, lo), torch.where(ok, hi, mid)
            theta = torch.where(need, lo, 1.0).amin(0)
            q[:, e] = torch.where((theta < 1)[None, :, None], a + theta[None, :, None] * dev, q[:, e])
        return q

    def time_step(self, q):
        rho, u, v, p = self.primitive(q)
        speed = ((u * u + v * v).sqrt() + (GAMMA * p / rho).sqrt()).amax(0)
        return 0.5 * float((self.dt_geometry / speed).min())

    def step(self, q, dt):
        """(new state, boundary flux, [min density, min pressure], most troubled cells of a stage)."""
        total, low, most, x = 0.0, [math.inf, math.inf], 0, q
        for k, weight in enumerate((1.0 / 6.0, 1.0 / 6.0, 2.0 / 3.0)):
            r, b = self.rhs(x)
            x = x + dt * r
            x = x if k == 0 else 0.75 * q + 0.25 * x if k == 1 else q / 3.0 + 2.0 * x / 3.0
            x, count = self.limit(x)
            total, most = total + dt * weight * b, max(most, count)
            low = [min(low[0], float(x[..., 0].min())), min(low[1], float(self.primitive(x)[3].min()))]
        return x, total, low, most

    def march(self, q, *, steps=None, until=math.inf):
        """Like step over a run with its own time steps; also the time reached, the steps and the next step size."""
        t, n, total, most = 0.0, 0, torch.zeros(4, dtype=q.dtype, device=q.device), 0
        low = [float(q[..., 0].min()), float(self.primitive(q)[3].min())]
        dt = self.time_step(q)
        while t < until and (steps is None or n < steps):
            last = dt >= until - t
            dt = until - t if last else dt
            q, b, m, count = self.step(q, dt)
            t, n, total, low, most = until if last else t + dt, n + 1, total + b, list(map(min, low, m)), max(most, count)
            dt = self.time_step(q)
        return q, total, low, most, t, n, dt


def exact(case: dict, seed: int):
    if case["kind"] == "batch":
        out = []
        for nx, ny, left, right in riemann_problems(case, seed):
            ends = {t: ("fixed", conserved(*(np.float64(a) for a in s))) for t, s in (("left", left), ("right", right))}
            plain = Plain(case, nx, ny, {**ends, "bottom": ("wall",), "top": ("wall",)})
            q = torch.from_numpy(split_state(plain_mesh(case, nx, ny)[0], left, right)).cuda()
            out.append({"state": plain.march(q, until=final_time(case))[0], "steps": None})
        return out
    plain = Plain(case, case["nx"], case["ny"], boundaries(case, seed))
    q = initial_state(case, seed, plain_mesh(case, case["nx"], case["ny"])[0])
    q = torch.from_numpy(q).cuda() if isinstance(q, np.ndarray) else q
    if case["kind"] == "run":
        x, flux, low, most, _, n, _ = plain.march(q, until=final_time(case))
        return {"state": x, "steps": n, "rejected": 0, "flux": flux, "minima": np.array(low), "troubled": None}
    if case["kind"] == "march":
        x, flux, low, _, t, n, dt = plain.march(q, steps=case["steps"])
        k = x.shape[1]
        out = torch.zeros((4, 15, (k + 63) // 64 * 64), dtype=torch.float64, device=x.device)
        out[..., :k] = x.permute(2, 0, 1)
        return {"state": out.reshape(60, -1), "steps": n, "rejected": 0, "times": np.array([t, dt]), "flux": flux,
                "minima": np.array(low)}
    if case["kind"] == "operators":
        rhs, bflux = plain.rhs(q)
        new, flux, low, _ = plain.step(q, 0.02 / (case["nx"] * 25))
        a = plain.averages(q)
        return {"rhs": rhs, "bflux": bflux, "limited": plain.limit(q)[0], "dt": plain.time_step(q), "averages": a,
                "integral": 2.0 * (plain.jac[:, None] * a).sum(0), "new": new, "flux": flux,
                "minima": np.array(low), "troubled": None}
    # the derivative of the positivity limiter's bisection is taken at its root: no value of a plain evaluation
    return {"final": plain.march(q, steps=case["steps"])[0], "grad": None, "bc_grad": None}
