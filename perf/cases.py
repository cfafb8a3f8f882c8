"""The work that is timed: what programs that use this framework have it do, one pass at a time.

A case names a kind of call, a tissue and its size. ``listed()`` gives the fixed cases, ``draw``
more of the same ranges; ``prepare`` builds the tissue (its mesh from the size, its material and
growth fields from the seed) and the solver handle a program keeps, ``run`` is one pass through
the public entry points and returns everything the pass computes.

Kinds
  steps      a short simulation from the rest state: the growth state is set back and the time loop
             runs ``steps`` implicit steps (what ``newton.simulate`` does, with the handle kept: one
             evaluation of a growth map)
  batch      the same for many uneven tissues in one context
  adjoint    one evaluation of a loss gradient: forward run with checkpoints, then the backward pass
  iteration  one Newton iteration at the method seam, for a host that keeps the Newton loop itself
  solve      the linear solve alone, refined once as the reference's direct solver is
  assemble   the residual and the Jacobian of one Newton iteration
"""
import functools
import math

import numpy as np
import torch

from tissueorigami_b200 import mesh
from tissueorigami_b200.newton import BatchSolver, NewtonRaphsonSolver

FLOPS_PER_ASSEMBLY = 15.2e3  # FP64 operations of one prism's forces and closed-form tangent
NEWTON_ITERS = 4             # Newton iterations a step of these tissues takes


def listed():
    return [
        # the smallest configuration: 342 prisms for ten steps, bound by latency and launches
        {"name": "rectangle_342", "kind": "steps", "tissue": "rectangle", "nx": 20, "ny": 10, "steps": 10},
        # a small clamped disc of odd size with smooth random growth: one tissue of a parameter study
        {"name": "disc_2713", "kind": "steps", "tissue": "disc", "prisms": 2713, "steps": 4},
        # the wing-disc configuration at its full size: two layers, ECM under columnar cells
        {"name": "wing_disc_80k", "kind": "steps", "tissue": "wing_disc", "points": 20000, "steps": 3},
        # a smaller wing disc with packing detection in every step, as the reference always runs
        {"name": "wing_disc_packing", "kind": "steps", "tissue": "wing_disc", "points": 6007, "steps": 3, "packing": True},
        # a tissue with internal viscosity: an unsymmetric Jacobian
        {"name": "wing_disc_viscous", "kind": "steps", "tissue": "wing_disc", "points": 1511, "steps": 2, "eta": 4.0},
        # a mid-size slab of three layers, odd in both directions
        {"name": "slab_151x97", "kind": "steps", "tissue": "slab", "nx": 151, "ny": 97, "steps": 2},
        # the large-slab configuration at its full size (3 M prisms, a 2.7 GB Jacobian), with packing detection
        {"name": "slab_1000x500", "kind": "steps", "tissue": "slab", "nx": 1000, "ny": 500, "steps": 2, "packing": True},
        # a parameter sweep over uneven tissues in one context
        {"name": "batch_48", "kind": "batch", "tissues": 48, "smallest": 500, "largest": 20000, "steps": 2},
        # one gradient of a growth-map fit
        {"name": "adjoint_wing_disc", "kind": "adjoint", "tissue": "wing_disc", "points": 5003, "steps": 6, "checkpoint": 3},
        # a host application that keeps the reference's Newton loop and calls one iteration at a time
        {"name": "iteration_disc_4801", "kind": "iteration", "tissue": "disc", "prisms": 4801},
        # the linear solve of a host that assembles elsewhere
        {"name": "solve_disc_1500", "kind": "solve", "tissue": "disc", "prisms": 1500},
        # the residual and Jacobian of a host that solves elsewhere
        {"name": "assemble_wing_disc", "kind": "assemble", "tissue": "wing_disc", "points": 4003},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_tissue(rng, largest_disc, largest_points, largest_slab):
    tissue = rng.choice(["rectangle", "disc", "disc", "wing_disc", "wing_disc", "slab"])
    if tissue == "rectangle":
        ny = rng.randint(6, 24)
        return {"tissue": tissue, "nx": ny + rng.randint(1, 24), "ny": ny}
    if tissue == "disc":
        return {"tissue": tissue, "prisms": _log_int(rng, 500, largest_disc)}
    if tissue == "wing_disc":
        return {"tissue": tissue, "points": _log_int(rng, 300, largest_points)}
    ny = _log_int(rng, 16, largest_slab)
    return {"tissue": tissue, "nx": int(ny * rng.uniform(1.0, 2.0)), "ny": ny}


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps", "batch", "adjoint", "iteration", "solve", "assemble"])
    if kind == "steps":
        case = {"kind": kind, **_draw_tissue(rng, 20000, 20000, 240), "steps": rng.randint(2, 4)}
        if case["tissue"] == "wing_disc" and case["points"] < 2000 and rng.random() < 0.3:
            case["eta"] = rng.choice([1.0, 2.0, 4.0])
        elif case["tissue"] != "rectangle" and rng.random() < 0.3:
            case["packing"] = True
        return case
    if kind == "batch":
        return {"kind": kind, "tissues": rng.randint(4, 48), "smallest": rng.randint(300, 600),
                "largest": rng.randint(3000, 20000), "steps": 2}
    if kind == "adjoint":
        case = {"kind": kind, "tissue": "wing_disc", "points": _log_int(rng, 500, 5000)}
        if rng.random() < 0.5:
            case = {"kind": kind, "tissue": "disc", "prisms": _log_int(rng, 500, 15000)}
        steps = rng.randint(3, 6)
        return {**case, "steps": steps, "checkpoint": rng.randint(2, steps)}
    tissue = _draw_tissue(rng, 4801 if kind != "assemble" else 15000, 1500 if kind != "assemble" else 4000, 48)
    while tissue["tissue"] == "rectangle":
        tissue = _draw_tissue(rng, 4801 if kind != "assemble" else 15000, 1500 if kind != "assemble" else 4000, 48)
    return {"kind": kind, **tissue}


# ---- tissues ---------------------------------------------------------------------------------

@functools.lru_cache(maxsize=8)
def _geometry(tissue, prisms, points, nx, ny):
    """The tissue of a size: its mesh and default fields (the seed's fields replace them)."""
    if tissue == "rectangle":
        return mesh.small_rectangle(nx=nx, ny=ny, newton_tol=1e-9)
    if tissue == "disc":
        return mesh.small_disc(11, prisms, 1000.0)
    if tissue == "wing_disc":
        return mesh.wing_disc(n_surface_points=points)
    return mesh.large_slab(nx=nx, ny=ny)


def _base(case):
    return _geometry(case["tissue"], case.get("prisms", 0), case.get("points", 0), case.get("nx", 0), case.get("ny", 0))


def _smooth(rng, xy, length):
    """A smooth random field of unit variance (random Fourier features)."""
    w = rng.normal(0.0, 1.0 / length, size=(24, 2))
    return np.cos(xy @ w.T + rng.uniform(0, 2 * math.pi, size=24)) @ rng.normal(size=24) * math.sqrt(2.0 / 24)


def _tissue(case, seed):
    """The case's tissue with the seed's stiffness and growth map."""
    t = _base(case).copy()
    rng = np.random.default_rng(seed)
    cen = t.xref.reshape(-1, 6, 3)[:, :, :2].mean(axis=1)
    if case["tissue"] == "rectangle":  # held by drag alone: uniform growth, uniform stiffness
        scale = rng.uniform(0.7, 1.3)
        t.lam, t.mu = t.lam * scale, t.mu * scale
        t.rates = t.rates * rng.uniform(0.7, 1.3)
    elif case["tissue"] == "slab":  # log-normal stiffness, anisotropic growth along a smooth direction field
        scale = np.exp(rng.normal(0.0, 0.3, t.n_elems))
        t.lam, t.mu = t.lam.mean() * scale, t.mu.mean() * scale
        t.angles = math.pi * _smooth(rng, cen, 20.0)
    else:  # stiffness differs from element to element, growth follows a smooth field
        scale = rng.uniform(0.9, 1.1, t.n_elems)
        t.lam, t.mu = t.lam * scale, t.mu * scale
        t.rates = t.rates * (1.0 + 0.2 * np.tanh(_smooth(rng, cen, 20.0)))[:, None]
    t.eta = np.full(t.n_elems, float(case.get("eta", 0.0)))
    return t


def _grown(t, rng):
    """Inverse growth tensors and a displaced iterate: the state inside a Newton loop."""
    fg = np.tile(np.eye(3), (t.n_elems, 1, 1))
    fg[:, 0, 0] = np.exp(t.rates[:, 0] * t.dt)
    fg[:, 1, 1] = np.exp(t.rates[:, 1] * t.dt)
    # the wiggle scales with the shortest element edge so that no element inverts
    x6 = t.xref.reshape(-1, 6, 3)
    edge = min(np.linalg.norm(x6[:, 1] - x6[:, 0], axis=1).min(), np.linalg.norm(x6[:, 3] - x6[:, 0], axis=1).min())
    uk = t.x + rng.uniform(-0.02, 0.02, t.x.shape) * edge * (t.fixed == 0)
    return np.linalg.inv(fg), uk


def _areas(t, x):
    """Exposed area of each node (Simulation::updateNodeViscositySurfaces)."""
    vs = np.zeros(t.n_nodes)
    for bit, i0 in ((1, 3), (2, 0)):
        tri = t.conn[(t.exposed & bit) != 0][:, i0:i0 + 3]
        n = np.cross(x[tri[:, 1]] - x[tri[:, 0]], x[tri[:, 2]] - x[tri[:, 0]])
        np.add.at(vs, tri, (np.linalg.norm(n, axis=1) / 6.0)[:, None])
    return vs


@functools.lru_cache(maxsize=2)
def _batch_geometry(tissues, smallest, largest):
    return mesh.batch_tissues(seed=1003 + tissues + largest, n_tissues=tissues, min_prisms=smallest, max_prisms=largest)


def _batch_tissues(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for t in _batch_geometry(case["tissues"], case["smallest"], case["largest"]):
        t = t.copy()
        scale = rng.uniform(0.5, 2.0)
        t.lam, t.mu = t.lam * scale, t.mu * scale
        t.rates = t.rates * rng.uniform(0.6, 1.2)
        out.append(t)
    return out


# ---- a pass ------------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ts = _batch_tissues(case, seed)
        solver = BatchSolver(ts)
        return {"case": case, "solver": solver, "x0": solver.join([t.x for t in ts]), "dt": ts[0].dt,
                "fg": np.concatenate([t.fg for t in ts])}
    t = _tissue(case, seed)
    if kind == "steps":
        solver = NewtonRaphsonSolver.from_tissue(t, packing=bool(case.get("packing", False)))
        return {"case": case, "solver": solver, "x0": t.x, "dt": t.dt, "fg": t.fg}
    if kind == "adjoint":
        solver = NewtonRaphsonSolver.from_tissue(t, krylov_rtol=1e-14)
        rng = np.random.default_rng(seed + 1)
        target = t.x * (1.0 + 0.01 * rng.uniform(size=3))
        return {"case": case, "solver": solver, "x0": t.x, "dt": t.dt, "fg": t.fg, "target": target}
    inv_fg, uk = _grown(t, np.random.default_rng(seed + 1))
    overrides = {"krylov_rtol": 1e-13, "krylov_refine": 1} if kind == "solve" else {"krylov_rtol": 1e-14}
    solver = NewtonRaphsonSolver.from_tissue(t, **overrides)
    solver.set_inv_fg(inv_fg)
    solver.set_viscosity_surface(_areas(t, t.x))
    state = {"case": case, "solver": solver, "uk": uk, "un": t.x, "dt": t.dt}
    if kind == "solve":
        state["g"], state["vals"], _, _, _ = solver.assemble(uk, t.x, t.dt)
    return state


def run(state):
    case, s = state["case"], state["solver"]
    kind = case["kind"]
    if kind in ("steps", "batch"):
        s.set_growth(fg=state["fg"])
        x = state["x0"]
        for _ in range(case["steps"]):
            x, _, _ = s.runOneStep(x, state["dt"])
        return {"x": x}
    if kind == "adjoint":
        s.set_growth(fg=state["fg"])
        x, _, _ = s.adjoint_forward(state["x0"], case["steps"], state["dt"], case["checkpoint"])
        rates, x0, _, _ = s.adjoint_backward(2.0 * (x - state["target"]), want_dx0=True)
        return {"x": x, "d_rates": rates, "d_x0": x0}
    if kind == "iteration":
        return {"du": s.newton_iteration(state["uk"], state["un"], state["dt"])[0]}
    if kind == "solve":
        return {"du": s.solveForDeltaU(state["vals"], state["g"])[0]}
    g, vals, _, _, _ = s.assemble(state["uk"], state["un"], state["dt"])
    return {"g": g, "vals": vals}


def work(case):
    """Positions in and out and every element's data once per assembly's inputs; the operations of
    the assemblies a pass makes (the linear solves' cost depends on the method and is left out)."""
    if case["kind"] == "batch":
        ts = _batch_geometry(case["tissues"], case["smallest"], case["largest"])
        nodes, elems = sum(t.n_nodes for t in ts), sum(t.n_elems for t in ts)
    else:
        t = _base(case)
        nodes, elems = t.n_nodes, t.n_elems
    steps = case.get("steps", 1)
    element_bytes = 24 + 144 + 72 + 24 + 32  # nodes, reference shape, growth tensor, material, rates and angle
    if case["kind"] == "assemble":
        blocks = nodes + 2 * _edges(case)
        return {"bytes": 72.0 * nodes + element_bytes * elems + 72.0 * blocks, "flops": FLOPS_PER_ASSEMBLY * elems}
    if case["kind"] == "solve":
        blocks = nodes + 2 * _edges(case)
        return {"bytes": 48.0 * nodes + 72.0 * blocks, "flops": 18.0 * blocks}
    if case["kind"] == "iteration":
        return {"bytes": 72.0 * nodes + element_bytes * elems, "flops": FLOPS_PER_ASSEMBLY * elems}
    assemblies = NEWTON_ITERS * steps
    if case["kind"] == "adjoint":  # forward, the recomputed segments and one assembly per backward step
        assemblies = (2 * NEWTON_ITERS + 1) * steps
    return {"bytes": steps * (48.0 * nodes + (element_bytes + 72.0) * elems), "flops": FLOPS_PER_ASSEMBLY * assemblies * elems}


@functools.lru_cache(maxsize=8)
def _edge_count(tissue, prisms, points, nx, ny):
    conn = _geometry(tissue, prisms, points, nx, ny).conn.astype(np.int64)
    a, b = np.triu_indices(6, 1)
    lo, hi = np.minimum(conn[:, a], conn[:, b]), np.maximum(conn[:, a], conn[:, b])
    return int(np.unique(lo * (conn.max() + 1) + hi).size)


def _edges(case):
    return _edge_count(case["tissue"], case.get("prisms", 0), case.get("points", 0), case.get("nx", 0), case.get("ny", 0))


# ---- the same results in plain torch, 64 bits ---------------------------------------------------

EXACT_DOFS = 12000    # dense solves up to this many unknowns
EXACT_ELEMS = 20000   # assemblies up to this many prisms


def _shape_gradients():
    """dN[g][k][n]: derivatives of the six shape functions at the six Gauss points (Prism.cpp:97-130)."""
    s = 1.0 / math.sqrt(3.0)
    out = np.zeros((6, 3, 6))
    for g in range(6):
        eta, nu = [(1 / 6, 1 / 6), (2 / 3, 1 / 6), (1 / 6, 2 / 3)][g % 3]
        zeta = s if g < 3 else -s
        a, b, l = (1 - zeta) / 2, (1 + zeta) / 2, 1 - eta - nu
        out[g] = [[-a, a, 0, -b, b, 0], [-a, 0, a, -b, 0, b], [-l / 2, -eta / 2, -nu / 2, l / 2, eta / 2, nu / 2]]
    return out


def _det3(m):
    return torch.dot(m[0], torch.linalg.cross(m[1], m[2]))


class _Plain:
    """The tissue in plain torch: the elastic energy of the prisms, differentiated by autograd."""

    def __init__(self, t):
        self.t = t
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.conn = torch.as_tensor(t.conn.astype(np.int64), device=self.dev)
        self.dN = self.up(_shape_gradients())
        self.xref = self.up(t.xref).reshape(-1, 6, 3)
        self.lam, self.mu = self.up(t.lam), self.up(t.mu)
        self.fixed = torch.as_tensor(t.fixed.reshape(-1) != 0, device=self.dev)
        self.ext_visc = self.up(t.ext_visc).reshape(-1)

    def up(self, a):
        return torch.as_tensor(np.array(a, dtype=np.float64), device=self.dev)

    def element_energy(self, x, xref, inv_fg, lam, mu):
        """Neo-Hookean energy of one prism at nodes x [6,3], per volume of the grown shape."""
        e = 0.0
        for g in range(6):
            dX = (self.dN[g] @ xref).T
            F = (self.dN[g] @ x).T @ torch.linalg.inv(dX)
            Fe = F @ inv_fg
            ln = torch.log(_det3(Fe))
            w = mu / 2 * ((Fe * Fe).sum() - 3) - mu * ln + lam / 2 * ln * ln
            e = e + w * _det3(dX) / _det3(inv_fg) / 6
        return e

    def elements(self, x, inv_fg):
        """Forces [E,18] and tangents [E,18,18] of every prism."""
        f = torch.func.grad(self.element_energy)
        h = torch.func.hessian(self.element_energy)
        args = (x.reshape(-1, 3)[self.conn], self.xref, inv_fg, self.lam, self.mu)
        both = torch.func.vmap(lambda *a: (f(*a), h(*a)), chunk_size=2048)(*args)
        return -both[0].reshape(-1, 18), both[1].reshape(-1, 18, 18)

    def system(self, uk, un, dt, inv_fg, vs):
        """Residual [3N], element tangents with fixed rows and columns dropped, diagonal terms."""
        dofs = (3 * self.conn[:, :, None] + torch.arange(3, device=self.dev)).reshape(-1, 18)
        f, K = self.elements(uk, inv_fg)
        drag = self.up(vs).repeat_interleave(3) * self.ext_visc / dt
        g = torch.zeros(uk.numel(), dtype=torch.float64, device=self.dev).index_add_(0, dofs.reshape(-1), f.reshape(-1))
        g = torch.where(self.fixed, 0.0, g - drag * (uk - un))
        free = (~self.fixed)[dofs].double()
        return g, K * free[:, :, None] * free[:, None, :], torch.where(self.fixed, 1.0, drag), dofs

    def solve(self, K, diag, dofs, g):
        n = g.numel()
        J = torch.zeros(n * n, dtype=torch.float64, device=self.dev)
        J.index_add_(0, (dofs[:, :, None] * n + dofs[:, None, :]).reshape(-1), K.reshape(-1))
        J = J.reshape(n, n)
        J.diagonal().add_(diag)
        x = torch.linalg.solve(J, g)
        return x + torch.linalg.solve(J, g - J @ x)

    def blocks(self, K, diag):
        """The Jacobian's 3x3 blocks, rows in order, columns ascending."""
        n = self.t.n_nodes
        key = (self.conn[:, :, None] * n + self.conn[:, None, :]).reshape(-1)
        key = torch.cat([key, torch.arange(n, device=self.dev) * (n + 1)])
        where, at = torch.unique(key, return_inverse=True)
        v = torch.zeros((where.numel(), 3, 3), dtype=torch.float64, device=self.dev)
        v.index_add_(0, at, torch.cat([K.reshape(-1, 6, 3, 6, 3).permute(0, 1, 3, 2, 4).reshape(-1, 3, 3),
                                       torch.diag_embed(diag.reshape(-1, 3))]))
        return v

    def grow(self, x, fg, dt):
        """The growth tensors after a step's growth (ShapeBase.cpp:1914-2041, 471-505, 1452-1506)."""
        t = self.t
        xe = x.cpu().numpy().reshape(-1, 3)[t.conn]
        F = 0.0
        for dN in _shape_gradients():
            F = F + (dN @ xe).transpose(0, 2, 1) @ np.linalg.inv((dN @ t.xref.reshape(-1, 6, 3)).transpose(0, 2, 1)) / 6
        U, _, Vt = np.linalg.svd(F)
        R = U @ Vt
        off = np.abs(R - R * np.eye(3)).max(axis=(1, 2)) > 0.017
        tz = np.arctan2(R[:, 0, 1], R[:, 0, 0])
        tz = np.where(off & (np.abs(tz) > 0.017), tz, 0.0)

        def rot(a):
            m = np.tile(np.eye(3), (a.size, 1, 1))
            m[:, 0, 0] = m[:, 1, 1] = np.cos(a)
            m[:, 1, 0] = np.sin(a)
            m[:, 0, 1] = -m[:, 1, 0]
            return m

        A, G = rot(t.angles), rot(-tz)
        inc = A @ (np.exp(t.rates * dt)[:, :, None] * A.transpose(0, 2, 1))
        return G.transpose(0, 2, 1) @ inc @ G @ fg

    def step(self, x, fg, dt, tol):
        fg = self.grow(x, fg, dt)
        inv_fg, vs = self.up(np.linalg.inv(fg)), _areas(self.t, x.cpu().numpy().reshape(-1, 3))
        uk = x.clone()
        for _ in range(20):
            g, K, diag, dofs = self.system(uk, x, dt, inv_fg, vs)
            du = self.solve(K, diag, dofs, g)
            uk = uk + du
            if float(du.norm()) <= tol:
                break
        return uk, fg


def _exact_steps(t, case):
    p = _Plain(t)
    x, fg = p.up(t.x).reshape(-1), t.fg.reshape(-1, 3, 3)
    for _ in range(case["steps"]):
        x, fg = p.step(x, fg, t.dt, t.newton_tol)
    return x.reshape(-1, 3).cpu()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("adjoint", "batch") or case.get("eta") or case.get("packing"):
        return None
    t = _tissue(case, seed)
    if kind == "steps":
        return {"x": _exact_steps(t, case)} if 3 * t.n_nodes <= EXACT_DOFS else None
    if t.n_elems > EXACT_ELEMS or (kind != "assemble" and 3 * t.n_nodes > 2 * EXACT_DOFS):
        return None
    inv_fg, uk = _grown(t, np.random.default_rng(seed + 1))
    p = _Plain(t)
    g, K, diag, dofs = p.system(p.up(uk).reshape(-1), p.up(t.x).reshape(-1), t.dt, p.up(inv_fg), _areas(t, t.x))
    if kind == "assemble":
        return {"g": g.cpu(), "vals": p.blocks(K, diag).cpu()}
    return {"du": p.solve(K, diag, dofs, g).cpu()}
