"""The work that a program using this solver has it do, as cases that can be timed and compared.

A case is a dict of plain values with a "kind":

  frame   one garment, the viewer's loop: `steps` plain PD steps, then its state
  resolve one garment on the runner's non-IPC branch: step, then the colliders' projections
  ipc     one garment with contact: a given state, `steps` step_with_ipc, then its positions
  batch   many garments in one batch: one plain step, then every position
  drapes  many garments in contact in one batch: new poses in, one contact step, every position out
  pairs   the broad phase over one mesh, as a call of its own (both entry points)
  solve   the sparse solver on its own: the three right-hand sides of a step with a kept factor
  refactor  the same after the matrix's numbers changed (another material or dt)

Meshes, materials and step configurations are those of the repository's scenarios and benchmark; the state each
garment starts from (small displacements and velocities), materials and numbers come from the seed.
"""
from __future__ import annotations

import concurrent.futures as cf
import math
import os

import numpy as np
import torch

from vistio_b200 import api, scenarios

DT = 1.0 / 60.0
D_HAT, KAPPA = 1e-3, 1e4  # drapes: m, read as a distance (barrier_d_hat is its square)
RIBBON_DT, RIBBON_D_HAT, RIBBON_KAPPA = 1.0 / 120.0, 5e-4, 1e3
CELL = 5e-3  # the ribbon's cells


def listed():
    return [
        # The reference's own headline scenario: the smallest step, launch and latency bound.
        dict(name="sheet 20x20 frame", kind="frame", cols=20, rows=20, model=0, bending=1, iters=10, refine=0, steps=1),
        # An odd-sized garment of the best material tier (anisotropic membrane, anisotropic Discrete Shells) with
        # the FP64 refinement that the accuracy option adds.
        dict(name="sheet 97x97 tier 3", kind="frame", cols=97, rows=97, model=3, bending=3, iters=10, refine=1, steps=2),
        # A narrow strip over a sphere and the ground without IPC: step + collider projections.
        dict(name="strip 10x40 resolve", kind="resolve", cols=10, rows=40, model=1, bending=2, iters=10, refine=0, steps=2),
        # The sphere drape scenario at its real size with the IPC barriers of the colliders (no self contact).
        dict(name="drape 64x64 colliders", kind="ipc", cols=64, rows=64, model=0, bending=1, iters=15, al=5, steps=2, self=False),
        # The self fold scenario at its real size: a folded ribbon whose layers touch (self contact, ground).
        dict(name="ribbon 40x400 self", kind="ipc", cols=40, rows=400, model=2, bending=1, iters=10, al=5, steps=2, self=True),
        # The benchmark's flagship: 512 sheets of 8 topologies, tuned once like the benchmark does.
        dict(name="512 sheets", kind="batch", count=512, topologies=8, lo=16, hi=128, model=0, bending=1, iters=10, refine=0, tune=True),
        # A served mix: few garments, every mesh its own size, materials of several kinds, not tuned.
        dict(name="24 ragged sheets", kind="batch", count=24, topologies=24, lo=17, hi=151, model=2, bending=2, iters=10, refine=0, tune=False),
        # The benchmark's contact workload: drapes of 8 topologies with collider and self contact, tuned.
        dict(name="64 drapes self", kind="drapes", count=64, topologies=8, lo=16, hi=128, iters=15, al=5),
        # A collision query of its own over the folded ribbon (32,000 triangles).
        dict(name="pairs 40x400", kind="pairs", cols=40, rows=400, layers=8, noalloc=False),
        # The per-frame query that may not allocate, on a smaller odd mesh.
        dict(name="pairs 61x183 noalloc", kind="pairs", cols=61, rows=183, layers=5, noalloc=True),
        # The sparse solver as a part: x, y and z of one global solve.
        dict(name="solve 75x75", kind="solve", cols=75, rows=75),
        # ... and a change of material or dt: new numbers in the same pattern, then the solve.
        dict(name="refactor 64x64", kind="refactor", cols=64, rows=64),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "resolve", "ipc", "ipc", "batch", "batch", "drapes", "pairs", "solve", "refactor"])
    if kind == "frame":
        return dict(kind=kind, cols=_log(rng, 7, 190), rows=_log(rng, 7, 190), model=rng.randrange(5), bending=rng.randrange(1, 4),
                    iters=rng.choice([5, 10, 15]), refine=rng.choice([0, 0, 1, 2]), steps=rng.randrange(1, 4))
    if kind == "resolve":
        return dict(kind=kind, cols=_log(rng, 5, 60), rows=_log(rng, 20, 160), model=rng.randrange(2), bending=rng.randrange(1, 4),
                    iters=10, refine=0, steps=rng.randrange(1, 4))
    if kind == "ipc":
        self_ = rng.random() < 0.5
        c = _log(rng, 12, 110)
        return dict(kind=kind, cols=_log(rng, 10, 48) if self_ else c, rows=_log(rng, 60, 420) if self_ else c,
                    model=rng.choice([0, 1, 2]), bending=1, iters=rng.choice([10, 15]), al=rng.choice([3, 5]), steps=2, self=self_)
    if kind == "batch":
        n = _log(rng, 2, 300)
        return dict(kind=kind, count=n, topologies=min(n, rng.choice([1, 3, 8, 24])), lo=rng.randrange(8, 40), hi=rng.randrange(60, 140),
                    model=rng.randrange(4), bending=rng.randrange(1, 3), iters=10, refine=0, tune=n > 64)
    if kind == "drapes":
        n = _log(rng, 3, 56)
        return dict(kind=kind, count=n, topologies=min(n, rng.choice([1, 3, 8])), lo=rng.randrange(10, 40), hi=rng.randrange(50, 128),
                    iters=rng.choice([10, 15]), al=rng.choice([3, 5]))
    if kind == "pairs":
        cols, rows = _log(rng, 8, 100), _log(rng, 40, 320)
        return dict(kind=kind, cols=cols, rows=rows, layers=rng.randrange(1, 10), noalloc=cols * rows < 12000 and rng.random() < 0.7)
    return dict(kind=kind, cols=_log(rng, 9, 110), rows=_log(rng, 9, 110))


# ---------------------------------------------------------------- inputs
def _sheet(case):
    """A hanging sheet (first row pinned) in the XZ plane, of the quad grid's triangulation."""
    cols, rows = case["cols"], case["rows"]
    px, py, pz, tris = scenarios.quad_grid(cols, rows, cols / max(cols, rows), rows / max(cols, rows))
    pinned = np.zeros(px.shape[0], np.uint8)
    pinned[: cols + 1] = 1
    return scenarios.Mesh(px, np.ones_like(px), py.copy(), tris, pinned)


def _drape(side):
    """A drape 1 mm above a sphere of radius 0.3 m at the origin: the barriers act from the first step."""
    return scenarios.sphere_drape(side=side, length=1.5, height=0.301)


def _folded(cols, rows, layers, cell, gap, turn, height):
    """A grid of square cells folded in `layers` layers `gap` apart, the lowest at `height`; towards a fold its two
    layers part to `turn`, and the row on the fold lies halfway between them, so that the edges keep their lengths."""
    per = max(1, rows // layers)
    j = np.repeat(np.arange(rows + 1), cols + 1)
    layer, at = j // per, j % per
    along = np.where(layer % 2 == 0, at, per - at)
    y = np.full(j.shape, height)
    for q in range(layer.max()):
        away = (per - along if q % 2 == 0 else along) / per  # from the fold that joins layers q and q + 1
        part = gap + (turn - gap) * np.maximum(0.0, 1.0 - 5.0 * away)
        y += part * ((layer > q) - 0.5 * ((layer == q + 1) & (at == 0)))
    x = np.tile(np.arange(cols + 1), rows + 1)
    return np.stack([x * cell, y, along * cell], 1).astype(np.float32)


def _dt(case):
    return RIBBON_DT if case.get("self", False) else DT


def _materials(case, seed, count):
    rng = np.random.default_rng(seed)
    setups = []
    for _ in range(count):
        setups.append(api.SetupDesc(
            model=case.get("model", 0), bending=case.get("bending", 1),
            stiffness=float(math.exp(rng.uniform(math.log(2e2), math.log(5e3)))),
            bend_stiffness=float(math.exp(rng.uniform(math.log(1e-5), math.log(1e-3)))),
            density_gsm=float(rng.uniform(80.0, 300.0)), warp_stiffness=float(rng.uniform(0.5, 1.0)),
            weft_stiffness=float(rng.uniform(0.2, 0.9)), bend_warp=float(rng.uniform(0.5, 1.0)),
            bend_weft=float(rng.uniform(0.1, 0.5)), matrix_dt=_dt(case)))
    return setups


def _sides(case, seed):
    """The grid sides of a batch: one per topology, spread over [lo, hi] whatever the seed, given out in turn."""
    t = case["topologies"]
    side = [int(round(case["lo"] + (case["hi"] - case["lo"]) * (k + 0.5) / t)) for k in range(t)]
    return [side[k % t] for k in range(case["count"])]


def _config(case):
    if case["kind"] in ("ipc", "drapes"):
        d_hat, kappa = (RIBBON_D_HAT, RIBBON_KAPPA) if case.get("self", False) else (D_HAT, KAPPA)
        return api.drape_config(max_iterations=case["iters"], al_max_iterations=case["al"], barrier_d_hat=d_hat * d_hat,
                                barrier_kappa=kappa)
    return api.drape_config(max_iterations=case["iters"], refinement_sweeps=case["refine"])


def _contact(case):
    if case["kind"] == "resolve":
        return api.Contact(has_ground=True, ground_height=0.75, has_sphere=True, sphere_center=(0.0, 0.7, 0.0), sphere_radius=0.32)
    if case.get("self", False):
        return api.Contact(has_ground=True, ground_height=0.0, self_collision=True, kappa=RIBBON_KAPPA, thickness=RIBBON_D_HAT)
    self_ = case["kind"] == "drapes"
    return api.Contact(has_ground=True, ground_height=-0.3, has_sphere=True, sphere_center=(0.0, 0.0, 0.0), sphere_radius=0.3,
                       self_collision=self_, kappa=KAPPA, thickness=1.5 * D_HAT if self_ else 0.0)


def _garment(case, seed):
    """(mesh, pinned or None, positions, velocities) of a single garment's case."""
    rng = np.random.default_rng(seed + 7)
    cols, rows, pinned = case["cols"], case["rows"], None
    if case.get("self", False):
        # the ribbon folded in four, its layers and the ground coming into each other's reach
        mesh = scenarios.self_fold(cols, rows, CELL * cols, CELL * rows)
        pos, amp, speed = _folded(cols, rows, 4, CELL, 8e-4, 1.6e-3, 2.2e-3), 3e-5, 0.01
    else:
        mesh = _drape(cols) if case["kind"] == "ipc" else _sheet(case)
        pos, amp, speed = np.stack([mesh.px, mesh.py, mesh.pz], 1), 5e-5, 0.02
        if case["kind"] != "ipc":
            pinned, amp, speed = mesh.pinned, 0.1 / max(cols, rows), 0.1
    free = (np.ones(len(pos)) if pinned is None else pinned == 0)[:, None]
    pos = pos + amp * rng.uniform(-1, 1, pos.shape) * free
    vel = speed * rng.normal(size=pos.shape) * free
    if pinned is not None:  # in mid-swing about the pinned row
        vel[:, 1] += rng.uniform(2.0, 4.0) * (pos[:, 2] - pos[0, 2])
    return mesh, pinned, pos.astype(np.float32), vel.astype(np.float32)


def _matrix(case, seed):
    """A cloth-like SPD matrix in CSR (f32): mass on the diagonal and a random stiffness on every edge of the grid's
    8-neighbourhood."""
    c, r = case["cols"] + 1, case["rows"] + 1
    rng = np.random.default_rng(seed)
    idx = np.arange(c * r).reshape(r, c)
    ends = [(idx[:, :-1], idx[:, 1:]), (idx[:-1], idx[1:]), (idx[:-1, :-1], idx[1:, 1:]), (idx[:-1, 1:], idx[1:, :-1])]
    i = np.concatenate([a.ravel() for a, _ in ends])
    j = np.concatenate([b.ravel() for _, b in ends])
    w = np.exp(rng.uniform(math.log(1.0), math.log(30.0), i.size)).astype(np.float32)
    diag = rng.uniform(0.5, 2.0, c * r)
    np.add.at(diag, i, w)
    np.add.at(diag, j, w)
    rows = np.concatenate([i, j, idx.ravel()])
    cols = np.concatenate([j, i, idx.ravel()])
    vals = np.concatenate([-w, -w, diag.astype(np.float32)]).astype(np.float32)
    order = np.lexsort((cols, rows))
    rows, cols, vals = rows[order], cols[order], vals[order]
    ptr = np.zeros(c * r + 1, np.uint32)
    np.add.at(ptr, rows + 1, 1)
    rhs = rng.normal(size=(3, c * r)).astype(np.float32)
    return np.cumsum(ptr).astype(np.uint32), cols.astype(np.uint32), vals, rhs


def _solvers(meshes, cfg, setups):
    def make(k):
        m = meshes[k]
        return api.ProjectiveDynamicsSolver().init_explicit(m, cfg, setups[k], pinned=m.pinned)

    api.default_context()
    with cf.ThreadPoolExecutor(min(16, os.cpu_count() or 4)) as pool:
        return list(pool.map(make, range(len(meshes))))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("frame", "resolve", "ipc"):
        mesh, pinned, pos, vel = _garment(case, seed)
        s = api.ProjectiveDynamicsSolver().init_explicit(mesh, _config(case), _materials(case, seed, 1)[0], pinned=pinned)
        s.set_state(pos, vel)
        return dict(case=case, solver=s, contact=None if kind == "frame" else _contact(case), pos=pos, vel=vel)
    if kind in ("batch", "drapes"):
        sides = _sides(case, seed)
        rng = np.random.default_rng(seed + 7)
        if kind == "batch":
            meshes = [scenarios.hanging_sheet(s, float(rng.uniform(0.5, 2.0))) for s in sides]
        else:
            kept = {s: _drape(s) for s in set(sides)}
            meshes = [kept[s] for s in sides]
        batch = api.Batch(_solvers(meshes, _config(case), _materials(case, seed, len(meshes))))
        if kind == "drapes" or case["tune"]:
            batch.tune()
        start = np.concatenate([np.stack([m.px, m.py, m.pz], 1) for m in meshes])
        free = np.concatenate([m.pinned == 0 for m in meshes])
        amp = 5e-5 if kind == "drapes" else 1e-3
        start = start + amp * rng.uniform(-1, 1, start.shape).astype(np.float32) * free[:, None]
        start = torch.from_numpy(start.astype(np.float32)).pin_memory()
        out = torch.empty_like(start).pin_memory()
        batch.upload_positions(start.numpy())
        return dict(case=case, batch=batch, contact=_contact(case) if kind == "drapes" else None, start=start, out=out)
    if kind == "pairs":
        tris = scenarios.quad_grid(case["cols"], case["rows"], 1.0, 1.0)[3]
        pos = _folded(case["cols"], case["rows"], case["layers"], CELL, 2e-3, 2e-3, 0.0)
        pos = pos + 2e-4 * np.random.default_rng(seed).uniform(-1, 1, pos.shape)
        return dict(case=case, pos=pos.astype(np.float32), tris=tris, out=np.zeros((40 * len(tris), 2), np.uint32))
    ptr, col, val, rhs = _matrix(case, seed)
    s = api.SparseSolver()
    s.factorize(ptr, col, val, len(ptr) - 1)
    return dict(case=case, solver=s, ptr=ptr, col=col, val=val, rhs=rhs)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "frame":
        for _ in range(case["steps"]):
            state["solver"].step(DT)
        return state["solver"].state()
    if kind == "resolve":
        for _ in range(case["steps"]):
            state["solver"].step(DT)
            state["solver"].resolve_contacts(state["contact"])
        return state["solver"].state()
    if kind == "ipc":
        state["solver"].set_state(state["pos"], state["vel"])
        for _ in range(case["steps"]):
            state["solver"].step_with_ipc(_dt(case), state["contact"])
        return state["solver"].state()[0]  # the last step moved on from the velocities of the one before
    if kind == "batch":
        state["batch"].step(DT)
        return state["batch"].download_positions(state["out"].numpy())
    if kind == "drapes":
        state["batch"].upload_positions(state["start"].numpy())
        state["batch"].step(DT, 1, state["contact"])
        return state["batch"].download_positions(state["out"].numpy())
    if kind == "pairs":
        query = api.broadphase_pairs_noalloc if case["noalloc"] else api.broadphase_pairs
        found = query(state["pos"], state["tris"], 1.5 * D_HAT)
        state["out"][: len(found)] = found  # the program's own list, as long as any pose needs
        state["out"][len(found) :] = 0
        return state["out"]
    solver = state["solver"]
    if kind == "refactor":
        solver = api.SparseSolver()
        solver.factorize(state["ptr"], state["col"], state["val"], len(state["ptr"]) - 1)
    return [solver.solve(b) for b in state["rhs"]]


# ------------------------------------------------------------------ work
def _grid(cols, rows):
    """(vertices, triangles, hinges, entries of the nested-dissection factor) of a quad grid."""
    v = (cols + 1) * (rows + 1)
    return v, 2 * cols * rows, 3 * cols * rows - cols - rows, v * max(6.0, 6.87 * math.log2(v) - 36.1)


def work(case):
    """Bytes: the garments' rest data and state in and out once per pass, and the factor's entries once per global
    solve (it is used whole by both sweeps of each). Flops: 2 per factor entry, sweep and axis, and the projections."""
    kind = case["kind"]
    if kind == "pairs":
        v, t, _, _ = _grid(case["cols"], case["rows"])
        return {"bytes": 12 * v + 12 * t + 8 * 12 * t, "flops": 0}
    if kind in ("solve", "refactor"):
        v, _, _, nnz = _grid(case["cols"], case["rows"])
        full = 16.0 * v ** 1.5  # the top separators of a grid's factorization
        return {"bytes": 3 * (8 * v + 4 * nnz) + (72 * v if kind == "refactor" else 0), "flops": 3 * 4 * nnz + (full if kind == "refactor" else 0)}
    if kind in ("batch", "drapes"):
        grids = [_grid(s, s) for s in _sides(case, 0)]
    else:
        grids = [_grid(case["cols"], case["rows"])]
    v, t, h, nnz = (sum(g[k] for g in grids) for k in range(4))
    solves = case["iters"] * case.get("steps", 1) * (1 if kind in ("ipc", "drapes") else 1 + case.get("refine", 0))
    return {"bytes": 36 * t + 40 * h + 96 * v + solves * (4 * nnz + 24 * v), "flops": solves * (12 * nnz + 300 * t + 150 * h)}


# ----------------------------------------------------- the same in 64 bits
DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.asarray(a), device=DEV).double()


def _f(v):
    """A parameter as the f32 that the solver's interface takes, in 64 bits."""
    return float(np.float32(v))


def _dot(a, b):
    return (a * b).sum(-1, keepdim=True)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


class _Cloth64:
    """Projective Dynamics on quad grids of one size (a leading axis over garments) in 64 bits: every global solve
    is a block tridiagonal Cholesky over pairs of grid rows, which hold all the stencils' couplings."""

    def __init__(self, rests, tris, pinned, setups, cols):
        self.x0 = _t(rests)  # (G, V, 3)
        g, v, _ = self.x0.shape
        self.g, self.v = g, v
        self.pinned = torch.as_tensor(pinned != 0, device=DEV)[None, :, None]
        self.setups = setups
        par = lambda name: _t([_f(getattr(s, name)) for s in setups])[:, None]  # noqa: E731
        self.tris = torch.as_tensor(tris.astype(np.int64), device=DEV)
        p = [self.x0[:, self.tris[:, k]] for k in range(3)]
        e1, e2 = p[1] - p[0], p[2] - p[0]
        n = torch.linalg.cross(e1, e2)
        area = 0.5 * n.norm(dim=-1)
        u = _unit(e1)
        w = _unit(torch.linalg.cross(n, u))
        dm = torch.stack([torch.cat([_dot(e1, u), _dot(e2, u)], -1), torch.cat([_dot(e1, w), _dot(e2, w)], -1)], -2)
        self.dm = torch.linalg.inv(dm)  # (G, T, 2, 2)
        self.tw = par("stiffness") * area
        grad = torch.cat([-self.dm.sum(-2, keepdim=True), self.dm], -2)  # (G, T, 3, 2): row k is corner k's gradient
        self.grad = grad
        mass = torch.zeros(g, v, device=DEV, dtype=torch.float64)
        for k in range(3):
            mass.index_add_(1, self.tris[:, k], area * (par("density_gsm") / 1000.0) / 3.0)
        self.mass = torch.where(self.pinned[..., 0], torch.full_like(mass, 1e8), mass)
        self._hinges(tris, par)
        h = _t([_f(s.matrix_dt) for s in setups])[:, None]
        self.inv_h2 = 1.0 / (h * h)
        self._matrix(cols)

    def _hinges(self, tris, par):
        edges = {}
        for t, tri in enumerate(tris.tolist()):
            for k in range(3):
                a, b = tri[k], tri[(k + 1) % 3]
                edges.setdefault((min(a, b), max(a, b)), []).append(tri[(k + 2) % 3])
        hv = np.array([[a, b, *w] for (a, b), w in sorted(edges.items()) if len(w) == 2], np.int64)
        self.hv = torch.as_tensor(hv, device=DEV)
        p0, p1, pa, pb = (self.x0[:, self.hv[:, k]] for k in range(4))
        e = p1 - p0
        el = e.norm(dim=-1)
        self.rest = torch.full(el.shape, math.pi, device=DEV, dtype=torch.float64)  # the scenarios' meshes are flat
        self.hw = par("bend_stiffness") * el
        kind = self.setups[0].bending
        st = torch.tensor([-1.0, -1.0, 1.0, 1.0], device=DEV, dtype=torch.float64).expand(*el.shape, 4)
        if kind >= 2:
            ca = el / torch.linalg.cross(e, pa - p0).norm(dim=-1)
            cb = el / torch.linalg.cross(e, pb - p0).norm(dim=-1)
            share = lambda q: (_dot(q, e)[..., 0] / (el * el))  # noqa: E731
            st = torch.stack([-share(p1 - pa) * ca - share(p1 - pb) * cb, -share(pa - p0) * ca - share(pb - p0) * cb, ca, cb], -1)
            st = _unit(st)
        if kind == 3:
            kw, kf = par("bend_warp"), par("bend_weft")
            hz = e * torch.tensor([1.0, 0.0, 1.0], device=DEV, dtype=torch.float64)
            cos2 = _unit(hz)[..., 0] ** 2
            self.hw = self.hw * (kf * cos2 + kw * (1 - cos2)) / ((kw + kf) / 2)
        self.st = st

    def _matrix(self, cols):
        bs = 2 * (cols + 1)
        nb = -(-self.v // bs)
        self.bs, self.nb = bs, nb
        diag = torch.zeros(self.g, nb * bs * bs, device=DEV, dtype=torch.float64)
        low = torch.zeros(self.g, nb * bs * bs, device=DEV, dtype=torch.float64)

        def add(i, j, val):
            bi, bj = i // bs, j // bs
            at = bj * bs * bs + (i % bs) * bs + j % bs
            same = bi == bj
            diag.index_add_(1, at[same], val[:, same])
            below = bi == bj + 1  # the entry above it is its mirror image
            low.index_add_(1, at[below], val[:, below])

        every = torch.arange(nb * bs, device=DEV)
        add(every[: self.v], every[: self.v], self.mass * self.inv_h2)
        add(every[self.v :], every[self.v :], torch.ones(self.g, nb * bs - self.v, device=DEV, dtype=torch.float64))
        for a in range(3):
            for b in range(3):
                add(self.tris[:, a], self.tris[:, b], self.tw * (self.grad[:, :, a] * self.grad[:, :, b]).sum(-1))
        for a in range(4):
            for b in range(4):
                add(self.hv[:, a], self.hv[:, b], self.hw * self.st[..., a] * self.st[..., b])
        d, lo = diag.view(self.g, nb, bs, bs), low.view(self.g, nb, bs, bs)
        self.chol, self.off = [], []
        s = d[:, 0]
        for k in range(nb):
            self.chol.append(torch.linalg.cholesky(s))
            if k + 1 < nb:  # off = low inv(chol)^T
                o = torch.linalg.solve_triangular(self.chol[k], lo[:, k].transpose(-1, -2), upper=False).transpose(-1, -2)
                self.off.append(o)
                s = d[:, k + 1] - o @ o.transpose(-1, -2)

    def solve(self, r):
        y = torch.zeros(self.g, self.nb * self.bs, 3, device=DEV, dtype=torch.float64)
        y[:, : self.v] = r
        y = list(y.view(self.g, self.nb, self.bs, 3).unbind(1))
        for k in range(self.nb):
            if k:
                y[k] = y[k] - self.off[k - 1] @ y[k - 1]
            y[k] = torch.linalg.solve_triangular(self.chol[k], y[k], upper=False)
        for k in range(self.nb - 1, -1, -1):
            if k + 1 < self.nb:
                y[k] = y[k] - self.off[k].transpose(-1, -2) @ y[k + 1]
            y[k] = torch.linalg.solve_triangular(self.chol[k].transpose(-1, -2), y[k], upper=True)
        return torch.cat(y, 1)[:, : self.v]

    def residual(self, x, pred, inv_dt2):
        """b - A x of one PD iteration: inertia, then what each element's target still asks for."""
        m = self.mass[..., None]
        r = (pred - x) * (m * self.inv_h2[..., None]) + pred * (m * (inv_dt2 - self.inv_h2[..., None]))
        p = [x[:, self.tris[:, k]] for k in range(3)]
        f = torch.stack([p[1] - p[0], p[2] - p[0]], -1) @ self.dm  # (G, T, 3, 2)
        d = (self._target(f) - f) * self.tw[..., None, None]
        for k in range(3):
            r.index_add_(1, self.tris[:, k], (d @ self.grad[:, :, k, :, None])[..., 0])
        p0, p1, pa, pb = (x[:, self.hv[:, k]] for k in range(4))
        ed, mid = _unit(p1 - p0), (p0 + p1) / 2
        qa, qb = (q - p0 - ed * _dot(q - p0, ed) for q in (pa, pb))
        cr = torch.linalg.cross(qa, qb)
        angle = torch.atan2(cr.norm(dim=-1, keepdim=True), _dot(qa, qb))
        half = (angle - self.rest[..., None]) / 2 * torch.where(_dot(cr, ed) >= 0, 1.0, -1.0)

        def turned(q, a):
            return (ed * _dot(ed, q) - q) * (1 - torch.cos(a)) + torch.linalg.cross(ed, q) * torch.sin(a)

        out = (turned(pa - mid, half) * self.st[..., 2:3] + turned(pb - mid, -half) * self.st[..., 3:4]) * self.hw[..., None]
        for k in range(4):
            r.index_add_(1, self.hv[:, k], out * self.st[..., k : k + 1])
        return r

    def _target(self, f):
        model, s = self.setups[0].model, self.setups
        if model == 4:
            return torch.eye(3, 2, device=DEV, dtype=torch.float64).expand_as(f)
        c = f.transpose(-1, -2) @ f
        a, b, d = c[..., 0, 0], c[..., 0, 1], c[..., 1, 1]
        th = 0.5 * torch.atan2(2 * b, a - d)
        v = torch.stack([torch.stack([th.cos(), -th.sin()], -1), torch.stack([th.sin(), th.cos()], -1)], -2)
        disc = torch.sqrt(((a - d) / 2) ** 2 + b * b)
        sig = torch.sqrt(torch.stack([(a + d) / 2 + disc, (a + d) / 2 - disc], -1).clamp_min(0))
        kw = _t([_f(q.warp_stiffness) for q in s])[:, None]
        kf = _t([_f(q.weft_stiffness) for q in s])[:, None]
        if model == 0:
            goal = torch.ones_like(sig)
        elif model == 1:
            goal = sig.clamp_max(1.0)
        elif model == 2:
            k = torch.stack([kw, kf], -1) / torch.maximum(kw, kf)[..., None]
            goal = sig + (1 - sig) * k
        else:
            c2 = v[..., 0, 0] ** 2
            k = torch.stack([kw * c2 + kf * (1 - c2), kw * (1 - c2) + kf * c2], -1)
            goal = torch.where(sig > 1, 1 + (sig - 1) * (1 - k), sig)
        return f @ (v * (goal / sig)[..., None, :]) @ v.transpose(-1, -2)


def _step64(c, cfg, x, vel, contact=None, lam=None):
    """One step of every garment; with `contact` the IPC step against ground and sphere (one garment)."""
    dt = _f(DT)
    grav = _t([_f(q) for q in cfg.gravity])
    prev, v = x, vel
    if contact is not None:
        d_hat = _f(cfg.barrier_d_hat) * _f(cfg.compliant_d_hat_scale)
        top = 0.5 * math.sqrt(d_hat) / dt
        speed = v.norm(dim=-1, keepdim=True)
        v = torch.where((speed > top) & ~c.pinned, v * (top / speed.clamp_min(1e-300)), v)
    pred = torch.where(c.pinned, x, x + dt * v + dt * dt * grav)
    if contact is not None:
        pred[..., 1] = torch.where(c.pinned[..., 0], pred[..., 1], pred[..., 1].clamp_min(_f(contact.ground_height)))
    x = pred
    if contact is None:
        for _ in range(cfg.max_iterations):
            d = c.solve(c.residual(x, pred, 1 / (dt * dt)))
            x = torch.where(c.pinned, prev, x + d)
    else:
        mu, active, normal = _f(cfg.al_mu_initial), 0, torch.zeros_like(x)
        for _ in range(cfg.al_max_iterations):
            grad, touch, n, _, _ = _barriers64(x, contact, d_hat)
            normal = torch.where(touch, n, normal)
            lam = torch.where(touch, lam, torch.zeros_like(lam))
            for _ in range(cfg.max_iterations):
                d = c.solve(c.residual(x, pred, 1 / (dt * dt)) - (mu * grad + lam))
                x = x + _alpha64(x, d, (grad * d).sum().item() * mu, (d * d).sum().item(), contact) * d
            grad, touch, n, active, worst = _barriers64(x, contact, d_hat)
            normal = torch.where(touch, n, normal)
            if worst < _f(cfg.al_tolerance):
                break
            lam = torch.where(touch, lam + mu * grad, lam)
            mu *= _f(cfg.al_mu_growth)
    v = (x - prev) / dt
    if contact is not None:
        v = _filter64(cfg, v, normal, active, x, _f(contact.ground_height))
    v = v * (1 - _f(cfg.damping))
    return x, torch.where(c.pinned, v, v / (1 + _f(cfg.rayleigh_mass_damping) * dt)), lam


def _barriers64(x, contact, d_hat):
    """(gradient, in contact, normal, contacts, deepest violation) of the ground and sphere barriers."""
    def slope(dsq):
        q = dsq.clamp(d_hat * 1e-3, d_hat)
        return torch.where(q >= d_hat, 0.0, -(q - d_hat) * (2 * torch.log(q / d_hat) + (q - d_hat) / q)) * _f(contact.kappa)

    off = x - _t([_f(q) for q in contact.sphere_center])
    r = off.norm(dim=-1, keepdim=True)
    up = torch.zeros_like(x)
    up[..., 1] = 1.0
    grad, normal = torch.zeros_like(x), torch.zeros_like(x)
    touch = torch.zeros_like(r, dtype=torch.bool)
    count, worst = 0, 0.0
    for dist, out in ((x[..., 1:2] - _f(contact.ground_height), up), (r - _f(contact.sphere_radius), off / r)):
        d = torch.where(dist <= 0, (-dist).clamp_min(1e-6), dist)
        near = (dist <= 0) | (dist * dist < d_hat)
        grad = grad + torch.where(near, slope(d * d) * 2 * d * out, torch.zeros_like(x))
        normal = normal + torch.where(near, out, torch.zeros_like(x))
        touch = touch | near
        count += int(near.sum())
        worst = max(worst, float((-dist).max()))
    return grad, touch, torch.where(touch, _unit(normal + (~touch) * up), normal), count, worst


def _alpha64(x, d, slope, dsq, contact):
    """The CCD bound of the step x -> x + d and the backtracking on it."""
    toi = 1.0
    h = _f(contact.ground_height)
    y0, y1 = x[..., 1], x[..., 1] + d[..., 1]
    hit = (y0 > h) & (y1 < h)
    if hit.any():
        toi = min(toi, float(((h - y0) / (y1 - y0))[hit].min()) * _f(0.9))
    p = x - _t([_f(q) for q in contact.sphere_center])
    a, b = _dot(d, d)[..., 0], 2 * _dot(p, d)[..., 0]
    k = _dot(p, p)[..., 0] - _f(contact.sphere_radius) ** 2
    disc = b * b - 4 * a * k
    t = (-b - disc.clamp_min(0).sqrt()) / (2 * a).clamp_min(1e-300)
    hit = (k >= 0) & (a > 1e-8) & (disc >= 0) & (t >= 0) & (t <= 1)
    if hit.any():
        toi = min(toi, float(t[hit].min()) * _f(0.9))
    alpha = max(toi, 1e-6)
    alpha = min(alpha * _f(0.8) if alpha < 1 else alpha, 1.0)
    for _ in range(4):
        if alpha < 0.1 or not slope > 1e-4 * dsq * 100.0:
            break
        alpha *= 0.5
    return alpha


def _filter64(cfg, v, normal, active, x, ground):
    """The inelastic velocity filter, friction and contact damping of the IPC step, and the ground's."""
    vn = _dot(v, normal)
    w = v - normal * vn
    speed = w.norm(dim=-1, keepdim=True)
    slip = _f(cfg.friction_coefficient) * vn.abs()
    w = torch.where(speed > 1e-8, w * (1 - slip / speed.clamp_min(1e-300)).clamp_min(0), w)
    slow = (1 - w.norm(dim=-1, keepdim=True) / _f(cfg.contact_velocity_threshold)).clamp(0, 1)
    cd = _f(cfg.contact_damping)
    w = w * (1 - (cd + slow * (_f(cfg.contact_damping_max) - cd)))
    v = torch.where(_dot(normal, normal) >= 0.5, w, v)
    if active:
        v = v * (1 - _f(0.05))
    low = x[..., 1] <= ground
    v[..., 1] = torch.where(low, v[..., 1].clamp_min(0), v[..., 1])
    for k in (0, 2):
        v[..., k] = torch.where(low, v[..., k] * 0.5, v[..., k])
    return v


def _resolve64(c, x, v, contact):
    free = ~c.pinned[..., 0]
    h = _f(contact.ground_height)
    low = (x[..., 1] < h) & free
    x, v = x.clone(), v.clone()
    x[..., 1] = torch.where(low, h, x[..., 1])
    v[..., 1] = torch.where(low, v[..., 1].clamp_min(0), v[..., 1])
    for k in (0, 2):
        v[..., k] = torch.where(low, v[..., k] * 0.5, v[..., k])
    off = x - _t([_f(q) for q in contact.sphere_center])
    r, n = off.norm(dim=-1, keepdim=True), _unit(off)
    inside = (r < _f(contact.sphere_radius)) & free[..., None]
    vn = _dot(v, n)
    x = torch.where(inside, x + n * (_f(contact.sphere_radius) - r), x)
    return x, torch.where(inside & (vn < 0), (v - n * vn) * 0.5, v)


def exact(case, seed):
    kind = case["kind"]
    if kind == "pairs" or kind == "drapes" or case.get("self", False):
        # pairs are whole numbers; a step with self contact would be the whole contact pipeline over again
        return None
    if kind in ("solve", "refactor"):
        ptr, col, val, rhs = _matrix(case, seed)
        n = len(ptr) - 1
        a = torch.zeros(n, n, device=DEV, dtype=torch.float64)
        rows = torch.as_tensor(np.repeat(np.arange(n), np.diff(ptr.astype(np.int64))), device=DEV)
        a[rows, torch.as_tensor(col.astype(np.int64), device=DEV)] = _t(val)
        return list(torch.cholesky_solve(_t(rhs).T.contiguous(), torch.linalg.cholesky(a)).T.cpu())
    cfg = _config(case)
    if kind == "batch":
        sides = _sides(case, seed)
        rng = np.random.default_rng(seed + 7)
        meshes = [scenarios.hanging_sheet(s, float(rng.uniform(0.5, 2.0))) for s in sides]
        setups = _materials(case, seed, len(meshes))
        start = np.concatenate([np.stack([m.px, m.py, m.pz], 1) for m in meshes])
        free = np.concatenate([m.pinned == 0 for m in meshes])
        start = (start + 1e-3 * rng.uniform(-1, 1, start.shape).astype(np.float32) * free[:, None]).astype(np.float32)
        at = np.cumsum([0] + [m.nv for m in meshes])
        out = np.zeros(start.shape)
        for s in sorted(set(sides)):
            mine = [k for k in range(len(sides)) if sides[k] == s]
            for some in (mine[k : k + 32] for k in range(0, len(mine), 32)):
                c = _Cloth64([np.stack([meshes[k].px, meshes[k].py, meshes[k].pz], 1) for k in some], meshes[some[0]].tris,
                             meshes[some[0]].pinned, [setups[k] for k in some], s)
                x = _t([start[at[k] : at[k + 1]] for k in some])
                x = _step64(c, cfg, x, torch.zeros_like(x))[0].cpu().numpy()
                for k, xk in zip(some, x):
                    out[at[k] : at[k + 1]] = xk
        return out
    mesh, pinned, pos, vel = _garment(case, seed)
    cols = case["cols"]
    c = _Cloth64([np.stack([mesh.px, mesh.py, mesh.pz], 1)], mesh.tris, np.zeros(mesh.nv) if pinned is None else pinned,
                 _materials(case, seed, 1), cols)
    x, v = _t(pos)[None], _t(vel)[None]
    lam = torch.zeros_like(x)
    for _ in range(case["steps"]):
        x, v, lam = _step64(c, cfg, x, v, _contact(case) if kind == "ipc" else None, lam)
        if kind == "resolve":
            x, v = _resolve64(c, x, v, _contact(case))
    return x[0].cpu() if kind == "ipc" else (x[0].cpu(), v[0].cpu())
