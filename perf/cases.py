"""Performance cases of the CBS step engine: the calls a user's program makes
through cbs-3d_b200/cbs3d/gpu.py, from the smallest meshes (where launches and
the latency of a solver iteration count) to the largest (where memory counts).

Kinds of case
  cavity     lid-driven cavity: steps of a running simulation, then the fields
  channel    parabolic inlet, outlet at zero pressure (another pressure system:
             many fixed-pressure rows, a long thin domain)
  cht        conjugate heat transfer slab: energy equation, material
             properties, solid elements without pressure rows
  coupled    the fields handed in, one step, the fields handed back: another
             code owns the state (partitioned coupling, data assimilation)
  batch      many cavities of uneven size advanced together
  pressure   the pressure-solver drop-in on host arrays
  adjoint    objective and its gradient for a body force: forward steps with
             checkpoints and the reverse sweep

A cavity may run with the multigrid or the two-level preconditioner or with
the mixed-precision solver.  Sizes are those of the repository's tests,
configurations and benchmark, and the range between them.
"""
from __future__ import annotations

import functools
import importlib
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "cbs-3d_b200"))
mesh_cases = importlib.import_module("cbs3d.cases")
gpu = importlib.import_module("cbs3d.gpu")

FOREVER = 10 ** 6   # ntime of a run that is stepped on by hand


def listed():
    return [
        # the smallest coupled call: launches, copies and iteration latency
        dict(name="coupled_8", kind="coupled", n=8, jitter=0.0, re=100.0),
        # the 16^3 validation cavity, twenty steps between two outputs
        dict(name="cavity_16", kind="cavity", n=16, jitter=0.0, re=100.0, steps=20, solver="jacobi"),
        # an odd size between the configurations, jittered
        dict(name="cavity_37", kind="cavity", n=37, jitter=0.15, re=400.0, steps=4, solver="jacobi"),
        # the 64^3 benchmark cavity, the ordinary production size
        dict(name="cavity_64", kind="cavity", n=64, jitter=0.15, re=400.0, steps=3, solver="jacobi"),
        # the largest: more than the register-resident solvers and L2 hold
        dict(name="cavity_88", kind="cavity", n=88, jitter=0.15, re=400.0, steps=1, solver="jacobi"),
        # the 96x16x16 channel configuration
        dict(name="channel_96", kind="channel", nx=96, ny=16, nz=16, length=6.0, re=100.0, steps=5),
        # the conjugate heat transfer configuration (552,960 tets)
        dict(name="cht_128", kind="cht", nx=128, ny=24, ny_solid=6, nz=24, re=200.0, steps=3),
        # the multigrid-preconditioned solve (the counterpart of an AMG option)
        dict(name="multigrid_48", kind="cavity", n=48, jitter=0.15, re=400.0, steps=3, solver="multigrid"),
        # FP32 inner solves, to a tolerance below FP32's own
        dict(name="mixed_24", kind="cavity", n=24, jitter=0.15, re=400.0, steps=3, solver="mixed"),
        # a parameter study: uneven cavities advanced together
        dict(name="batch_12", kind="batch", count=12, n_lo=10, n_hi=32, sizes=2024, steps=2),
        # the pressure backend inside another code's step loop
        dict(name="pressure_31", kind="pressure", n=31, jitter=0.15),
        # gradient of a mean kinetic energy for a body force
        dict(name="adjoint_48", kind="adjoint", nx=48, ny=8, nz=8, steps=20, every=5),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["cavity", "coupled", "channel", "cht", "batch", "pressure", "adjoint"],
                       [40, 10, 15, 10, 9, 8, 8])[0]
    if kind in ("cavity", "coupled"):
        solver = "jacobi" if kind == "coupled" else rng.choices(["jacobi", "multigrid", "two_level", "mixed"],
                                                                [6, 2, 1, 1])[0]
        # the mixed solver takes several times the iterations; the two-level
        # preconditioner exists for meshes of this size and above
        n = _log_int(rng, 50 if solver == "two_level" else 4, {"mixed": 40, "two_level": 72, "multigrid": 72}.get(solver, 86))
        c = dict(kind=kind, n=n, jitter=rng.choice([0.0, 0.15]), re=round(rng.uniform(50.0, 400.0), 1))
        if kind == "cavity":
            most = 3 if solver == "mixed" else max(1, min(20, int(5e6 / n ** 3.5)))
            c.update(steps=rng.randint(1, most), solver=solver)
        return c
    if kind == "channel":
        ny = _log_int(rng, 4, 24)
        return dict(kind=kind, nx=_log_int(rng, 8, 128), ny=ny, nz=max(3, ny + rng.randint(-2, 2)),
                    length=float(rng.choice([2.0, 4.0, 6.0])), re=round(rng.uniform(50.0, 150.0), 1),
                    steps=rng.randint(1, 5))
    if kind == "cht":
        ny = _log_int(rng, 4, 24)
        return dict(kind=kind, nx=_log_int(rng, 8, 128), ny=ny, ny_solid=max(2, ny // 4), nz=max(3, ny + rng.randint(-2, 2)),
                    re=round(rng.uniform(100.0, 200.0), 1), steps=rng.randint(1, 3))
    if kind == "batch":
        lo = rng.randint(4, 12)
        return dict(kind=kind, count=rng.randint(3, 24), n_lo=lo, n_hi=lo + rng.randint(4, 18),
                    sizes=rng.randint(1, 9999), steps=rng.randint(1, 3))
    if kind == "pressure":
        return dict(kind=kind, n=_log_int(rng, 4, 48), jitter=rng.choice([0.0, 0.15]))
    m = rng.randint(4, 9)
    return dict(kind=kind, nx=_log_int(rng, 10, 48), ny=m, nz=max(3, m + rng.randint(-1, 1)), steps=rng.randint(4, 16),
                every=rng.randint(2, 8))


# ------------------------------------------------------------------- meshes
@functools.lru_cache(maxsize=3)
def _cavity(n, jitter, re, rel_tol):
    return mesh_cases.cavity(n, re=re, ntime=FOREVER, jitter=jitter, seed=1234, relToler=rel_tol)


def _mesh_case(c):
    if c["kind"] in ("cavity", "coupled"):
        mixed = c.get("solver") == "mixed"
        return _cavity(c["n"], c["jitter"], c["re"], 1e-12 if mixed else 1e-10)
    if c["kind"] == "channel":
        return mesh_cases.channel(c["nx"], c["ny"], c["nz"], length=c["length"], re=c["re"], ntime=FOREVER)
    if c["kind"] == "cht":
        return mesh_cases.cht_slab(c["nx"], c["ny"], c["ny_solid"], c["nz"], re=c["re"], ntime=FOREVER)
    return mesh_cases.channel_adjoint(c["nx"], c["ny"], c["nz"], length=c["nx"] / 16.0, dtfix=0.01, ntime=FOREVER)


def _disturbed(case, u, p, t, seed):
    """The initial fields with a smooth seeded disturbance that vanishes on
    the fluid's boundary: the state of a run that is under way."""
    rng = np.random.default_rng(seed)
    x = case.mesh.coord
    hi = x.max(axis=0)
    s = np.clip(x / hi, 0.0, 1.0)     # the solid of a slab lies at y < 0
    u = u.reshape(-1, 3).copy()
    t = t.copy()
    fluid = np.ones(x.shape[0], dtype=bool)
    if case.mesh.mat_elem is not None:
        fluid[np.unique(case.mesh.intma[case.mesh.mat_elem != 0]) - 1] = False
    for _ in range(3):
        k = rng.integers(1, 4, size=3)
        mode = np.prod(np.sin(np.pi * k * s), axis=1) * fluid
        u += 0.05 * mode[:, None] * rng.normal(size=3)
        t += 0.05 * mode * rng.normal()
    return u.ravel(), p, t


# ----------------------------------------------------------------- pressure
_PAIRS = ((0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3))


@functools.lru_cache(maxsize=2)
def _stiffness(n, jitter):
    """Element Laplacians of a cavity mesh: (intma, diagonals [E,4], pairs [E,6])."""
    m = mesh_cases.box_mesh(n, n, n, jitter=jitter, seed=1234)
    x = m.coord[m.intma - 1]
    jac = x[:, 1:] - x[:, :1]
    grad = np.empty((m.nelem, 4, 3))
    grad[:, 1:] = np.linalg.inv(jac).transpose(0, 2, 1)
    grad[:, 0] = -grad[:, 1:].sum(axis=1)
    k = np.einsum("ead,ebd->eab", grad, grad) * (np.linalg.det(jac) / 6.0)[:, None, None]
    return m.intma, k[:, range(4), range(4)], np.stack([k[:, a, b] for a, b in _PAIRS], axis=1)


def _pressure_system(c, seed):
    """A step's pressure system on host arrays: element time steps, the
    operator they scale, a right-hand side and the previous pressure."""
    rng = np.random.default_rng(seed)
    intma, diag, pairs = _stiffness(c["n"], c["jitter"])
    npoin = int(intma.max())
    dt = rng.uniform(0.5, 1.5, size=len(intma)) * 0.25 / c["n"]
    pdiag = np.bincount((intma - 1).ravel(), (diag * dt[:, None]).ravel(), minlength=npoin)
    rhs = rng.normal(size=npoin) / c["n"] ** 3
    rhs -= rhs.mean()
    pres = 0.1 * rng.normal(size=npoin)
    pres[0] = 0.0
    return intma, np.ascontiguousarray(pairs * dt[:, None]), pdiag, rhs, pres


# ------------------------------------------------------------------ prepare
def _batch_case(c, seed):
    cs = mesh_cases.cavity_batch(count=c["count"], n_lo=c["n_lo"], n_hi=c["n_hi"], seed=c["sizes"], ntime=FOREVER,
                                 rel_tol=1e-10)
    re = np.exp(np.random.default_rng(seed).uniform(np.log(50.0), np.log(400.0), size=len(cs)))
    for case, r in zip(cs, re):
        case.params["re"] = float(r)
    return cs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return kind, gpu.Batch(_batch_case(case, seed), autotune=False), case["steps"]
    if kind == "pressure":
        intma, pairs, pdiag, rhs, pres = _pressure_system(case, seed)
        solver = gpu.PressureSolver(intma, None, np.array([1]), np.array([0.0]))
        return kind, solver, (pairs, pdiag, rhs, pres)
    mc = _mesh_case(case)
    solver = case.get("solver", "jacobi")
    ctx = gpu.Context(mc, multigrid=solver == "multigrid", two_level=solver == "two_level",
                      precision=gpu.MIXED if solver == "mixed" else gpu.FP64)
    if kind == "adjoint":
        rng = np.random.default_rng(seed)
        ctx.set_body_force(rng.normal(0.0, 0.01, size=3 * mc.mesh.npoin))
        hi = float(mc.mesh.coord[:, 0].max())
        weights = mesh_cases.region_weights(mc, lo=0.6 * hi, hi=0.8 * hi)
        return kind, ctx, (case["steps"], weights, case["every"])
    fields = _disturbed(mc, *ctx.fields(), seed)
    ctx.upload(*fields)
    if kind == "coupled":
        return kind, ctx, fields
    return kind, ctx, (case["steps"], kind == "cht")


def run(state):
    kind, handle, args = state
    if kind == "batch":
        handle.step(args)
        return [handle.fields(i)[:2] for i in range(handle.n)]
    if kind == "pressure":
        return handle.solve(*args, relToler=1e-12)[:3]
    if kind == "adjoint":
        steps, weights, every = args
        objective, grad = handle.adjoint(steps, weights, every=every)
        return {"objective": np.array([objective]), "grad": grad}
    if kind == "coupled":
        handle.upload(*args)
        handle.step(1)
        return handle.fields()[:2]
    steps, with_temperature = args
    handle.step(steps)
    return handle.fields()[:3 if with_temperature else 2]


# --------------------------------------------------------------------- work
def _size(c):
    """(tets, nodes, pressure iterations of a solve): the iterations of
    Jacobi-PCG grow with the mesh's width -- about 12 n for a cavity and 4 per
    cell of the longest side where an outlet fixes the pressure; a multigrid
    takes about 60 whatever the size."""
    if c["kind"] in ("cavity", "coupled", "pressure"):
        n = c["n"]
        its = {"multigrid": 60, "two_level": 5 * n}.get(c.get("solver"), 12 * n)
        return 6 * n ** 3, (n + 1) ** 3, its
    ny = c["ny"] + c.get("ny_solid", 0)
    return 6 * c["nx"] * ny * c["nz"], (c["nx"] + 1) * (ny + 1) * (c["nz"] + 1), 4 * max(c["nx"], ny, c["nz"])


def work(case):
    """Bytes: per step the mesh (16 B of connectivity per tet, coordinates)
    and the fields read once and written once.  Operations: about 1,500 per
    tet outside the pressure solve, and per pressure iteration 15 multiply-
    adds of the operator's row and 6 of the vectors for every node."""
    if case["kind"] == "batch":
        rng = np.random.default_rng(case["sizes"])
        sizes = [(6 * n ** 3, (n + 1) ** 3, 12 * n)
                 for n in rng.integers(case["n_lo"], case["n_hi"] + 1, size=case["count"]).tolist()]
        steps = case["steps"]
    else:
        sizes = [_size(case)]
        steps = case.get("steps", 1) * (3 if case["kind"] == "adjoint" else 1)   # forward, again, and back
    if case["kind"] == "pressure":
        e, n, its = sizes[0]
        return {"bytes": 48.0 * e + 48.0 * n, "flops": 42.0 * n * its}
    return {"bytes": float(steps * sum(16 * e + 104 * n for e, n, _ in sizes)),
            "flops": float(steps * sum(1500 * e + 42 * n * its for e, n, its in sizes))}


# -------------------------------------------------------------------- exact
def exact(case, seed):
    """The pressure system's solution in 64 bits (conjugate gradients of plain
    torch, restarted on the true residual until it stops falling).  A whole
    step has no closed value to state here: None."""
    if case["kind"] != "pressure":
        return None
    intma, pairs, pdiag, rhs, pres = _pressure_system(case, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    e = torch.as_tensor(intma.astype(np.int64) - 1, device=dev)
    g = torch.as_tensor(pairs, device=dev)
    d = torch.as_tensor(pdiag, device=dev)
    b = torch.as_tensor(rhs, device=dev)
    n = d.numel()
    rows = torch.cat([e[:, a] for a, _ in _PAIRS] + [e[:, c] for _, c in _PAIRS] + [torch.arange(n, device=dev)])
    cols = torch.cat([e[:, c] for _, c in _PAIRS] + [e[:, a] for a, _ in _PAIRS] + [torch.arange(n, device=dev)])
    vals = torch.cat([g[:, k] for k in range(6)] * 2 + [d])
    free = (rows != 0) & (cols != 0)     # node 1 is fixed at zero
    A = torch.sparse_coo_tensor(torch.stack([rows[free], cols[free]]), vals[free], (n, n)).coalesce().to_sparse_csr()
    b = b.clone()
    b[0] = 0.0
    x = torch.zeros_like(b)
    best = math.inf
    for _ in range(6):
        r = b - A @ x
        norm = float(r.norm())
        if norm >= 0.5 * best:
            break
        best = norm
        y, z = torch.zeros_like(b), r / d
        p, rz = z.clone(), torch.dot(r, z)
        for it in range(40 * case["n"] + 200):
            q = A @ p
            alpha = rz / torch.dot(p, q)
            y += alpha * p
            r -= alpha * q
            if it % 50 == 49 and float(r.norm()) < 1e-13 * norm:
                break
            z = r / d
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
        x += y
    rhs, pdiag = rhs.copy(), pdiag.copy()
    rhs[0], pdiag[0] = 0.0, 1.0
    return x.cpu().numpy(), rhs, pdiag
