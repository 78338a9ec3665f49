"""Performance cases of gschism_b200: the calls a forecast program makes, over the sizes, precisions
and options it makes them with.

Kinds of case (`kind`):

* ``forecast``   a forecast in a resident member slot: the slot's start state is put back from
                 page-locked memory (`Model.put_member_state`), the model steps to the horizon and the
                 elevation and the nodal velocities and tracers come back to page-locked memory.
* ``step``       a running simulation advances by a few steps and its elevation and nodal velocities
                 are read: one basin, or an ensemble of members of uneven size in one context.
* ``elevation``  the wave-equation block alone on a given elevation and solution history: side terms,
                 assembly, the JCG solve and the elevation update (`Model.phase`).
* ``transport``  offline tracer transport: the flow is held and the tracers take several steps
                 (upwind, TVD, or TVD with the flux-corrected vertical step).
* ``csr``        the stand-alone JCG on a caller's CSR matrix (`PCGSolverMultiGPU`), a new right-hand
                 side at every call.
* ``noalloc``    the allocation-free FP64 JCG on a caller's CSR matrix (`gs_jcg_solve_csr_noalloc`).

Meshes and forcing come from `gschism_b200.cases` (jittered lattices, 500 m spacing, Gaussian random
field bathymetry), seeded by `seed`.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from gschism_b200 import _lib as L
from gschism_b200 import cases
from gschism_b200.model import INT_FIELDS, Model
from gschism_b200.solver import PCGSolverMultiGPU

SPACING = 500.0
SOLVE_FIELDS = ("ETA2", "JCG_X", "JCG_X1", "JCG_X2")
ELEVATION_PHASES = ("PREPARE", "ASSEMBLE", "SOLVE", "UPDATE_ELEV")


def listed():
    return [
        # the 10 km channel of the parity tests, plain FP64: the smallest mesh that is run in earnest,
        # where kernel launches and the solver's synchronisation count
        dict(name="channel_forecast_fp64", kind="forecast", nx=63, ny=32, levels=10, tracers=1, precision="fp64",
             steps=10, storm=False),
        # a storm-surge request on a region mesh of the serving scenario, admitted into its slot
        dict(name="storm_forecast_30k", kind="forecast", nx=173, ny=173, levels=20, tracers=1, precision="fp32_ir",
             steps=8, storm=True),
        # the single large mesh of the benchmark (30 SZ levels, T and S) at a sixth of its node count
        dict(name="basin_step_160k", kind="step", members=1, nodes_min=160000, nodes_max=160000, levels=30,
             tracers=2, precision="fp32_ir", steps=4),
        # the plain FP64 form of the step on a ragged mid-size mesh
        dict(name="basin_step_fp64_62k", kind="step", members=1, nodes_min=63001, nodes_max=63001, levels=8,
             tracers=1, precision="fp64", steps=4),
        # ensemble members of uneven size in one context, one launch per phase
        dict(name="ensemble_step", kind="step", members=8, nodes_min=8000, nodes_max=50000, levels=20, tracers=1,
             precision="fp32_ir", steps=4),
        # the elevation block of the benchmark's mesh (1M rows; levels do not enter the solve)
        dict(name="elevation_1M", kind="elevation", side=1000, levels=4, precision="fp32_ir"),
        # the same block in plain FP64 on an ordinary mesh
        dict(name="elevation_fp64_200k", kind="elevation", side=447, levels=4, precision="fp64"),
        # transport of T and S with the reference's upwind scheme
        dict(name="transport_upwind", kind="transport", side=300, levels=30, tracers=2, itr_met=1, limiter=3,
             dfh0=0.0, steps=6),
        # transport stress: sharp fronts, 40 levels, 5 tracers, TVD with vertical diffusion
        dict(name="transport_tvd", kind="transport", side=200, levels=40, tracers=5, itr_met=3, limiter=3,
             dfh0=1e-4, steps=4),
        # TVD with the flux-corrected vertical step on a small mesh
        dict(name="transport_fct_small", kind="transport", side=101, levels=23, tracers=1, itr_met=4, limiter=4,
             dfh0=0.0, steps=4),
        # a caller's own matrix through the drop-in solver class, mixed precision
        dict(name="csr_250k", kind="csr", side=500, precision="fp32_ir"),
        # a small system from a caller that cannot allocate
        dict(name="noalloc_10k", kind="noalloc", side=101),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forecast", "step", "step", "elevation", "elevation", "transport", "csr", "noalloc"])
    prec = rng.choice(["fp32_ir", "fp32_ir", "fp64"])
    if kind == "forecast":
        storm = rng.random() < 0.5
        nx = _logint(rng, 20, 170)
        return dict(kind=kind, nx=nx, ny=nx if storm else _logint(rng, 15, 90), levels=rng.randint(8, 20),
                    tracers=1, precision=prec, steps=rng.randint(4, 8), storm=storm)
    if kind == "step":
        members = rng.choice([1, 1, 2, 3, 5, 8])
        lo = _logint(rng, 2500, 12000)
        hi = _logint(rng, lo, 150000 // members)
        levels = rng.randint(6, 30)
        return dict(kind=kind, members=members, nodes_min=lo, nodes_max=max(lo, hi), levels=levels,
                    tracers=rng.randint(1, 2), precision=prec, steps=rng.randint(1, 4))
    if kind == "elevation":
        return dict(kind=kind, side=_logint(rng, 40, 900 if prec == "fp32_ir" else 440), levels=rng.randint(4, 6),
                    precision=prec)
    if kind == "transport":
        tracers = rng.randint(1, 5)
        return dict(kind=kind, side=_logint(rng, 30, 240 if tracers < 3 else 170), levels=rng.randint(9, 40),
                    tracers=tracers, itr_met=rng.choice([1, 3, 4]), limiter=rng.randint(1, 4),
                    dfh0=rng.choice([0.0, 1e-4]), steps=rng.randint(2, 6))
    if kind == "csr":
        return dict(kind=kind, side=_logint(rng, 30, 490), precision=prec)
    return dict(kind=kind, side=_logint(rng, 20, 250))


# ------------------------------------------------------------------------------- inputs ----

def _pinned(shape, dtype):
    t = torch.zeros(shape, dtype=dtype).pin_memory()
    return t, t.numpy()


def _out(model, members, fields):
    """Page-locked output arrays per (member, field), and the tensors that own them."""
    keep, out = [], []
    for m in range(members):
        for f in fields:
            t, a = _pinned(model.shape(m, f), torch.int32 if f in INT_FIELDS else torch.float64)
            keep.append(t)
            out.append((m, f, a))
    return keep, out


def _read(state):
    res = {}
    for m, f, a in state["out"]:
        res["%s_%d" % (f, m)] = state["model"].get_into(m, f, a)
    return res


def _basin(seed, side, levels, tracers):
    """A basin at the benchmark's spacing, tide ramped up over about an hour, so that the flow has
    developed after the spin-up steps."""
    rng = np.random.default_rng(seed)
    mag, ang = rng.uniform(0.05, 0.3), rng.uniform(0.0, 2.0 * math.pi)
    c = cases.basin(seed=seed, n=side, nvrt=levels, nz=max(2, levels // 3), ntr=tracers, length=SPACING * side,
                    amp=rng.uniform(0.6, 1.2), tau=(mag / 1025.0 * math.cos(ang), mag / 1025.0 * math.sin(ang)))
    c.params.dramp = 0.05
    return c


def _prepare_forecast(case, seed):
    if case["storm"]:
        c = _basin(seed, case["nx"], case["levels"], case["tracers"])
        vortex = cases.storm_on(c, seed)
    else:
        c = cases.channel(seed=seed, nx=case["nx"], ny=case["ny"], nvrt=case["levels"])
        c.params.dramp = 0.05
        vortex = None
    m = Model([c], precision=case["precision"])
    if vortex is not None:
        m.set_vortex(0, vortex)
    m.step(6)
    start = m.current_step()
    keep, out = _out(m, 1, ("ETA2", "NODE_U2", "NODE_TR"))
    return dict(kind="forecast", model=m, start=m.member_state(0, pinned=True), first=start, steps=case["steps"],
                keep=keep, out=out)


def _prepare_step(case, seed):
    rng = np.random.default_rng(seed + 1)
    lo, hi = case["nodes_min"], case["nodes_max"]
    cs = []
    for k in range(case["members"]):
        # the members' sizes span the range whatever the seed, so that every seed is the same work
        f = (k + 0.5) / case["members"]
        side = max(8, int(round(math.sqrt(lo * (hi / lo) ** f))))
        cs.append(_basin(int(rng.integers(1, 2 ** 31 - 1)), side, case["levels"], case["tracers"]))
    m = Model(cs, precision=case["precision"])
    m.step(24)
    m.sync()
    keep, out = _out(m, len(cs), ("ETA2", "NODE_U2"))
    return dict(kind="step", model=m, steps=case["steps"], keep=keep, out=out)


def _prepare_elevation(case, seed):
    m = Model([_basin(seed, case["side"], case["levels"], 1)], precision=case["precision"])
    m.step(8)
    m.phase("BEGIN", 9)
    m.phase("BTRACK", 9)
    keep, start = [], {}
    for f in SOLVE_FIELDS:
        t, a = _pinned(m.shape(0, f), torch.float64)
        m.get_into(0, f, a)
        keep.append(t)
        start[f] = a
    k2, out = _out(m, 1, ("ETA2",))
    return dict(kind="elevation", model=m, start=start, keep=keep + k2, out=out)


def _prepare_transport(case, seed):
    c = cases.transport_stress(seed=seed, n=case["side"], nvrt=case["levels"], ntr=case["tracers"], tau_mag=0.3,
                               limiter=case["limiter"], dfh0=case["dfh0"])
    c.params.itr_met = case["itr_met"]
    m = Model([c])
    m.step(8)
    m.sync()
    keep, out = _out(m, 1, ("NODE_TR",))
    return dict(kind="transport", model=m, steps=case["steps"], keep=keep, out=out)


def _system(side, seed):
    """CSR of an elevation-like system on a jittered lattice of side x side nodes (linear triangles:
    mass plus (theta c dt)^2 stiffness over a smooth random depth, one essential side), built on the
    GPU in FP64, columns sorted; and four smooth right-hand sides."""
    dev, f8 = torch.device("cuda", 0), torch.float64
    g = torch.Generator(device=dev).manual_seed(seed)
    n = side * side
    ids = torch.arange(n, device=dev)
    i, j = ids % side, ids // side
    jit = (torch.rand(2, n, generator=g, device=dev, dtype=f8) - 0.5) * 0.4
    edge_x, edge_y = (i == 0) | (i == side - 1), (j == 0) | (j == side - 1)
    x = (i + torch.where(edge_x, torch.zeros_like(jit[0]), jit[0])) * SPACING
    y = (j + torch.where(edge_y, torch.zeros_like(jit[1]), jit[1])) * SPACING

    def smooth(waves):
        v = torch.zeros(n, device=dev, dtype=f8)
        p = torch.rand(waves, 4, generator=g, device=dev, dtype=f8)
        for k in range(waves):
            kx, ky = (p[k, 0] - 0.5) * 4e-4, (p[k, 1] - 0.5) * 4e-4
            v += (0.2 + p[k, 2]) * torch.cos(kx * x + ky * y + 6.283185307179586 * p[k, 3])
        return v

    h = smooth(8)
    h = 5.0 + 3000.0 * (h - h.min()) / (h.max() - h.min())
    cell = ids[(i < side - 1) & (j < side - 1)]
    a, b, c, d = cell, cell + 1, cell + 1 + side, cell + side
    tri = torch.cat([torch.stack([a, b, c], 1), torch.stack([a, c, d], 1)])
    X, Y = x[tri], y[tri]
    bx = torch.stack([Y[:, 1] - Y[:, 2], Y[:, 2] - Y[:, 0], Y[:, 0] - Y[:, 1]], 1)
    by = torch.stack([X[:, 2] - X[:, 1], X[:, 0] - X[:, 2], X[:, 1] - X[:, 0]], 1)
    area = 0.5 * (bx[:, 0] * by[:, 1] - bx[:, 1] * by[:, 0])
    coef = 9.81 * (0.6 * 120.0) ** 2 * h[tri].mean(1)
    rows, cols, vals = [], [], []
    for p in range(3):
        for q in range(3):
            rows.append(tri[:, p])
            cols.append(tri[:, q])
            vals.append(area * (2.0 if p == q else 1.0) / 12.0
                        + coef * (bx[:, p] * bx[:, q] + by[:, p] * by[:, q]) / (4.0 * area))
    R, C, V = torch.cat(rows), torch.cat(cols), torch.cat(vals)
    ess = i == 0                                   # identity rows, their columns moved to the right-hand side
    V = torch.where(ess[R] | ess[C], torch.zeros_like(V), V)
    R, C, V = torch.cat([R, ids]), torch.cat([C, ids]), torch.cat([V, ess.to(f8)])
    # entries of one position are added in a fixed order, so that a seed gives one matrix
    key, order = torch.sort(R * n + C, stable=True)
    key, counts = torch.unique_consecutive(key, return_counts=True)
    val = torch.segment_reduce(V[order], "sum", lengths=counts)
    row = key // n
    ptr = torch.zeros(n + 1, device=dev, dtype=torch.int64)
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    rhs = [smooth(6) * SPACING * SPACING for _ in range(4)]
    for r in rhs:
        r[ess] = 0.5
    return ptr.to(torch.int32), (key % n).to(torch.int32), val, rhs


def _prepare_csr(case, seed):
    ptr, idx, val, rhs = _system(case["side"], seed)
    s = PCGSolverMultiGPU(None, [rhs[0].numel()], [val.numel()], precision=case["precision"])
    s.csr_indptr(0).copy_(ptr)
    s.csr_indices(0).copy_(idx)
    s.csr_data(0).copy_(val)
    torch.cuda.synchronize()
    return dict(kind="csr", solver=s, rhs=rhs, turn=0)


def _prepare_noalloc(case, seed):
    ptr, idx, val, rhs = _system(case["side"], seed)
    return dict(kind="noalloc", lib=L.load(), ptr=ptr, idx=idx, val=val, rhs=rhs, turn=0,
                x=torch.zeros_like(rhs[0]))


def prepare(case, seed):
    seed = int(seed) % (2 ** 31 - 1) + 1
    return {"forecast": _prepare_forecast, "step": _prepare_step, "elevation": _prepare_elevation,
            "transport": _prepare_transport, "csr": _prepare_csr, "noalloc": _prepare_noalloc}[case["kind"]](case, seed)


# ------------------------------------------------------------------------------- passes ----

def run(state):
    kind = state["kind"]
    if kind == "forecast":
        m = state["model"]
        m.put_member_state(0, state["start"])
        # the member's clock: its step is the context's step less this offset
        m.set_member_start(0, m.current_step() - state["first"])
        m.step(state["steps"])
        return _read(state)
    if kind == "step":
        state["model"].step(state["steps"])
        return _read(state)
    if kind == "elevation":
        m = state["model"]
        for f in SOLVE_FIELDS:
            m.put(0, f, state["start"][f])
        for ph in ELEVATION_PHASES:
            m.phase(ph, 9)
        return _read(state)
    if kind == "transport":
        m = state["model"]
        for _ in range(state["steps"]):
            m.phase("TRANSPORT", 9)
        return _read(state)
    b = state["rhs"][state["turn"] % len(state["rhs"])]
    state["turn"] += 1
    if kind == "csr":
        s = state["solver"]
        s.b_m[0].copy_(b)
        s.solve(rtol=1e-12, maxiter=4000, checkEvery=10)
        return s.x_m[0].clone()
    x = state["x"].zero_()
    its = ctypes.c_int(0)
    p = [ctypes.c_void_p(t.data_ptr()) for t in (state["ptr"], state["idx"], state["val"], b, x)]
    L.check(state["lib"].gs_jcg_solve_csr_noalloc(x.numel(), *p, 1e-12, 4000, 10,
                                                  ctypes.c_void_p(torch.cuda.current_stream().cuda_stream),
                                                  ctypes.byref(its)), None, "gs_jcg_solve_csr_noalloc")
    return x


# ------------------------------------------------------------------ bytes, tolerances ----

def _counts(n):
    """Nodes, elements, sides and matrix entries of a triangulated lattice of n nodes."""
    e = 2.0 * n
    s = 3.0 * n
    return n, e, s, 7.0 * n


def _elevation_bytes(n, levels):
    """Velocity and backtracked-velocity columns and level heights of the sides, connectivity, the
    elevations; the matrix is made and used in place, so only the solution comes out."""
    n, e, s, _ = _counts(n)
    return s * levels * 40.0 + s * 60.0 + e * 60.0 + n * 60.0


def _transport_bytes(n, levels, tracers):
    n, e, s, _ = _counts(n)
    return 2.0 * e * levels * tracers * 8.0 + s * levels * 8.0 + 2.0 * e * levels * 8.0 + n * levels * tracers * 8.0


def _step_bytes(n, levels, tracers):
    """One step: the prognostic state (nodal and side velocities, heights, tracers) read and written
    once, the mesh read once."""
    _, e, s, nnz = _counts(n)
    state = n * levels * (32.0 + 8.0 * tracers) + s * levels * 24.0 + e * levels * (8.0 + 8.0 * tracers)
    return 2.0 * state + n * 100.0 + s * 60.0 + e * 160.0


def work(case):
    kind = case["kind"]
    if kind == "forecast":
        n = float(case["nx"] * case["ny"])
        b = case["steps"] * _step_bytes(n, case["levels"], case["tracers"])
        points = n * case["levels"] * case["steps"]
    elif kind == "step":
        lo, hi, k = case["nodes_min"], case["nodes_max"], case["members"]
        n = sum(lo * (hi / lo) ** ((i + 0.5) / k) for i in range(k))
        b = case["steps"] * _step_bytes(n, case["levels"], case["tracers"])
        points = n * case["levels"] * case["steps"]
    elif kind == "elevation":
        n = float(case["side"] ** 2)
        b, points = _elevation_bytes(n, case["levels"]), n * case["levels"]
    elif kind == "transport":
        n = float(case["side"] ** 2)
        b = case["steps"] * _transport_bytes(n, case["levels"], case["tracers"])
        points = n * case["levels"] * case["steps"]
    else:
        n = float(case["side"] ** 2)
        b, points = 7.0 * n * 12.0 + 24.0 * n, n
    return {"bytes": b, "flops": 100.0 * points}


def tolerance(case):
    # Everything is FP64 at the outside; what two correct implementations differ by is the solver's
    # tolerance (1e-12 of |b|) times the conditioning, carried through the steps.  Measured between the
    # FP64 and the mixed-precision solve from the same start: elevations 1e-12 to 9e-12 (largest value
    # 3e-11), nodal velocities after 30 steps 1e-11 to 3e-10 (2e-7), a stand-alone solve 5e-13 (1e-11).
    # Transport has no solve: differences are the rounding of FP64 sums of a few terms over a few steps.
    return {"forecast": {"rel": 2e-9, "max": 2e-6}, "step": {"rel": 2e-9, "max": 2e-6},
            "elevation": {"rel": 4e-11, "max": 4e-10}, "transport": {"rel": 1e-12, "max": 1e-10},
            "csr": {"rel": 1e-11, "max": 1e-10}, "noalloc": {"rel": 1e-11, "max": 1e-10}}[case["kind"]]


def exact(case, seed):
    """The stand-alone solves in plain torch: Jacobi-PCG in FP64 with restarts from the true residual
    until it no longer falls.  The other kinds have no value without the framework's own step."""
    if case["kind"] not in ("csr", "noalloc"):
        return None
    ptr, idx, val, rhs = _system(case["side"], int(seed) % (2 ** 31 - 1) + 1)
    n = rhs[0].numel()
    A = torch.sparse_csr_tensor(ptr.to(torch.int64), idx.to(torch.int64), val, size=(n, n))
    row = torch.repeat_interleave(torch.arange(n, device=val.device), (ptr[1:] - ptr[:-1]).to(torch.int64))
    inv = 1.0 / val[row == idx.to(torch.int64)]
    x, b = torch.zeros_like(rhs[0]), rhs[0]
    for _ in range(4):
        r = b - A @ x
        d, p, rz = torch.zeros_like(b), torch.zeros_like(b), None
        stop = 1e-20 * float(r @ r)
        for it in range(4000):
            z = inv * r
            new = r @ z
            p = z if rz is None else z + (new / rz) * p
            q = A @ p
            al = new / (p @ q)
            d, r, rz = d + al * p, r - al * q, new
            if it % 50 == 49 and float(r @ r) <= stop:
                break
        x = x + d
    return x
