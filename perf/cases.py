"""Measured workloads of the flux pass: what a program has it do, through the public entry
points, from the smallest mesh to the largest ones of the shipped workloads.

Every case loads an initial state from host memory, runs the pass for the stated number of
steps and reads the final state back, as a host code does between two snapshots (the mesh is
uploaded once, beforehand).  Sizes and step counts are those of ``workloads`` (Sod tube,
Sedov blast, random field, batch of step states, request stream) or odd ones of the same
ranges.  Small tessellations are made from the seed; large ones take the host builder
seconds, so they come from a pool with one mesh per shape, as the request stream's do, with
the states made from the seed.

Plain-FP64 results are returned as they come (float64).  The split pass keeps its cell states
in single precision and its results carry that accuracy, so a program keeps them in that
type; the totals of the conserved quantities, which it accumulates in FP64, stay float64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from shadowfax_b200 import _lib as L
from shadowfax_b200 import workloads as wl
from shadowfax_b200.hydro import Context, FluxPass, Group, RiemannSolverFactory
from shadowfax_b200.mesh import build_voronoi, random_generators
from shadowfax_b200.serve import Server

GAMMA = wl.GAMMA
# generators above which a mesh comes from the pool (about 0.1 s of tessellation)
POOL_FROM = {2: 50_000, 3: 4_000}
_pool: dict = {}


def listed():
    """kind run: one mesh, `steps` global steps; group: many meshes in one launch group;
    serve: a batch of requests through the request server; moving: one step of a moving mesh;
    local: system steps with per-cell (hierarchical) time steps.  split: the FP32/FP64 split
    pass, otherwise plain FP64."""
    return [
        # the shipped Sod tube: 10,000 cells, exact solver, 100 steps of 1e-4
        dict(name="sod2d_exact_fp64", kind="run", dim=2, n=10_000, field="sod", periodic=False,
             solver="Exact", split=False, steps=100),
        # the smallest mesh of the batch and of the stream: a kernel launch outweighs its work
        dict(name="step2d_small_hllc_split", kind="run", dim=2, n=1_000, field="step",
             periodic=False, solver="HLLC", split=True, steps=20),
        # the shipped Sedov blast: 64^3 cells, HLLC, 50 steps at CFL 0.4
        dict(name="sedov3d_hllc_split", kind="run", dim=3, n=262_144, field="sedov",
             periodic=False, solver="HLLC", split=True, steps=50),
        # the same blast in plain FP64, which a result is checked with
        dict(name="sedov3d_hllc_fp64", kind="run", dim=3, n=65_537, field="sedov",
             periodic=False, solver="HLLC", split=False, steps=20),
        # the supersonic random field, plain FP64 with the exact solver
        dict(name="random3d_exact_fp64", kind="run", dim=3, n=100_003, field="random",
             periodic=True, solver="Exact", split=False, steps=4),
        # the same field in the split pass: large request of the stream, 3D
        dict(name="random3d_exact_split", kind="run", dim=3, n=160_001, field="random",
             periodic=True, solver="Exact", split=True, steps=20),
        # large requests of the stream in 2D (70% of it), both solvers
        dict(name="random2d_exact_split", kind="run", dim=2, n=464_159, field="random",
             periodic=True, solver="Exact", split=True, steps=20),
        dict(name="random2d_hllc_fp64", kind="run", dim=2, n=150_001, field="random",
             periodic=True, solver="HLLC", split=False, steps=10),
        # the shipped batch (1,024 meshes of 1e3 to 1e5 cells), a slice of it
        dict(name="batch2d_hllc_group", kind="group", dim=2, count=64, lo=1_000, hi=50_000,
             solver="HLLC", steps=20),
        # a burst of requests, both dimensions and solvers, uneven sizes and step counts
        dict(name="serve_burst", kind="serve", requests=24, hi=40_000, lo_steps=10, hi_steps=60),
        # one step of a moving mesh (one per tessellation)
        dict(name="moving3d_hllc_split", kind="moving", dim=3, n=27_000, periodic=True,
             solver="HLLC", split=True),
        # local time steps
        dict(name="local2d_exact_fp64", kind="local", dim=2, n=20_011, solver="Exact",
             split=False, steps=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["group", "serve", "moving", "local"])
    dim = rng.choice([2, 3])
    solver = rng.choice(["Exact", "HLLC"])
    split = rng.random() < 0.5
    if kind == "group":
        return dict(kind=kind, dim=2, count=rng.randint(3, 48), lo=1_000,
                    hi=_log_int(rng, 2_000, 40_000), solver=solver, steps=rng.randint(5, 20))
    if kind == "serve":
        return dict(kind=kind, requests=rng.randint(4, 24), hi=_log_int(rng, 2_000, 40_000),
                    lo_steps=10, hi_steps=rng.randint(15, 60))
    if kind == "moving":
        k = round(_log_int(rng, 1_000, 27_000) ** (1 / dim))
        return dict(kind=kind, dim=dim, n=k**dim, periodic=rng.random() < 0.5, solver=solver,
                    split=split)
    if kind == "local":
        return dict(kind=kind, dim=dim, n=_log_int(rng, 900, 20_000 if dim == 2 else 8_000),
                    solver=solver, split=split, steps=rng.randint(2, 6))
    n = _log_int(rng, 700, 300_000 if dim == 2 else 60_000)
    field = rng.choice(["step", "random", "sod"] if dim == 2 else ["random", "sedov"])
    most = 4 if not split and solver == "Exact" else 20
    steps = rng.randint(1, most)
    return dict(kind=kind, dim=dim, n=n, field=field, periodic=field == "random", solver=solver,
                split=split, steps=steps)


# ------------------------------------------------------------------ inputs


def _mesh(dim, n, periodic, seed, lattice=False):
    """a tessellation of n generators: from the seed, or (large) the pool's mesh of the shape"""
    pooled = n > POOL_FROM[dim]
    key = (dim, n, periodic, lattice)
    if pooled and key in _pool:
        return _pool[key]
    s = 7_919 + n if pooled else seed
    if lattice:
        # lattice points moved by up to a quarter cell: generators of a moving mesh stay apart
        k = round(n ** (1 / dim))
        rng = np.random.Generator(np.random.PCG64(s))
        g = np.stack(np.meshgrid(*[np.arange(k)] * dim, indexing="ij"), -1).reshape(-1, dim)
        pos = np.ascontiguousarray((g + 0.5 + rng.uniform(-0.25, 0.25, g.shape)) / k)
    else:
        pos = random_generators(n, dim, s)
    mesh = build_voronoi(pos, periodic=periodic)
    if pooled:
        _pool[key] = mesh
    return mesh


def _state(field, mesh, seed):
    """initial primitive variables of one of the shipped workloads, varied by the seed, and
    the time step"""
    rng = np.random.Generator(np.random.PCG64(seed + 101))
    n, D, pos = mesh.n_cells, mesh.dim, mesh.cell_pos
    W = np.zeros((n, D + 2))
    if field == "random":
        W = wl.random_field_state(mesh, seed + 1000)
        # a quarter of the CFL step of the initial state: the supersonic field steepens in the
        # run, and a fixed step near the limit drives a few cells to negative energy
        return W, 0.25 * wl.cfl_dt(mesh, W)
    if field == "smooth":
        # subsonic waves, for the moving mesh and the local steps
        ph = rng.uniform(0, 2 * math.pi, 4)
        W[:, 0] = 1.0 + 0.3 * np.sin(2 * math.pi * pos[:, 0] + ph[0])
        for k in range(D):
            W[:, 1 + k] = 0.2 * np.sin(2 * math.pi * pos[:, (k + 1) % D] + ph[1 + k])
        W[:, D + 1] = 1.0 + 0.2 * np.cos(2 * math.pi * pos[:, D - 1] + ph[0])
        return W, wl.cfl_dt(mesh, W)
    if field == "sod":
        left = pos[:, 0] < rng.uniform(0.4, 0.6)
        W[:, 0] = np.where(left, rng.uniform(0.9, 1.1), 0.125)
        W[:, D + 1] = np.where(left, rng.uniform(0.9, 1.1), 0.1)
        return W, min(1e-4, wl.cfl_dt(mesh, W))
    if field == "sedov":
        W[:, 0] = 1.0
        W[:, D + 1] = 1e-6
        d2 = ((pos - rng.uniform(0.4, 0.6, D)) ** 2).sum(1)
        hot = np.argsort(d2, kind="stable")[:32]
        W[hot, D + 1] = (GAMMA - 1.0) * (1.0 / 32) / mesh.cell_volume[hot]
        return W, wl.cfl_dt(mesh, W)
    rhoL, pL, rhoR, pR = rng.uniform(0.1, 1.0, 4)
    th = rng.uniform(0.0, 2 * math.pi)
    side = (pos[:, :2] - 0.5) @ np.array([math.cos(th), math.sin(th)]) < 0
    W[:, 0] = np.where(side, rhoL, rhoR)
    W[:, D + 1] = np.where(side, pL, pR)
    return W, wl.cfl_dt(mesh, W)


def _problem(case, seed):
    """mesh, state and time step of a one-mesh case"""
    if case["kind"] == "run":
        mesh = _mesh(case["dim"], case["n"], case["periodic"], seed)
        return mesh, *_state(case["field"], mesh, seed)
    if case["kind"] == "moving":
        mesh = _mesh(case["dim"], case["n"], case["periodic"], seed, lattice=True)
        return mesh, *_state("smooth", mesh, seed)
    mesh = _mesh(case["dim"], case["n"], True, seed)
    return mesh, *_state("smooth", mesh, seed)


def _members(case, seed):
    """the meshes, states and time steps of a group case"""
    rng = np.random.Generator(np.random.PCG64(99 + case["count"] + case["hi"]))
    sizes = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"]))
    key = ("group", case["count"], case["lo"], case["hi"])
    if key not in _pool:
        _pool[key] = [build_voronoi(random_generators(int(n), 2, 31 * j + 4), periodic=False)
                      for j, n in enumerate(sizes)]
    return [(m, *_state("step", m, seed * 1000 + j)) for j, m in enumerate(_pool[key])]


def _requests(case, seed):
    """pool meshes (four sizes in each dimension) and the requests on them"""
    hi = case["hi"]
    sizes = [int(round(1_000 * (hi / 1_000) ** (k / 3))) for k in range(4)]
    meshes = [_mesh(2, n, True, 50 + n) for n in sizes]
    meshes += [_mesh(3, max(900, n // 2), True, 60 + n) for n in sizes]
    rng = np.random.Generator(np.random.PCG64(seed + 5))
    shape = np.random.Generator(np.random.PCG64(17))  # sizes and steps: the same for any seed
    reqs = []
    for k in range(case["requests"]):
        mid = int(shape.integers(4)) + (0 if shape.random() < 0.7 else 4)
        steps = int(shape.integers(case["lo_steps"], case["hi_steps"] + 1))
        solver = "Exact" if k % 2 else "HLLC"
        W, dt = _state("smooth", meshes[mid], int(rng.integers(1 << 30)))
        reqs.append((mid, W, solver, dt, steps))
    return meshes, reqs


# --------------------------------------------------------------- the calls


def _precision(case):
    return L.PREC_SPLIT if case["split"] else L.PREC_FP64


def prepare(case, seed):
    kind = case["kind"]
    if kind == "serve":
        meshes, reqs = _requests(case, seed)
        srv = Server(precision=L.PREC_SPLIT)
        for m in meshes:
            srv.add_mesh(m)
        return dict(kind=kind, server=srv, requests=reqs)
    if kind == "group":
        ctx = Context(2, RiemannSolverFactory.generate(case["solver"]), L.PREC_SPLIT)
        problems = _members(case, seed)
        members = [FluxPass(ctx, m) for m, _, _ in problems]
        group = Group(ctx, members, [dt for _, _, dt in problems])
        return dict(kind=kind, ctx=ctx, members=members, group=group,
                    W0=[W for _, W, _ in problems], steps=case["steps"])
    mesh, W0, dt = _problem(case, seed)
    ctx = Context(case["dim"], RiemannSolverFactory.generate(case["solver"]), _precision(case))
    return dict(kind=kind, ctx=ctx, fp=FluxPass(ctx, mesh), W0=W0, dt=dt,
                steps=case.get("steps", 1), split=case["split"],
                periodic=case.get("periodic", True))


def _kept(split, *arrays):
    """results as a program keeps them: single precision from the split pass"""
    return [torch.from_numpy(a).float() if split else a for a in arrays]


def run(state):
    kind = state["kind"]
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(*r) for r in state["requests"]]
        srv.drain()
        got = [srv.poll(i) for i in ids]
        W, Q = zip(*[_kept(True, r.W.ravel(), r.Q.ravel()) for r in got])
        return dict(W=torch.cat(W), Q=torch.cat(Q),
                    status=np.array([r.status for r in got]),
                    steps=np.array([r.steps_done for r in got]))
    if kind == "group":
        for fp, W0 in zip(state["members"], state["W0"]):
            fp.set_primitive(W0)
        status = state["group"].step(state["steps"], graph=True)
        W, Q = zip(*[_kept(True, *fp.state()) for fp in state["members"]])
        return dict(W=torch.cat(W), Q=torch.cat(Q), status=status)
    fp = state["fp"]
    fp.set_primitive(state["W0"])
    if kind == "moving":
        pos = fp.step_moving(state["dt"], state["periodic"])
        W, Q = _kept(state["split"], *fp.state())
        return dict(W=W, Q=Q, positions=_kept(state["split"], pos)[0])
    if kind == "local":
        zero = np.zeros(fp.mesh.n_cells, np.uint64)
        fp.set_timesteps(zero, zero)
        tick = fp.run_local(64 * state["dt"], state["steps"])
        W, Q = _kept(state["split"], *fp.state())
        return dict(W=W, Q=Q, tick=int(tick))
    st = fp.step(state["dt"], state["steps"])
    W, Q = _kept(state["split"], *fp.state())
    return dict(W=W, Q=Q, totals=np.array(st.totals[:fp.S]))


def work(case):
    """algorithmic bytes of the face steps of a pass (per face step 144 / 120 bytes in plain
    FP64 and 92 / 70 in the split pass, 2D / 3D) plus the states in and out; operations of
    the gradient, reconstruction and flux expressions (the exact solver's iteration on top)"""
    def part(dim, n, steps, split, solver):
        faces = n * (3.0 if dim == 2 else 7.77)
        per = {(2, False): 144, (3, False): 120, (2, True): 92, (3, True): 70}[(dim, split)]
        ops = 600 if solver == "HLLC" else 1_500
        return faces * steps * per + 3 * 8 * n * (dim + 2), faces * steps * ops
    if case["kind"] == "group":
        mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
        b, f = part(2, case["count"] * mean, case["steps"], True, case["solver"])
    elif case["kind"] == "serve":
        mean = sum(1_000 * (case["hi"] / 1_000) ** (k / 3) for k in range(4)) / 4
        steps = 0.5 * (case["lo_steps"] + case["hi_steps"])
        n = case["requests"] * mean
        b2, f2 = part(2, 0.7 * n, steps, True, "Exact")
        b3, f3 = part(3, 0.15 * n, steps, True, "Exact")
        b, f = b2 + b3, f2 + f3
    else:
        b, f = part(case["dim"], case["n"], case.get("steps", 1), case["split"], case["solver"])
    return {"bytes": b, "flops": f}


# ------------------------------------- the pass in 64 bits, in plain torch


def exact(case, seed):
    """static global steps by the torch restatement below; None for the moving mesh and the
    local steps"""
    if case["kind"] == "serve":
        meshes, reqs = _requests(case, seed)
        got = [_steps64(meshes[m], W, dt, s, steps) for m, W, s, dt, steps in reqs]
    elif case["kind"] == "group":
        got = [_steps64(m, W, dt, case["solver"], case["steps"])
               for m, W, dt in _members(case, seed)]
    elif case["kind"] == "run":
        mesh, W0, dt = _problem(case, seed)
        W, Q = _steps64(mesh, W0, dt, case["solver"], case["steps"])
        return dict(W=W, Q=Q, totals=Q.sum(0))
    else:
        return None
    cat = (lambda x: torch.cat([a.reshape(-1) for a in x])) if case["kind"] == "serve" else torch.cat
    return dict(W=cat([g[0] for g in got]), Q=cat([g[1] for g in got]), status=None, steps=None)


class _Mesh64:
    def __init__(self, m):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        on = m.face_area != 0
        self.x, self.cen, self.V = t(m.cell_pos), t(m.cell_centroid), t(m.cell_volume)
        self.tarea, self.A, self.mid = t(m.cell_total_area), t(m.face_area[on]), t(m.face_midpoint[on])
        self.xr, self.kind = t(m.face_right_pos[on]), t(m.face_kind[on])
        self.L = t(m.face_left[on].astype(np.int64))
        self.R = t(np.maximum(m.face_right[on], 0).astype(np.int64))
        self.mirror, self.real = self.kind == 2, self.kind == 0
        self.r = self.x[self.L] - self.xr
        self.rn = self.r.norm(dim=1)
        self.n = -self.r / self.rn[:, None]


def _get_W(Q, V):
    D = Q.shape[1] - 2
    W = torch.zeros_like(Q)
    ke = 0.5 * (Q[:, 1:D + 1] ** 2).sum(1) / Q[:, 0]
    W[:, 0] = Q[:, 0] / V
    W[:, 1:D + 1] = Q[:, 1:D + 1] / Q[:, :1]
    p = (GAMMA - 1) * (Q[:, D + 1] - ke) / V
    W[:, D + 1] = p.clamp(min=1e-30)
    Q[:, D + 1] = torch.where(p < 1e-30, ke + 1e-30 * V / (GAMMA - 1), Q[:, D + 1])
    return W


def _gradients(g, W):
    n, S = W.shape
    D = S - 2
    WL = W[g.L]
    Wj = W[g.R].clone()
    vn = (WL[:, 1:D + 1] * g.n).sum(1, keepdim=True)
    mir = WL.clone()
    mir[:, 1:D + 1] -= 2 * vn * g.n
    Wj[g.mirror] = mir[g.mirror]
    c = g.mid - 0.5 * (g.x[g.L] + g.xr)
    s = (g.A / g.rn)[:, None, None]
    t = s * ((Wj - WL)[:, None, :] * c[:, :, None] - 0.5 * (Wj + WL)[:, None, :] * g.r[:, :, None])
    delta = torch.zeros(n, D, S, dtype=W.dtype, device=W.device)
    delta.index_add_(0, g.L, t)
    delta.index_add_(0, g.R[g.real], -t[g.real])
    delta /= g.V[:, None, None]
    hi, lo = W.clone(), W.clone()
    idx = g.L[:, None].expand(-1, S)
    hi.scatter_reduce_(0, idx, Wj, "amax")
    lo.scatter_reduce_(0, idx, Wj, "amin")
    idx = g.R[g.real][:, None].expand(-1, S)
    hi.scatter_reduce_(0, idx, WL[g.real], "amax")
    lo.scatter_reduce_(0, idx, WL[g.real], "amin")
    alpha = torch.ones_like(W)
    for cell, sel in ((g.L, slice(None)), (g.R[g.real], g.real)):
        dp = (delta[cell] * (g.mid[sel] - g.cen[cell])[:, :, None]).sum(1)
        q = torch.where(dp > 0, hi[cell] - W[cell], lo[cell] - W[cell])
        q = torch.where(dp == 0, torch.ones_like(q), q / torch.where(dp == 0, torch.ones_like(dp), dp))
        alpha.scatter_reduce_(0, cell[:, None].expand(-1, S), q, "amin")
    return delta * alpha[:, None, :]


def _dWdt(W, G):
    S = W.shape[1]
    D = S - 2
    rho, p = W[:, 0], W[:, D + 1]
    div = sum(G[:, k, 1 + k] for k in range(D))
    d = torch.empty_like(W)
    adv = lambda q: sum(W[:, 1 + l] * G[:, l, q] for l in range(D))  # noqa: E731
    d[:, 0] = -rho * div - adv(0)
    for k in range(D):
        d[:, 1 + k] = -adv(1 + k) - G[:, k, D + 1] / rho
    if D == 2:  # the published scheme's 2D row takes d(vy)/dy in both terms
        d[:, 2] = -(W[:, 1] + W[:, 2]) * G[:, 1, 2] - G[:, 1, 3] / rho
    d[:, D + 1] = -GAMMA * p * div - adv(D + 1)
    return d


def _limit(mid, L_, R_, w):
    d1, d2 = 0.5 * (L_ - R_).abs(), 0.25 * (L_ - R_).abs()
    lo, hi = torch.minimum(L_, R_), torch.maximum(L_, R_)
    bar = L_ + w[:, None] * (R_ - L_)
    up = L_ < R_
    ext = torch.where(up, lo, hi)
    b = torch.where(up, ext - d1, ext + d1)
    b = torch.where(b * ext > 0, b, ext / (1 + d1 / ext.abs()))
    r = torch.where(up, torch.maximum(b, torch.minimum(bar + d2, mid)),
                    torch.minimum(b, torch.maximum(bar - d2, mid)))
    return torch.where(L_ == R_, L_, r)


def _predict(dt, Ws, Wo, G, d, has_other, dist):
    D = Ws.shape[1] - 2
    W = Ws + (G * d[:, :, None]).sum(1)
    lim = _limit(W, Ws, Wo, d.norm(dim=1) / torch.where(has_other, dist, torch.ones_like(dist)))
    W = torch.where(has_other[:, None], lim, W)
    neg = ((W[:, 0] < 0) | (W[:, D + 1] < 0))[:, None]
    W = torch.where(neg, Ws, W)
    N = W + 0.5 * dt * _dWdt(Ws, G)
    neg = ((N[:, 0] < 0) | (N[:, D + 1] < 0))[:, None]
    return torch.where(neg, W, N)


def _sample(rho, p, a, v, ps, us, zero):
    """state at x/t = 0 left of the contact moving at us >= 0 (mirrored by the caller for the
    right side): density, normal velocity and pressure"""
    g = GAMMA
    r = ps / p
    shock = ps > p
    S = v - a * (0.5 * (g + 1) / g * r + 0.5 * (g - 1) / g).sqrt()
    rs = rho * (r + (g - 1) / (g + 1)) / ((g - 1) / (g + 1) * r + 1)
    rr = rho * r ** (1 / g)
    head, tail = v - a, us - a * r ** (0.5 * (g - 1) / g)
    base = (2 / (g + 1) + (g - 1) / (g + 1) * v / a).clamp(min=0)
    out = []
    for star_s, star_r, fan, own in ((rs, rr, rho * base ** (2 / (g - 1)), rho),
                                     (us, us, 2 / (g + 1) * (a + 0.5 * (g - 1) * v), v),
                                     (ps, ps, p * base ** (2 * g / (g - 1)), p)):
        q = torch.where(shock, torch.where(S < 0, star_s, own),
                        torch.where(head < 0, torch.where(tail > 0, fan, star_r), own))
        # a vacuum state opens between the fans
        q = torch.where(zero, torch.where(head < 0, torch.where(v + 2 * a / (g - 1) > 0, fan, 0 * q), own), q)
        out.append(q)
    return out


def _exact_flux(WL, WR, n):
    """density, velocity and pressure of the exact solution at rest, its flux along n"""
    g, D = GAMMA, WL.shape[1] - 2
    rL, rR, pL, pR = WL[:, 0], WR[:, 0], WL[:, D + 1], WR[:, D + 1]
    vL, vR = (WL[:, 1:D + 1] * n).sum(1), (WR[:, 1:D + 1] * n).sum(1)
    aL, aR = (g * pL / rL).sqrt(), (g * pR / rR).sqrt()
    vac = 2 * (aL + aR) / (g - 1) <= vR - vL

    def side(p, rho, pk, a):
        w = (2 / (g + 1) / rho / (p + (g - 1) / (g + 1) * pk)).sqrt()
        z = (p / pk) ** (0.5 * (g - 1) / g)
        s = p > pk
        f = torch.where(s, (p - pk) * w, 2 * a / (g - 1) * (z - 1))
        d = torch.where(s, (1 - 0.5 * (p - pk) / (p + (g - 1) / (g + 1) * pk)) * w,
                        z * pk / (p * rho * a))
        return f, d
    e = 0.5 * (g - 1) / g
    # two-rarefaction pressure: never below the root's left Newton start after one step
    num = (aL + aR - 0.5 * (g - 1) * (vR - vL)).clamp(min=1e-300)
    p = (num / (aL / pL ** e + aR / pR ** e)) ** (1 / e)
    p = torch.where(vac, pL, p)
    lo, hi = torch.zeros_like(p), torch.full_like(p, math.inf)
    for _ in range(60):
        fL, dL = side(p, rL, pL, aL)
        fR, dR = side(p, rR, pR, aR)
        f = fL + fR + vR - vL
        lo, hi = torch.where(f < 0, p, lo), torch.where(f > 0, p, hi)
        q = p - f / (dL + dR)
        p = torch.where((q > lo) & (q < hi), q,
                        torch.where(q >= hi, 0.5 * (lo + hi), torch.where(f == 0, p, 0.5 * (lo + p))))
        p = torch.where(vac, pL, p)
    fL, _ = side(p, rL, pL, aL)
    fR, _ = side(p, rR, pR, aR)
    us = 0.5 * (vL + vR) + 0.5 * (fR - fL)
    sl = _sample(rL, pL, aL, vL, p, us, vac)
    sr = _sample(rR, pR, aR, -vR, p, -us, vac)
    SR, SL = vR - 2 * aR / (g - 1), vL + 2 * aL / (g - 1)
    left = torch.where(vac, SL >= 0, us >= 0)
    rho, pr = torch.where(left, sl[0], sr[0]), torch.where(left, sl[2], sr[2])
    un = torch.where(left, sl[1], -sr[1])
    empty = vac & (SR > 0) & (SL < 0)
    rho, pr = torch.where(empty, 0 * rho, rho), torch.where(empty, 0 * pr, pr)
    Wk, vk = torch.where(left[:, None], WL, WR), torch.where(left, vL, vR)
    v = Wk[:, 1:D + 1] + (un - vk)[:, None] * n
    F = torch.empty_like(WL)
    F[:, 0] = rho * un
    F[:, 1:D + 1] = (rho * un)[:, None] * v + pr[:, None] * n
    F[:, D + 1] = (0.5 * rho * (v**2).sum(1) + g / (g - 1) * pr) * un
    return F, vac


def _hllc_flux(WL, WR, n):
    g, D = GAMMA, WL.shape[1] - 2
    rL, rR, pL, pR = WL[:, 0], WR[:, 0], WL[:, D + 1], WR[:, D + 1]
    uL, uR = (WL[:, 1:D + 1] * n).sum(1), (WR[:, 1:D + 1] * n).sum(1)
    aL, aR = (g * pL / rL).sqrt(), (g * pR / rR).sqrt()
    ps = (0.5 * (pL + pR) - 0.125 * (uR - uL) * (rL + rR) * (aL + aR)).clamp(min=0)
    q = lambda a, p, r: torch.where(ps > p, (g * (p + 0.5 * (g + 1) / g * (ps - p)) / r).sqrt(), a)  # noqa: E731
    SL, SR = uL - q(aL, pL, rL), uR + q(aR, pR, rR)
    Ss = (pR - pL + rL * uL * (SL - uL) - rR * uR * (SR - uR)) / (rL * (SL - uL) - rR * (SR - uR))
    left = Ss >= 0
    W = torch.where(left[:, None], WL, WR)
    u, Sk = torch.where(left, uL, uR), torch.where(left, SL, SR)
    rho, p = W[:, 0], W[:, D + 1]
    e = p / (g - 1) / rho + 0.5 * (W[:, 1:D + 1] ** 2).sum(1)
    F = torch.empty_like(W)
    F[:, 0] = rho * u
    F[:, 1:D + 1] = (rho * u)[:, None] * W[:, 1:D + 1] + p[:, None] * n
    F[:, D + 1] = (rho * e + p) * u
    star = torch.where(left, SL < 0, SR > 0)
    fac = rho * (Sk - u) / (Sk - Ss)
    U = torch.empty_like(W)
    U[:, 0] = fac
    U[:, 1:D + 1] = fac[:, None] * (W[:, 1:D + 1] + (Ss - u)[:, None] * n)
    U[:, D + 1] = fac * (e + (Ss - u) * (Ss + p / (rho * (Sk - u))))
    C = torch.cat([rho[:, None], rho[:, None] * W[:, 1:D + 1], (rho * e)[:, None]], 1)
    F = torch.where(star[:, None], F + Sk[:, None] * (U - C), F)
    vac = 2 * (aL + aR) / (g - 1) <= uR - uL
    if bool(vac.any()):
        F[vac] = _exact_flux(WL[vac], WR[vac], n[vac])[0]
    return F


def _steps64(mesh, W0, dt, solver, steps):
    g = _Mesh64(mesh)
    W = torch.from_numpy(W0).to(g.x.device)
    D = W.shape[1] - 2
    V = g.V[:, None]
    Q = torch.cat([W[:, :1] * V, W[:, :1] * V * W[:, 1:D + 1],
                   (0.5 * W[:, :1] * (W[:, 1:D + 1] ** 2).sum(1, keepdim=True)
                    + W[:, D + 1:] / (GAMMA - 1)) * V], 1)
    other = ~g.mirror
    for _ in range(steps):
        G = _gradients(g, W)
        WL, WR = W[g.L], W[g.R]
        dist = (g.cen[g.L] - g.cen[g.R]).norm(dim=1)
        PL = _predict(dt, WL, WR, G[g.L], g.mid - g.cen[g.L], other, dist)
        PR = _predict(dt, WR, WL, G[g.R], g.mid - g.cen[g.R] + g.x[g.R] - g.xr, other, dist)
        vn = (PL[:, 1:D + 1] * g.n).sum(1, keepdim=True)
        mir = PL.clone()
        mir[:, 1:D + 1] -= 2 * vn * g.n
        PR = torch.where(g.mirror[:, None], mir, PR)
        F = _exact_flux(PL, PR, g.n)[0] if solver == "Exact" else _hllc_flux(PL, PR, g.n)
        dQ = dt * g.A[:, None] * F
        # over-flux limiter: no cell loses more than the face's share of its mass
        cap = g.A / g.tarea[g.L] * Q[g.L, 0]
        dQ = torch.where((dQ[:, 0] > cap)[:, None], dQ * (cap / dQ[:, 0]).abs()[:, None], dQ)
        cap = g.A / g.tarea[g.R] * Q[g.R, 0]
        over = other & (-dQ[:, 0] > cap)
        dQ = torch.where(over[:, None], dQ * (cap / dQ[:, 0]).abs()[:, None], dQ)
        Q.index_add_(0, g.L, -dQ)
        Q.index_add_(0, g.R[g.real], dQ[g.real])
        W = _get_W(Q, g.V)
    return W, Q
