"""The work a user of this framework has it do, as cases to measure.

Each case is one of the framework's public calls (or the few calls that a
program makes together) on a seeded synthetic mesh:

  run       the adaptive BDF2 time loop from rest (``FetdGPU.run``), one or many sources;
  solve     triangular solves with a factor in hand (``FetdGPU.solve``);
  pardiso   factor + solve of a host CSR matrix through the PARDISO-shaped calls;
  refresh   new conductivities: media, assembly, factorisation, one solve (the
            inner step of an inversion or of a finite-difference gradient);
  spmv      the sparse product the Fortran driver asks for each step;
  adjoint   a recorded forward run and the gradient of its dB/dt misfit;
  batch     several layered models stepped together (``FetdBatch.run``).

Meshes: "halfspace" (circular loop, one receiver), "block" (a conductor under
a square loop, a line of receivers), "multiloop" (a grid of small loops, one
column each), "layered".  The conductivity of the earth is log-normal per tet
around the model's value, drawn from the seed; air stays at 1e-12 S/m, which
is what makes the systems ill-conditioned and the path FP64 throughout.
"""
import functools
import math

import numpy as np
import torch

from temf3dt_b200 import fetd, inversion, meshio, synth

MU0 = 4.0e-7 * math.pi
PAIRS = ((0, 1), (0, 2), (0, 3), (1, 2), (3, 1), (2, 3))  # local edge -> local vertices
GATES = np.logspace(-6, -5, 8)
DENSE = 30000  # unknowns up to which exact() factors dense matrices

SMALL = dict(radius=200.0, half=20000.0, z_core=100.0)  # the short-offset half-space of the smallest meshes


# --- the cases ---------------------------------------------------------------
def listed():
    return [
        # one solve on the smallest mesh in use: launches and host calls are what it costs
        dict(name="solve-7k", kind="solve", mesh="halfspace", small=True, h=200.0, hz=100.0, ratio=5.0, cols=1, dt=1e-7),
        # a block of sources that does not fill the 64 columns
        dict(name="solve-39k-13col", kind="solve", mesh="halfspace", small=False, h=250.0, hz=50.0, ratio=2.5, cols=13, dt=4e-7),
        # the Fortran driver's mkl_sparse_d_mv replacement
        dict(name="spmv-150k", kind="spmv", mesh="halfspace", small=False, h=125.0, hz=25.0, ratio=2.0, cols=1, which=0),
        # the drop-in PARDISO module: a dt-doubling point of the reference's own loop
        dict(name="pardiso-27k", kind="pardiso", mesh="halfspace", small=True, h=170.0, hz=75.0, ratio=2.6, cols=1, dt=2e-7),
        # one conductivity update of an inversion on a mid-size block model
        dict(name="refresh-301k", kind="refresh", mesh="block", h=125.0, hz=62.5, ratio=1.6, cols=1, dt=1.6e-6),
        # a forward run at the size of the reference's smallest shipped example
        dict(name="run-27k", kind="run", mesh="halfspace", small=True, h=170.0, hz=75.0, ratio=2.6, cols=1, steps=64, double=20),
        # the plain half-space workload: a hundred steps and a doubling trial
        dict(name="run-150k", kind="run", mesh="halfspace", small=False, h=125.0, hz=25.0, ratio=2.0, cols=1, steps=110, double=100),
        # the large 3-D block model with its line of 64 receivers
        dict(name="run-1.48M", kind="run", mesh="block", shared=True, h=44.0, hz=22.0, ratio=1.5, cols=1, steps=60, double=60),
        # few transmitter positions at once, a ragged block
        dict(name="run-120k-9col", kind="run", mesh="multiloop", loops=3, h=80.0, hz=40.0, ratio=2.4, cols=9, steps=24, double=20),
        # a full block of 64 transmitter positions
        dict(name="run-250k-64col", kind="run", mesh="multiloop", loops=8, h=60.0, hz=30.0, ratio=2.4, cols=64, steps=14, double=12),
        # one gradient of an inversion step
        dict(name="adjoint-27k", kind="adjoint", mesh="halfspace", small=True, h=170.0, hz=75.0, ratio=2.6, cols=1, steps=36, double=30, every=10),
        # layered models of uneven size stepped together
        dict(name="batch-5", kind="batch", mesh="layered", scales="0.12,0.2,0.15,0.3,0.1", hz=20.0, ratio=3.0, cols=1, steps=24, double=20),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    def single():  # a mesh with one source: 7k to about 400k edges
        if rng.random() < 0.35:
            return dict(mesh="halfspace", small=True, h=round(log(90.0, 260.0), 2), hz=round(log(40.0, 110.0), 2),
                        ratio=round(rng.uniform(1.9, 5.0), 3))
        if rng.random() < 0.6:
            return dict(mesh="halfspace", small=False, h=round(log(95.0, 500.0), 2), hz=round(log(20.0, 100.0), 2),
                        ratio=round(rng.uniform(1.8, 2.6), 3))
        return dict(mesh="block", h=round(log(100.0, 300.0), 2), hz=round(log(50.0, 150.0), 2),
                    ratio=round(rng.uniform(1.6, 2.4), 3))

    kind = rng.choice(("run", "run", "run", "runs", "runs", "solve", "solve", "refresh", "refresh", "pardiso", "spmv",
                       "adjoint", "batch"))
    if kind == "run":
        return dict(kind="run", **single(), cols=1, steps=rng.randint(15, 130), double=rng.choice((12, 20, 50, 100)))
    if kind == "runs":
        loops = rng.randint(2, 8)
        return dict(kind="run", mesh="multiloop", loops=loops, h=round(log(55.0, 140.0), 2), hz=round(log(30.0, 70.0), 2),
                    ratio=round(rng.uniform(2.0, 3.0), 3), cols=rng.randint(2, loops * loops), steps=rng.randint(8, 16),
                    double=rng.choice((6, 10, 20)))
    if kind == "solve":
        return dict(kind="solve", **single(), cols=rng.choice((1, 1, 2, 5, 16, 33, 70)), dt=1e-7 * 2 ** rng.randint(0, 9))
    if kind == "refresh":
        return dict(kind="refresh", **single(), cols=1, dt=1e-7 * 2 ** rng.randint(0, 9))
    if kind == "pardiso":
        return dict(kind="pardiso", mesh="halfspace", small=True, h=round(log(90.0, 260.0), 2),
                    hz=round(log(40.0, 110.0), 2), ratio=round(rng.uniform(1.9, 5.0), 3), cols=1,
                    dt=1e-7 * 2 ** rng.randint(0, 9))
    if kind == "spmv":
        return dict(kind="spmv", **single(), cols=rng.choice((1, 1, 3, 16)), which=rng.randint(0, 1))
    if kind == "adjoint":
        return dict(kind="adjoint", mesh="halfspace", small=True, h=round(log(90.0, 260.0), 2),
                    hz=round(log(40.0, 110.0), 2), ratio=round(rng.uniform(1.9, 5.0), 3), cols=1,
                    steps=rng.randint(15, 45), double=rng.choice((12, 20, 30)), every=rng.randint(5, 30))
    scales = ",".join("%.3f" % log(0.08, 0.35) for _ in range(rng.randint(2, 7)))
    return dict(kind="batch", mesh="layered", scales=scales, hz=round(rng.uniform(14.0, 30.0), 2),
                ratio=round(rng.uniform(2.2, 3.5), 3), cols=1, steps=rng.randint(10, 30), double=rng.choice((12, 20)))


# --- models --------------------------------------------------------------------
class Model:
    """A synthetic model's arrays: mesh, topology, media per tet, sources, receivers."""

    def __init__(self, m):
        self.m, self.ctl = m, m.ctl
        self.nod, self.tet = m.mesh.nod_cor, m.mesh.tet_vex
        self.edg, self.te, self.td = fetd.mesh_topology(self.tet)
        self.sig, self.mu = meshio.media_per_tet(m.mesh.tet_phy, m.ctl)
        self.sources = m.source_columns(self.edg)
        self.n = len(self.edg)

    def media(self, seed):
        rng = np.random.default_rng([seed, self.n])
        s = self.sig * 10.0 ** (0.1 * rng.standard_normal(len(self.sig)))
        return np.where(self.sig > 1e-6, s, self.sig)

    def columns(self, cols):
        return self.sources[:cols]

    def receivers(self, cols):
        keep = self.m.rec_rhs < cols
        return self.m.receivers[keep], self.m.rec_rhs[keep]

    def smooth(self, cols, seed):
        """Tangential edge values (n, cols) of smooth azimuthal fields around seeded centres."""
        rng = np.random.default_rng([seed, self.n, 7])
        p, q = self.nod[self.edg[:, 0] - 1], self.nod[self.edg[:, 1] - 1]
        mid, t = 0.5 * (p + q), (q - p) / np.linalg.norm(q - p, axis=1)[:, None]
        out = np.empty((self.n, cols))
        for k in range(cols):
            c = np.append(rng.uniform(-100.0, 100.0, 2), 0.0)
            size = 10.0 ** rng.uniform(2.3, 3.2)
            d = (mid - c) / size
            out[:, k] = 1e-5 * rng.uniform(0.5, 2.0) * np.exp(-(d * d).sum(axis=1)) * (d[:, 0] * t[:, 1] - d[:, 1] * t[:, 0])
        return out


@functools.lru_cache(maxsize=8)
def _synth(mesh, key):
    kw = dict(key)
    return Model(synth.build_model(mesh, **kw))


def models(case):
    """The case's models (one, or several for a batch)."""
    if case["mesh"] == "layered":
        return [_synth("layered", tuple(sorted(dict(seed=100 + i, scale=float(s), h_z=case["hz"], ratio=case["ratio"]).items())))
                for i, s in enumerate(case["scales"].split(","))]
    kw = dict(seed=0, h_core=case["h"], h_z=case["hz"], ratio=case["ratio"])
    if case.get("small"):
        kw.update(SMALL)
    if case["mesh"] == "multiloop":
        kw.update(n_loops=case["loops"])
    if case.get("shared"):
        kw.update(shared_grid=True)
    return [_synth(case["mesh"], tuple(sorted(kw.items())))]


def load(M, cols, seed):
    """A context with the model loaded, as a driver sets it up."""
    gpu = fetd.FetdGPU(0)
    gpu.set_mesh(M.nod, M.tet, M.edg, M.te, M.td)
    gpu.set_media(M.media(seed), M.mu)
    gpu.set_boundary(0)
    gpu.analyse()
    gpu.assemble()
    gpu.set_sources(M.columns(cols), 1, 1, M.ctl.t0, 1.0)
    rec, rhs = M.receivers(cols)
    gpu.set_receivers(gpu.locate(rec, M.ctl.rec_charac), rec, rhs)
    return gpu


def schedule(case):
    return dict(sp_division=10, sp_double=case["double"], sp_dblesize=2, time_maximum=1e-2, max_steps=case["steps"])


def right_hand_sides(M, cols, dt, seed):
    """b = M_sigma w - 2 dt s of a step in the middle of a run."""
    b = element_product(M, M.media(seed), 0, M.smooth(cols, seed))
    for k in range(cols):
        e, d = M.sources[k % len(M.sources)]
        b[e - 1, k] -= 2.0 * dt * 1e3 * d * _geometry(M)["elen"][e - 1]
    return b[:, 0].copy() if cols == 1 else b


def observed(M, cols, seed):
    """Observed dB/dt at the gates: a power-law decay with log-normal noise."""
    rng = np.random.default_rng([seed, 11])
    nrec = len(M.receivers(cols)[0])
    return 1e-5 * (GATES[:, None] / 1e-6) ** -1.5 * 10.0 ** (0.1 * rng.standard_normal((len(GATES), nrec)))


def cells(M):
    grid = inversion.InversionGrid((8, 8, 4), ((-300.0, 300.0), (-300.0, 300.0), (0.0, 200.0)))
    cell = grid.tet_cells(M.nod, M.tet)
    return np.where(M.sig > 1e-6, cell, -1), grid.ncell


# --- what is measured -------------------------------------------------------------
def prepare(case, seed):
    kind, cols = case["kind"], case["cols"]
    many = models(case)
    M = many[0]
    if kind == "batch":
        gpus = [load(m, 1, seed + i) for i, m in enumerate(many)]
        return dict(kind=kind, gpus=gpus, batch=fetd.FetdBatch(gpus), args=schedule(case))
    gpu = load(M, min(cols, len(M.sources)), seed)
    s = dict(kind=kind, gpu=gpu)
    if kind in ("run", "adjoint"):
        s["args"] = schedule(case)
    if kind == "adjoint":
        gpu.adjoint_record(case["every"])
        s["cell"], s["ncell"] = cells(M)
        s["d_obs"] = observed(M, cols, seed)
    if kind == "spmv":
        s["which"] = case["which"]
        s["x"] = M.smooth(cols, seed)
        s["x"] = s["x"][:, 0].copy() if cols == 1 else s["x"]
    if kind in ("solve", "refresh", "pardiso"):
        s["b"], s["dt"] = right_hand_sides(M, cols, case["dt"], seed), case["dt"]
    if kind == "solve":
        gpu.factor(1, case["dt"])
    if kind == "refresh":
        s["sig"], s["mu"] = M.media(seed + 1000), M.mu
        s["b"] = right_hand_sides(M, cols, case["dt"], seed + 1000)
    if kind == "pardiso":
        gpu.pardiso_alloc(2)
        s["csr"] = upper_csr(M, M.media(seed), case["dt"])
    return s


def _rows(o):
    # the trials' error estimates are left to their decisions: each is one number, the difference
    # of two nearly equal vectors whose air entries are rounding
    return dict(steps=o.steps, times=o.times, dts=o.dts, fields=o.fields, accepted=o.trial_accepted)


def run(s):
    kind = s["kind"]
    if kind == "batch":
        return [_rows(o) for o in s["batch"].run(**s["args"])]
    gpu = s["gpu"]
    if kind == "run":
        return _rows(gpu.run(**s["args"]))
    if kind == "solve":
        return gpu.solve(1, s["b"])
    if kind == "spmv":
        return gpu.spmv(s["which"], s["x"])
    if kind == "pardiso":
        gpu.pardiso_direct_1(1, *s["csr"])
        return gpu.pardiso_direct_2(1, s["b"])
    if kind == "refresh":
        gpu.set_media(s["sig"], s["mu"])
        gpu.assemble()
        gpu.factor(1, s["dt"])
        return gpu.solve(1, s["b"])
    o = gpu.run(**s["args"])
    J, dJ = inversion.dbdt_misfit(o.fields, o.times, GATES, s["d_obs"])
    cell, tet, _ = gpu.adjoint(dJ, s["cell"], s["ncell"])
    return dict(_rows(o), misfit=J, cell=cell, tet=tet)


def work(case):
    """Bytes and FP64 operations of one pass.  The factor's size and operations follow
    n^(4/3) and n^2 on these meshes under nested dissection (7.3 n^(4/3) nonzeros of L and
    3.4 n^2 operations per factorisation within 10 % from 0.15M to 5M unknowns)."""
    total = {"bytes": 0.0, "flops": 0.0}
    for M in models(case):
        n, cols, nnz = M.n, case["cols"], 16.4 * M.n
        L = 7.3 * n ** (4.0 / 3.0)
        factor = (8.0 * (2 * nnz + L), 3.4 * n * n)
        solve = (16.0 * L + 16.0 * n * cols, 4.0 * L * cols)
        spmv = (12.0 * nnz + 16.0 * n * cols, 2.0 * nnz * cols)
        T = len(M.tet)
        if case["kind"] in ("run", "batch", "adjoint"):
            trials = case["steps"] // case["double"]
            solves = case["steps"] + 2 * trials
            parts = [(factor, 1 + trials), (solve, solves), (spmv, solves)]
            if case["kind"] == "adjoint":  # states recomputed, then one solve, product and tet gather per node
                parts += [(factor, 1 + trials), (solve, 2 * solves), (spmv, 2 * solves), ((8.0 * (21 + 24) * T, 150.0 * T), solves)]
        else:
            parts = {"solve": [(solve, 1)], "spmv": [(spmv, 1)], "pardiso": [(factor, 1), (solve, 1)],
                     "refresh": [((16.0 * T + 16.0 * nnz, 600.0 * T), 1), (factor, 1), (solve, 1)]}[case["kind"]]
        for (b, f), k in parts:
            total["bytes"] += b * k
            total["flops"] += f * k
    return total


# --- the same in plain numpy and torch, 64 bits ---------------------------------------
@functools.lru_cache(maxsize=4)
def _geometry(M):
    """Unit element matrices (T, 6, 6) with orientation signs, edge lengths, simplex gradients."""
    edges = np.asarray(M.edg, dtype=np.int64)
    elen = np.linalg.norm(M.nod[edges[:, 1] - 1] - M.nod[edges[:, 0] - 1], axis=1)
    X = M.nod[np.asarray(M.tet) - 1]
    T = len(X)
    B = np.concatenate([np.ones((T, 1, 4)), X.transpose(0, 2, 1)], axis=1)   # lambda = B^-1 (1, x, y, z)
    inv = np.linalg.inv(B)
    grad, vol = inv[:, :, 1:], np.abs(np.linalg.det(B)) / 6.0
    P, Q = [p for p, _ in PAIRS], [q for _, q in PAIRS]
    ln = np.linalg.norm(X[:, Q] - X[:, P], axis=2)
    lo = np.minimum(M.tet[:, P], M.tet[:, Q]).astype(np.int64)
    hi = np.maximum(M.tet[:, P], M.tet[:, Q]).astype(np.int64)
    big = int(M.tet.max()) + 1
    key = edges[:, 0] * big + edges[:, 1]
    te = np.searchsorted(key, lo * big + hi)
    sgn = np.where(M.tet[:, P] < M.tet[:, Q], 1.0, -1.0)
    w = ln * sgn
    gram = np.einsum("tka,tla->tkl", grad, grad)
    K = 2.0 * np.cross(grad[:, P], grad[:, Q])
    curl = np.einsum("tia,tja->tij", K, K) * vol[:, None, None]
    mass = np.empty((T, 6, 6))
    for i, (pi, qi) in enumerate(PAIRS):
        for j, (pj, qj) in enumerate(PAIRS):
            mass[:, i, j] = ((1 + (pi == pj)) * gram[:, qi, qj] - (1 + (pi == qj)) * gram[:, qi, pj]
                             - (1 + (qi == pj)) * gram[:, pi, qj] + (1 + (qi == qj)) * gram[:, pi, pj]) * vol / 20.0
    ww = w[:, :, None] * w[:, None, :]
    return dict(elen=elen, te=te, mass=mass * ww, curl=curl * ww, inv=inv, w=w, vol=vol)


def element_product(M, sig, which, x):
    """(M_sigma or K) x, summed element by element."""
    G = _geometry(M)
    E = G["mass"] * sig[:, None, None] if which == 0 else G["curl"] / M.mu[:, None, None]
    x = x.reshape(M.n, -1)
    y = np.empty_like(x)
    for k in range(x.shape[1]):
        v = np.einsum("tij,tj->ti", E, x[G["te"], k])
        y[:, k] = np.bincount(G["te"].ravel(), weights=v.ravel(), minlength=M.n)
    return y


def upper_csr(M, sig, dt):
    """1-based upper CSR of 3 M_sigma + 2 dt K (order, row pointers, columns, values)."""
    G = _geometry(M)
    E = 3.0 * G["mass"] * sig[:, None, None] + 2.0 * dt * G["curl"] / M.mu[:, None, None]
    i, j = np.broadcast_to(G["te"][:, :, None], E.shape), np.broadcast_to(G["te"][:, None, :], E.shape)
    up = i <= j
    key, where = np.unique(i[up] * M.n + j[up], return_inverse=True)
    va = np.bincount(where, weights=E[up])
    ia = np.concatenate([[0], np.cumsum(np.bincount(key // M.n, minlength=M.n))]) + 1
    return ia.astype(np.int32), (key % M.n + 1).astype(np.int32), va


class Dense:
    """Dense matrices of a small model on the GPU, in plain torch."""

    def __init__(self, M, sig):
        G = _geometry(M)
        te = torch.as_tensor(G["te"], device="cuda")
        at = (te[:, :, None] * M.n + te[:, None, :]).reshape(-1)

        def full(E):
            A = torch.zeros(M.n * M.n, dtype=torch.float64, device="cuda")
            return A.index_add_(0, at, torch.as_tensor(E.reshape(-1), device="cuda")).view(M.n, M.n)

        self.M = full(G["mass"] * sig[:, None, None])
        self.K = full(G["curl"] / M.mu[:, None, None])
        self.dt, self.L = None, None

    def solve(self, dt, b):
        if self.dt != dt:
            self.dt, self.L = dt, None
            A = 3.0 * self.M + 2.0 * dt * self.K
            self.L = torch.linalg.cholesky(A)
        b = torch.as_tensor(b, device="cuda").reshape(len(self.M), -1)
        return torch.cholesky_solve(b, self.L)


def pulse(t, t0):
    return 5.0 / (math.sqrt(math.pi) * t0) * math.exp(-25.0 * ((t - 0.5 * t0) / t0) ** 2)


def march(M, sig, case, seed):
    """The adaptive loop (fine pair against one coarse step at every doubling point) with dense matrices."""
    G, cols = _geometry(M), min(case["cols"], len(M.sources))
    D = Dense(M, sig)
    S = torch.zeros(M.n, cols, dtype=torch.float64, device="cuda")
    for k, (e, d) in enumerate(M.columns(cols)):
        S[torch.as_tensor(e.astype(np.int64) - 1, device="cuda"), k] = torch.as_tensor(d * G["elen"][e - 1], device="cuda")
    rec, rhs = M.receivers(cols)
    pos = np.concatenate([np.ones((len(rec), 1)), rec], axis=1)
    W, at = [], []
    for p in pos:
        lam = G["inv"] @ p
        t = int(np.argmax(lam.min(axis=1)))
        g, lam = G["inv"][t][:, 1:], lam[t]
        P, Q = [a for a, _ in PAIRS], [b for _, b in PAIRS]
        w = G["w"][t][:, None]
        W.append(np.concatenate([w * (lam[P, None] * g[Q] - lam[Q, None] * g[P]), -2.0 * w * np.cross(g[P], g[Q])], axis=1))
        at.append(G["te"][t])
    W, at, rhs = np.array(W), torch.as_tensor(np.array(at), device="cuda"), torch.as_tensor(rhs.astype(np.int64), device="cuda")
    div, double, t0 = 10, case["double"], M.ctl.t0
    dt, time, step, kept = t0 / div, 0.0, 0, 0
    nodes = [dict(x=torch.zeros_like(S))]  # the solves in order: state, dt, source factor, the two states it reads
    out = dict(steps=[], times=[], dts=[], node=[], accepted=[])

    def solve(step, time, dt, a, b):
        c = 2.0 * dt * pulse(time, t0) if step < div else 0.0
        x = D.solve(dt, D.M @ (4.0 * nodes[a]["x"] - nodes[b]["x"]) - c * S)
        nodes.append(dict(x=x, dt=dt, a=a, b=b))
        return len(nodes) - 1

    def row(step, time, dt, k):
        for name, v in (("steps", step), ("times", time), ("dts", dt), ("node", k)):
            out[name].append(v)

    row(0, 0.0, dt, 0)
    e2 = e3 = 0
    past = []
    while step < case["steps"]:
        step, time = step + 1, time + dt
        if step % double:
            e2, e3 = solve(step, time, dt, e2, e3), e2
            past.append(e2)
            row(step, time, dt, e2)
            continue
        f1 = solve(step, time, dt, e2, e3)
        f2 = solve(step, time + dt, dt, f1, e2)
        c = solve(step, time + dt, 2 * dt, past[-1], past[-3])
        d, f = nodes[c]["x"] - nodes[f2]["x"], nodes[f2]["x"]
        error = float((d.norm(dim=0) / f.norm(dim=0)).max())
        ok = not (error > 1e-4 and kept < 2)
        out["accepted"].append(ok)
        if ok:
            time, dt, kept, e2, e3 = time + dt, 2 * dt, 0, f2, past[-1]
        else:
            kept, e2, e3 = kept + 1, f1, e2
        past = []
        row(step, time, dt, e2)
    e = np.array([nodes[k]["x"][at, rhs[:, None]].cpu().numpy() for k in out["node"]])   # rows x receivers x 6
    f = np.einsum("rjc,irj->irc", W, e)
    f[np.array(out["steps"]) == 0, :, 3:] = 0.0
    b = np.cumsum(f[:, :, 3:] * np.array(out["dts"])[:, None, None], axis=0)
    got = dict(steps=np.array(out["steps"], dtype=np.int32), times=np.array(out["times"]), dts=np.array(out["dts"]),
               fields=np.concatenate([f, b], axis=2), accepted=np.array(out["accepted"], dtype=bool))
    return got, dict(nodes=nodes, row_node=out["node"], D=D, W=W, at=at, G=G)


def gradient(M, sig, got, g, d_obs):
    """The misfit of dBz/dt at the gates and its gradient, by the adjoint recursion on the solves."""
    times, rows = got["times"], len(got["times"])
    Wg = np.zeros((len(GATES), rows))
    for k, t in enumerate(GATES):
        i = int(np.searchsorted(times, t))
        if i >= rows:
            continue
        i = max(i, 1)
        s = (t - times[i - 1]) / (times[i] - times[i - 1])
        Wg[k, i - 1], Wg[k, i] = 1.0 - s, s
    res = Wg @ got["fields"][:, :, 5] - d_obs
    dJ = Wg.T @ res
    dJ[got["steps"] == 0] = 0.0
    nodes, D, G = g["nodes"], g["D"], g["G"]
    push = [torch.zeros_like(nodes[0]["x"]) for _ in nodes]
    for i, k in enumerate(g["row_node"]):
        v = torch.as_tensor(dJ[i][:, None] * g["W"][:, :, 5], device="cuda")
        push[k][:, 0].index_add_(0, g["at"].reshape(-1), -v.reshape(-1))
    te = torch.as_tensor(G["te"], device="cuda")
    mass = torch.as_tensor(G["mass"], device="cuda")
    tet = torch.zeros(len(G["te"]), dtype=torch.float64, device="cuda")
    for k in range(len(nodes) - 1, 0, -1):
        v = nodes[k]
        lam = D.solve(v["dt"], push[k])
        m = D.M @ lam
        push[v["a"]] += 4.0 * m
        push[v["b"]] -= m
        w = 3.0 * v["x"] - 4.0 * nodes[v["a"]]["x"] + nodes[v["b"]]["x"]
        tet += torch.einsum("ti,tij,tj->t", lam[te, 0], mass, w[te, 0])
    tet = tet.cpu().numpy()
    cell, ncell = cells(M)
    by = np.bincount(cell[cell >= 0], weights=(sig * tet)[cell >= 0], minlength=ncell)
    return dict(misfit=0.5 * float((res * res).sum()), cell=by, tet=tet)


def exact(case, seed):
    many = models(case)
    M, kind = many[0], case["kind"]
    if kind == "spmv":
        y = element_product(M, M.media(seed), case["which"], M.smooth(case["cols"], seed))
        return y[:, 0] if case["cols"] == 1 else y
    if kind == "batch":
        got = [march(m, m.media(seed + i), case, seed)[0] if m.n <= DENSE else None for i, m in enumerate(many)]
        return got if any(g is not None for g in got) else None
    if M.n > DENSE:
        return None
    if kind in ("run", "adjoint"):
        sig = M.media(seed)
        got, graph = march(M, sig, case, seed)
        return dict(got, **gradient(M, sig, got, graph, observed(M, 1, seed))) if kind == "adjoint" else got
    at = seed + 1000 if kind == "refresh" else seed
    b = right_hand_sides(M, case["cols"], case["dt"], at)
    x = Dense(M, M.media(at)).solve(case["dt"], b).cpu().numpy()
    return x[:, 0] if case["cols"] == 1 else x
