"""The work that a user of the library has it do, one call pattern per case, for timing two builds side by side.

A case names an entry point ("op"), a mesh ("dim", "nx", "ny", "nz") and the options of the call.  Meshes come from
the library's own generators: the jittered two-layer plane (5 m deep) and the lognormal box (cells of 1 m) of its
configurations, at those sizes and others.  Every state is its own problem: mesh jitter, conductivities and vectors
follow from the seed.  All vectors are device tensors, as the calls take them.
"""
import math

import numpy as np
import torch

import fvmpor_b200 as fb

RTOL = ATOL = 1e-6


def listed():
    return [
        # One residual F(t, y, y') of the 81 x 41 plane, the smallest configured mesh: what an outside integrator
        # calls two to three times per step; a call is launches and latency.
        {"name": "residual_plane", "op": "residual", "dim": 2, "nx": 81, "ny": 41, "nz": 0},
        # The same on the 214,221-node box of the headline configuration.
        {"name": "residual_box", "op": "residual", "dim": 3, "nx": 100, "ny": 100, "nz": 20},
        # The start of a step (upwind directions frozen, then the first residual with them) on the 1,050,426-node
        # box, the largest configured mesh.
        {"name": "step_box1m", "op": "step", "dim": 3, "nx": 200, "ny": 200, "nz": 25},
        # One Jacobian-vector product by difference quotient, the call of a matrix-free Krylov solver.
        {"name": "jv_box", "op": "jv", "dim": 3, "nx": 100, "ny": 100, "nz": 20},
        # Preconditioner set-up and four applies in FP64 on a plane of an ensemble member's size (odd extents).
        {"name": "precond_plane_fp64", "op": "precond", "dim": 2, "nx": 151, "ny": 93, "nz": 0, "precision": 0,
         "applies": 4},
        # The same with the FP32 factor on the headline box, as the integration guide's bridge calls it.
        {"name": "precond_box_fp32", "op": "precond", "dim": 3, "nx": 100, "ny": 100, "nz": 20, "precision": 1,
         "applies": 4},
        # A whole adaptive run on the 81 x 41 plane (ten simulated minutes): many short steps, bound by latency.
        {"name": "integrate_plane", "op": "integrate", "dim": 2, "nx": 81, "ny": 41, "nz": 0, "precision": 1,
         "assembled": True, "krylov_dim": 30, "t_end": 600.0},
        # A whole adaptive run on the headline box with the headline options (two simulated days of the thirty).
        {"name": "integrate_box", "op": "integrate", "dim": 3, "nx": 100, "ny": 100, "nz": 20, "precision": 1,
         "assembled": True, "krylov_dim": 40, "t_end": 172800.0},
        # The plain FP64 Jacobian-free method on a box of 42,439 nodes, its steps given.
        {"name": "replay_box_fp64", "op": "replay", "dim": 3, "nx": 36, "ny": 36, "nz": 30, "precision": 0,
         "assembled": False, "krylov_dim": 40, "steps": 14},
        # The headline options on a box of 380,666 nodes, its steps given: between the two configured boxes.
        {"name": "replay_box_large", "op": "replay", "dim": 3, "nx": 120, "ny": 120, "nz": 25, "precision": 1,
         "assembled": True, "krylov_dim": 40, "steps": 7},
        # The learned iterate's network over every node of the headline box.
        {"name": "mlp_forward", "op": "mlp_forward", "rows": 214221},
        # One epoch of its training in mini-batches of 8,192 rows, as the benchmark trains it.
        {"name": "mlp_train", "op": "mlp_train", "rows": 65536, "batch": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """extents of a box of lo to hi nodes (spread over the logarithm)"""
    while True:
        n = _log_int(rng, lo, hi)
        nz = rng.randint(6, 30)
        side = math.sqrt(n / (nz + 1))
        nx = max(6, int(side * rng.uniform(0.75, 1.33)))
        ny = max(6, int(n / ((nz + 1) * (nx + 1))) - 1)
        if lo <= (nx + 1) * (ny + 1) * (nz + 1) <= hi:
            return {"dim": 3, "nx": nx, "ny": ny, "nz": nz}


def _plane(rng, lo, hi):
    n = _log_int(rng, lo, hi)
    nx = max(11, int(math.sqrt(2.0 * n) * rng.uniform(0.85, 1.2)))
    return {"dim": 2, "nx": nx, "ny": max(6, n // nx), "nz": 0}


def draw(rng):
    """One more case of the same ranges."""
    op = rng.choice(["residual", "residual", "step", "jv", "precond", "precond", "integrate", "replay", "replay",
                     "mlp_forward", "mlp_train"])
    if op in ("residual", "step", "jv"):
        return {"op": op, **(_plane(rng, 200, 40000) if rng.random() < 0.4 else _box(rng, 1000, 500000))}
    if op == "precond":
        mesh = _plane(rng, 200, 40000) if rng.random() < 0.5 else _box(rng, 1000, 214000)
        return {"op": op, **mesh, "precision": rng.randint(0, 1), "applies": rng.randint(1, 8)}
    if op == "integrate":
        return {"op": op, **_plane(rng, 200, 16000), "precision": 1, "assembled": True,
                "krylov_dim": rng.choice([20, 30, 40]), "t_end": float(rng.randint(60, 600))}
    if op == "replay":
        # the FP32 fused cycle takes boxes from 40,000 nodes on; above 237,000 the partition changes
        mesh = _box(rng, 40000, 212000) if rng.random() < 0.7 else _box(rng, 240000, 380000)
        fp32 = rng.random() < 0.7
        return {"op": op, **mesh, "precision": int(fp32), "assembled": fp32, "krylov_dim": rng.choice([20, 30, 40]),
                "steps": rng.randint(3, 9)}
    if op == "mlp_forward":
        return {"op": op, "rows": _log_int(rng, 200, 1000000)}
    rows = _log_int(rng, 1000, 130000)
    return {"op": op, "rows": rows, "batch": min(rows, rng.choice([2048, 4096, 8192, 37888]))}


# ------------------------------------------------------------------ states
def _problem(case, seed):
    if case["dim"] == 2:
        return fb.make_problem("richards2d", nx=case["nx"], ny=case["ny"], seed=seed % 100003 + 1)
    return fb.make_problem("richards3d", nx=case["nx"], ny=case["ny"], nz=case["nz"], Lx=float(case["nx"]),
                           Ly=float(case["ny"]), Lz=float(case["nz"]), seed=seed % 100003 + 1)


def _vectors(case, seed, problem):
    """Head near the hydrostatic one (the Dirichlet rows on their values up to the same noise), a slow time
    derivative, and the increment and shift of a mid-run step."""
    a = problem.arrays()
    z = a["coords"][:, 1 if case["dim"] == 2 else 2]
    rng = np.random.default_rng(seed)
    n = problem.n_nodes
    y = problem.water_table - z + 0.05 * rng.standard_normal(n)
    yp = 1e-7 * rng.standard_normal(n)
    ewt = 1.0 / (RTOL * np.abs(y) + ATOL)
    v = rng.standard_normal(n) / ewt
    return a, y, yp, ewt, v


CJ, STEP = 2e-3, 500.0


def _steps(count):
    """h grows from 600 s to a steady 4 h, orders 1 then 2"""
    s = np.zeros(count, dtype=[("h", "f8"), ("order", "i4")])
    for i in range(count):
        s["h"][i] = min(600.0 * 2.0 ** max(0, i - 1), 14400.0)
        s["order"][i] = min(i + 1, 2)
    return s


def _samples(case, seed):
    """Features and targets of the sizes that recorded trajectories have, and a fresh network's parameters."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    n = case["rows"]
    scale = torch.tensor([4.0, 0.02, 0.002, 0.8, 1.0, 5.0, 0.3, 0.0], device="cuda")
    shift = torch.tensor([-3.0, 0.001, 0.0, 3.5, -11.5, 10.0, 3.0, 0.0], device="cuda")
    u = torch.randn(n, 8, generator=g, device="cuda")
    y = torch.sin(u[:, 0]) + 0.5 * u[:, 1] * u[:, 2] - 0.3 * u[:, 4] + 0.1 * torch.randn(n, generator=g, device="cuda")
    return u * scale + shift, y.contiguous()


def prepare(case, seed):
    op = case["op"]
    s = {"case": case}
    if op.startswith("mlp"):
        s["problem"] = fb.make_problem("richards2d", nx=21, ny=11)
        s["physics"] = fb.Physics(s["problem"])
        s["X"], s["Y"] = _samples(case, seed)
        s["net"] = fb.Predictor(s["physics"])
        s["net"].init(s["X"], seed=seed % 100003)
        s["params"] = s["net"].get_params()
        s["out"] = torch.empty(case["rows"], dtype=torch.float32, device="cuda")
        return s
    p = s["problem"] = _problem(case, seed)
    ph = s["physics"] = fb.Physics(p)
    y = s["y"] = torch.empty(p.n_nodes, dtype=torch.float64, device="cuda")
    s["out"] = torch.empty_like(y)
    if op in ("integrate", "replay"):
        ph.initial_head(y)
        s["integrator"] = fb.Integrator(ph, rtol=RTOL, atol=ATOL, krylov_dim=case["krylov_dim"], max_restarts=5,
                                        precision=case["precision"], krylov_operator=int(case["assembled"]))
        if op == "replay":
            s["steps"] = _steps(case["steps"])
        return s
    _, yn, ypn, ewt, v = _vectors(case, seed, p)
    y.copy_(torch.from_numpy(yn))
    s["yp"] = torch.from_numpy(ypn).cuda()
    if op != "step":
        ph.begin_step(0.0, y, s["yp"])
    if op in ("jv", "precond"):
        s["v"] = torch.from_numpy(v).cuda()
        s["F0"] = torch.empty_like(y)
        ph.residual(0.0, y, s["yp"], s["F0"])
    if op == "precond":
        s["ewt"] = torch.from_numpy(ewt).cuda()
        s["r"] = [torch.from_numpy(np.random.default_rng((seed, k)).standard_normal(p.n_nodes)).cuda()
                  for k in range(case["applies"])]
        s["z"] = [torch.empty_like(y) for _ in s["r"]]
        s["precond"] = fb.Preconditioner(ph)
        # the pattern, once per mesh
        s["precond"].setup(0.0, CJ, STEP, y, s["yp"], s["F0"], s["ewt"], case["precision"])
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "mlp_forward":
        s["net"].forward(s["X"], s["out"])
        return s["out"]
    if op == "mlp_train":
        s["net"].set_params(s["params"])
        _, losses = s["net"].train(s["X"], s["Y"], epochs=1, batch=case["batch"], lr=2e-3)
        return s["net"].get_params(), losses
    ph, y, out = s["physics"], s["y"], s["out"]
    if op == "integrate":
        s["integrator"].integrate(0.0, case["t_end"], y, out)
        return out
    if op == "replay":
        s["integrator"].replay(0.0, y, float(s["steps"]["h"][0]), s["steps"], out, newton_tol=1e-5)
        return out
    if op == "residual":
        ph.residual(0.0, y, s["yp"], out)
        return out
    if op == "step":
        ph.begin_step(0.0, y, s["yp"])
        ph.residual(0.0, y, s["yp"], out)
        return out
    if op == "jv":
        ph.jv(0.0, CJ, y, s["yp"], s["F0"], s["v"], 1.0, out)
        return out
    s["precond"].setup(0.0, CJ, STEP, y, s["yp"], s["F0"], s["ewt"], case["precision"])
    for r, z in zip(s["r"], s["z"]):
        s["precond"].apply(r, z)
    return s["z"]


# ------------------------------------------------------------------ what a pass cannot do without
def _counts(case):
    d = case["dim"]
    if d == 2:
        n = case["nx"] * case["ny"]
        e, nnz = 2 * n, 7 * n
    else:
        n = (case["nx"] + 1) * (case["ny"] + 1) * (case["nz"] + 1)
        e, nnz = 6 * case["nx"] * case["ny"] * case["nz"], 15 * n
    return n, e, nnz


def work(case):
    """Bytes: vectors in and out, and per element its node ids, conductivity and upwind flags with the vertices once
    (for the factor and the assembled operator: values and columns once).  Flops: the face fluxes (about 120 per
    tetrahedron, 40 per triangle) and 100 per node for the soil functions."""
    op = case["op"]
    if op == "mlp_forward":
        return {"bytes": 36.0 * case["rows"], "flops": 2.0 * case["rows"] * (8 * 64 + 2 * 64 * 64 + 64)}
    if op == "mlp_train":
        return {"bytes": 36.0 * case["rows"], "flops": 6.0 * case["rows"] * (8 * 64 + 2 * 64 * 64 + 64)}
    n, e, nnz = _counts(case)
    mesh = (4.0 * (case["dim"] + 1) + 16) * e + 8.0 * case["dim"] * n
    flux = (120.0 if case["dim"] == 3 else 40.0) * e + 100.0 * n
    residual = {"bytes": mesh + 48.0 * n, "flops": flux}
    if op == "residual":
        return residual
    if op == "step":
        return {"bytes": 2 * mesh + 64.0 * n, "flops": 2 * flux}
    if op == "jv":
        return {"bytes": mesh + 64.0 * n, "flops": flux + 2.0 * n}
    value = 4 if case["precision"] else 8
    setup = {"bytes": mesh + 40.0 * n + (value + 2.0) * nnz, "flops": 4 * flux + 4.0 * nnz}
    apply = {"bytes": (value + 2.0) * nnz + 16.0 * n, "flops": 2.0 * nnz}
    if op == "precond":
        return {k: setup[k] + case["applies"] * apply[k] for k in setup}
    # per step: its start, two residuals, a set-up and four Krylov iterations
    steps = case["steps"] if op == "replay" else 46 if case["dim"] == 3 else 65
    krylov = {"bytes": 2 * apply["bytes"] + 8.0 * n * value, "flops": 2 * apply["flops"] + 16.0 * n}
    return {k: steps * (4 * residual[k] + setup[k] + 4 * krylov[k]) for k in setup}


# ------------------------------------------------------------------ the same results in 64-bit numpy
def _faces(dim):
    """(a, b, others) of an element's control-volume faces"""
    if dim == 2:
        return [(0, 1, (2,)), (1, 2, (0,)), (2, 0, (1,))]
    return [(0, 1, (2, 3)), (1, 2, (0, 3)), (2, 0, (1, 3)), (0, 3, (1, 2)), (1, 3, (0, 2)), (2, 3, (0, 1))]


class _Cvfe:
    """Median-dual control volumes of a simplex mesh, Richards' equation with frozen upwinding."""

    def __init__(self, problem, a):
        m, ph, d = problem.mesh, problem.phys, problem.mesh.dim
        self.d, self.en, self.zone = d, a["elem_nodes"].astype(np.int64), a["elem_zone"]
        self.zones = [ph.zones[i] for i in range(ph.n_zones)]
        bcs = {ph.bcs[i].tag: ph.bcs[i] for i in range(ph.n_bcs)}
        self.rho, n = ph.rho0, problem.n_nodes
        x = a["coords"][:, :d]
        X = x[self.en]
        jac = X[:, 1:] - X[:, :1]
        vol = np.abs(np.linalg.det(jac)) / math.factorial(d)
        inv = np.linalg.inv(jac)
        self.grad = np.concatenate([-inv.sum(axis=2, keepdims=True), inv], axis=2)
        K = np.array([[z.Kxx, z.Kyy, z.Kzz][:d] for z in self.zones])[self.zone]
        if "elem_K" in a:
            K = np.repeat(a["elem_K"][:, None], d, axis=1)
        self.KS, self.area = [], []
        for fa, fb_, rest in _faces(d):
            if d == 2:
                t = (2 * X[:, rest[0]] - X[:, fa] - X[:, fb_]) / 6
                S = np.stack([t[:, 1], -t[:, 0]], axis=1)
            else:
                S = np.cross(X[:, rest[0]] + X[:, rest[1]] - X[:, fa] - X[:, fb_], X[:, rest[1]] - X[:, rest[0]]) / 24
            S *= np.where((S * (X[:, fb_] - X[:, fa])).sum(1) < 0, -1.0, 1.0)[:, None]
            self.area.append(np.linalg.norm(S, axis=1))
            self.KS.append(K * S)
        share = np.repeat(vol[:, None] / (d + 1), d + 1, axis=1)
        self.V = np.bincount(self.en.ravel(), share.ravel(), n)
        self.w = [np.bincount(self.en[self.zone == z].ravel(), share[self.zone == z].ravel(), n) / self.V
                  for z in range(len(self.zones))]
        self.fixed, self.hD, self.inflow = np.zeros(n, bool), np.zeros(n), np.zeros(n)
        for i in np.flatnonzero(a["node_tag"]):
            bc = bcs[a["node_tag"][i]]
            if bc.type in (1, 4):
                self.fixed[i] = True
                self.hD[i] = bc.value if bc.type == 1 else (1 + bc.eta) * (bc.b - x[i, d - 1])
        for f, tag in zip(a["bface_nodes"], a["bface_tag"]):
            bc = bcs[tag]
            if bc.type == 3:
                e = [x[k] - x[f[0]] for k in f[1:]]
                size = np.linalg.norm(e[0]) if d == 2 else 0.5 * np.linalg.norm(np.cross(e[0], e[1]))
                self.inflow[f] -= self.rho * bc.value * size / d
        self.weight = np.full((len(_faces(d)), len(self.en)), 0.5)

    def soil(self, h):
        krw, phi, dsw = [], 0.0, 0.0
        for z, w in zip(self.zones, self.w):
            m = 1 - 1 / z.nVG
            dry = h < 0
            hn = np.where(dry, h, -1.0)
            a = (-z.alphaVG * hn) ** z.nVG
            Se = (1 + a) ** -m
            ab = a / (1 + a)
            krw.append(np.where(dry, np.sqrt(Se) * (ab ** m - 1) ** 2, 1.0))
            phi = phi + z.phi * w
            dsw = dsw + w * np.where(dry, -(1 - z.S_r) * (z.nVG - 1) * ab * Se / hn, 0.0)
        return krw, self.rho * phi * dsw

    def fluxes(self, h):
        g = np.einsum("edk,ek->ed", self.grad, h[self.en])
        g[:, self.d - 1] += 1.0
        return [-(ks * g).sum(1) for ks in self.KS]

    def mobility(self, krw):
        at = np.empty(self.en.shape)
        for z, k in enumerate(krw):
            at[self.zone == z] = k[self.en[self.zone == z]]
        return at

    def freeze(self, h):
        """upwind weight of each face's first node, from its edge's summed flux"""
        at, q = self.mobility(self.soil(h)[0]), self.fluxes(h)
        key, flow = [], []
        for (fa, fb_, _), qf in zip(_faces(self.d), q):
            i, j = self.en[:, fa], self.en[:, fb_]
            key.append(np.minimum(i, j) * len(self.V) + np.maximum(i, j))
            flow.append(np.where(i < j, 1.0, -1.0) * qf * 0.5 * (at[:, fa] + at[:, fb_]))
        _, edge = np.unique(np.concatenate(key), return_inverse=True)
        total = np.bincount(edge, np.concatenate(flow))[edge].reshape(len(q), -1)
        for f, (fa, fb_, _) in enumerate(_faces(self.d)):
            up = np.where(self.en[:, fa] < self.en[:, fb_], total[f], -total[f])
            self.weight[f] = np.where(up > 0, 1.0, 0.0)

    def residual(self, h, hp):
        krw, ahh = self.soil(h)
        at, acc = self.mobility(krw), self.inflow.copy()
        for (fa, fb_, _), qf, w in zip(_faces(self.d), self.fluxes(h), self.weight):
            f = self.rho * qf * (w * at[:, fa] + (1 - w) * at[:, fb_])
            acc += np.bincount(self.en[:, fb_], f, len(h)) - np.bincount(self.en[:, fa], f, len(h))
        return np.where(self.fixed, self.hD - h, acc / self.V - ahh * hp)


def _layers(P):
    P = torch.as_tensor(P, dtype=torch.float64)
    out, at = [], 0
    for rows, cols in ((64, 8), (64, 64), (64, 64), (1, 64)):
        out += [P[at:at + rows * cols].reshape(rows, cols).clone(), P[at + rows * cols:at + rows * cols + rows].clone()]
        at += rows * cols + rows
    return out, P[at:at + 8], P[at + 8:at + 16]


def _network(L, x):
    for k in range(3):
        x = torch.nn.functional.gelu(x @ L[2 * k].T + L[2 * k + 1])
    return (x @ L[6].T + L[7])[:, 0]


def exact(case, seed):
    op = case["op"]
    if op.startswith("mlp"):
        X, Y = (t.double().cpu() for t in _samples(case, seed))
        with torch.no_grad():
            # the same fresh network: weights normal(0, 1 / fan in), features scaled by their mean and deviation
            rng = np.random.default_rng(seed % 100003)
            parts = []
            for rows, cols in ((64, 8), (64, 64), (64, 64), (1, 64)):
                parts += [rng.normal(0, 1 / np.sqrt(cols), rows * cols), np.zeros(rows)]
            Xc = X.float()
            parts += [Xc.mean(0).double().numpy(), Xc.std(0).double().numpy() + 1e-6]
            P = np.concatenate(parts).astype(np.float32)
        L, mu, sd = _layers(P)
        X = (X - mu) / sd
        if op == "mlp_forward":
            with torch.no_grad():
                return _network(L, X)
        L = [t.requires_grad_() for t in L]
        opt = torch.optim.Adam(L, lr=2e-3, eps=1e-8)
        total = 0.0
        for at in range(0, len(X), case["batch"]):
            opt.zero_grad()
            x, y = X[at:at + case["batch"]], Y[at:at + case["batch"]]
            loss = ((_network(L, x) - y) ** 2).mean()
            loss.backward()
            opt.step()
            total += loss.item() * len(x)
        P = torch.cat([t.detach().reshape(-1) for t in L] + [mu, sd])
        return P.numpy(), np.array([total / len(X)])
    n, e, _ = _counts(case)
    if op not in ("residual", "step", "jv") or e > 1500000:
        return None   # no closed form, or too long in numpy
    problem = _problem(case, seed)
    a, y, yp, _, v = _vectors(case, seed, problem)
    c = _Cvfe(problem, a)
    c.freeze(y)
    if op != "jv":
        return c.residual(y, yp)
    return c.residual(y + v, yp + CJ * v) - c.residual(y, yp)
