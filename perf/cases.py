"""Work that a user of the framework has it do, as cases that can be timed.

Five kinds, over grids of 642 to 163842 nodes and stencils of 17 to 101 nodes
(the grid and stencil sizes of the benchmark's cosine bell, heat, tracer,
weight and serving workloads, and sizes between and beside them):

  deriv    one derivative of a field: RBFFD.applyWeightsForDeriv on host arrays or
           applyWeightsForDerivDev on device buffers, 1 to 16 tracers
  advance  a time-dependent PDE from its initial values to its solution: heat, the cosine
           bell or advection in a vortex flow; set the state, RK4 steps, read the state
  weights  the weights of all stencils of a grid, read back or applied once
  knn      the nearest-neighbour stencils of a node set, searched on the device
  serve    a batch of requests through the serving loop, submitted together

Nodes are Fibonacci points under a seeded rotation and stencils their exact
nearest neighbours; shape parameters, polynomial degrees, hyperviscosity and
time steps follow the benchmark's, scaled with the node distance.
"""
import math

import numpy as np
import torch

import rbffd_gpu_b200 as R
from rbffd_gpu_b200.api import RHS_ADVECTION

_CTX = []


def _ctx():
    """The one context of this program."""
    if not _CTX:
        _CTX.append(R.Context(0))
    return _CTX[0]


def listed():
    return [
        # one derivative of one field on the cosine-bell grid, buffers on the device: a call's latency
        dict(name="deriv_bell", kind="deriv", N=4096, n=31, T=1, dtype="f64", host=False, op="lambda"),
        # the reference's own signature: host arrays in and out, on a serving-size grid
        dict(name="deriv_host", kind="deriv", N=40962, n=50, T=1, dtype="f64", host=True, op="lsfc"),
        # one operator over 16 tracers, the benchmark's tracer count and stencil, FP32
        dict(name="deriv_tracers", kind="deriv", N=163842, n=101, T=16, dtype="f32", host=False, op="theta"),
        # the reference's experiment: the cosine bell on 4096 nodes, three operators, FP64
        dict(name="bell", kind="advance", pde="bell", N=4096, n=31, T=1, dtype="f64", steps=200, graph=True, fused=False),
        # the headline: heat in FP64 on 163842 nodes, captured steps
        dict(name="heat_f64", kind="advance", pde="heat", N=163842, n=50, T=1, dtype="f64", steps=200, graph=True,
             fused=False),
        # heat in FP32 with default arguments (steps not captured) and odd sizes
        dict(name="heat_f32_odd", kind="advance", pde="heat", N=40003, n=37, T=1, dtype="f32", steps=100, graph=False,
             fused=False),
        # 16 tracers in a steady vortex flow, FP32, the fused operator
        dict(name="tracers_f32", kind="advance", pde="vortex", N=163842, n=101, T=16, dtype="f32", steps=60, graph=True,
             fused=True),
        # 4 tracers in FP64 with the reference's three operators
        dict(name="tracers_f64", kind="advance", pde="vortex", N=40962, n=50, T=4, dtype="f64", steps=25, graph=True,
             fused=False),
        # the experiment's weights: LAMBDA, THETA and HV, the reference's constant basis, read back
        dict(name="weights_bell", kind="weights", N=4096, n=31, mixed=False, deg=0, ops="advect", back=True),
        # the benchmark's batched weights: stencils of 17 to 101 nodes, degrees 1 to 4, applied once
        dict(name="weights_mix", kind="weights", N=100000, n=101, mixed=True, deg=1, ops="sfc", back=False),
        # stencil generation ahead of the headline grid
        dict(name="knn", kind="knn", N=163842, n=50),
        # requests of several grids, right-hand sides and types, batched by the serving loop
        dict(name="serve", kind="serve", N=40962, n=50, requests=24, steps=40),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["deriv", "deriv", "advance", "advance", "advance", "weights", "weights", "knn", "serve"])
    n = rng.randint(17, 101)
    if kind == "deriv":
        T = rng.choice([1, 1, 2, 3, 4, 5, 8, 16])
        host = T == 1 and rng.random() < 0.4
        return dict(kind=kind, N=_log_int(rng, 642, 163842), n=n, T=T, dtype=rng.choice(["f32", "f64"]), host=host,
                    op=rng.choice(["lsfc", "lambda", "theta", "hv"]))
    if kind == "advance":
        pde = rng.choice(["bell", "heat", "heat", "vortex"])
        T = 1 if pde == "bell" else rng.choice([1, 1, 2, 4, 7, 16])
        dtype = rng.choice(["f32", "f64"])
        fused = pde != "heat" and rng.random() < 0.4
        return dict(kind=kind, pde=pde, N=_log_int(rng, 642, 163842 if T == 1 else 40962), n=n, T=T, dtype=dtype,
                    steps=rng.randint(5, 60 if T == 1 else 20), graph=rng.random() < 0.7, fused=fused)
    if kind == "weights":
        mixed = rng.random() < 0.4
        return dict(kind=kind, N=_log_int(rng, 642, 30000), n=101 if mixed else n, mixed=mixed,
                    deg=1 if mixed else rng.choice([0, 2, 3] if n >= 25 else [0, 2]),
                    ops=rng.choice(["advect", "sfc", "heat"]), back=rng.random() < 0.3)
    if kind == "knn":
        return dict(kind=kind, N=_log_int(rng, 642, 163842), n=n)
    return dict(kind=kind, N=_log_int(rng, 1000, 40962), n=rng.randint(25, 50), requests=rng.randint(4, 24),
                steps=rng.randint(10, 40))


# ---------------------------------------------------------------------------
# inputs

def nodes(N, seed):
    """Fibonacci points on the unit sphere (z falling with the index), and the
    same points under a seeded rotation, as every program here uses them."""
    k = np.arange(N) + 0.5
    z = 1.0 - 2.0 * k / N
    lam = math.pi * (1.0 + math.sqrt(5.0)) * k
    rho = np.sqrt(1.0 - z * z)
    base = np.stack([rho * np.cos(lam), rho * np.sin(lam), z], axis=1)
    q, _ = np.linalg.qr(np.random.default_rng([7, seed]).standard_normal((3, 3)))
    return np.ascontiguousarray(base @ q.T)


def neighbours(xyz, n):
    """The n nearest nodes of every node, itself first.  A node's neighbours
    within distance r lie within r N / 2 of its index along the spiral."""
    N = len(xyz)
    x = torch.from_numpy(xyz).cuda()
    half = int(1.5 * math.sqrt(n * N)) + 16
    width = min(N, 2 * half + 1)
    out = torch.empty((N, n), dtype=torch.int32, device="cuda")
    rows = max(1, int(1.2e7) // width)
    for a in range(0, N, rows):
        i = torch.arange(a, min(N, a + rows), device="cuda")
        j = (i - half).clamp(0, N - width)[:, None] + torch.arange(width, device="cuda")[None, :]
        d2 = torch.zeros(j.shape, dtype=torch.float64, device="cuda")
        for c in range(3):
            d2 += (x[:, c][j] - x[i, c][:, None]) ** 2
        d2[torch.arange(len(i), device="cuda"), i - j[:, 0]] = -1.0  # the centre first
        k = torch.topk(d2, n, dim=1, largest=False, sorted=True).indices
        out[i] = torch.gather(j, 1, k).to(torch.int32)
    return out.cpu().numpy()


def spacing(N):
    return math.sqrt(4.0 * math.pi / N)


def smooth_field(xyz, T, seed):
    """T smooth fields: cubics in the coordinates, seeded coefficients."""
    rng = np.random.default_rng([11, seed])
    x, y, z = xyz.T
    basis = np.stack([np.ones_like(x), x, y, z, x * y, y * z, x * z, x * x - y * y, x * y * z, z ** 3], axis=1)
    u = basis @ rng.standard_normal((basis.shape[1], T))
    return np.ascontiguousarray(u if T > 1 else u[:, 0])


def vortex_flow(xyz, seed):
    """Velocity components (east, north) of a vortex turning about a seeded axis."""
    p = np.random.default_rng([13, seed]).standard_normal(3)
    p /= np.linalg.norm(p)
    s = np.clip(xyz @ p, -1.0, 1.0)
    rho = 3.0 * np.sqrt(1.0 - s * s) + 1e-12
    omega = 1.5 * math.sqrt(3.0) * np.tanh(rho) / np.cosh(rho) ** 2 / rho
    v = omega[:, None] * np.cross(p[None, :], xyz)
    lam, th = np.arctan2(xyz[:, 1], xyz[:, 0]), np.arctan2(xyz[:, 2], np.hypot(xyz[:, 0], xyz[:, 1]))
    east = np.stack([-np.sin(lam), np.cos(lam), 0 * lam], axis=1)
    north = np.stack([-np.sin(th) * np.cos(lam), -np.sin(th) * np.sin(lam), np.cos(th)], axis=1)
    return np.ascontiguousarray((v * east).sum(1)), np.ascontiguousarray((v * north).sum(1))


OPS = {"lsfc": R.LSFC, "lambda": R.LAMBDA, "theta": R.THETA, "hv": R.HV, "xsfc": R.XSFC, "ysfc": R.YSFC, "zsfc": R.ZSFC}
OP_SETS = {"advect": ("hv", "lambda", "theta"), "sfc": ("xsfc", "ysfc", "zsfc"), "heat": ("lsfc",)}
MIX = ((17, 1), (31, 2), (50, 3), (101, 4))  # stencil size and polynomial degree
HV_K, HV_GAMMA = 4, 1e-3
DTYPES = {"f32": (R.F32, torch.float32, np.float32), "f64": (R.F64, torch.float64, np.float64)}
REVOLUTION = 1036800.0  # seconds, the cosine bell's


def shape_parameter(n, op_set, N):
    return (0.25 if op_set == "heat" and n >= 25 else 0.4) / spacing(N)


def degree(n, op_set):
    return 2 if n < 25 or op_set == "advect" else 3


class Problem:
    """A grid with its stencils and the settings of its weights."""

    def __init__(self, case, seed, op_set, deg, mixed=False):
        N, n = case["N"], case["n"]
        self.xyz = nodes(N, seed)
        self.st = neighbours(self.xyz, n)
        self.ops = OP_SETS[op_set]
        self.deg, self.lens, self.degs = deg, None, None
        self.eps = np.full(N, shape_parameter(n, op_set, N))
        if mixed:
            rng = np.random.default_rng([17, seed])
            pick = rng.integers(0, len(MIX), N)
            self.lens = np.array([m[0] for m in MIX], dtype=np.int32)[pick]
            self.degs = np.array([m[1] for m in MIX], dtype=np.int32)[pick]
            self.eps = rng.uniform(0.35, 0.6, N) / spacing(N)

    def library(self):
        """The same as the framework's grid and operator objects."""
        self.grid = R.Grid(_ctx(), self.xyz, self.st, st_len=self.lens)
        types = 0
        for o in self.ops:
            types |= OPS[o]
        self.der = R.RBFFD(types, self.grid, 2)
        self.der.setEpsilon(self.eps)
        self.der.setHVScalars(HV_K, HV_GAMMA)
        self.der.setPolynomialDegree(self.deg, self.degs)
        return self


def op_set_of(op):
    return next(k for k, v in OP_SETS.items() if op in v)


def time_step(case):
    """Stable steps: the benchmark's, scaled with the node distance."""
    N = case["N"]
    if case["pde"] == "heat":
        return 0.05 / N
    if case["pde"] == "bell":
        return REVOLUTION / 1000.0 * math.sqrt(4096.0 / N)
    return 0.3 * spacing(N)


class State:
    """What one case has in hand; its handles end with it."""

    def __init__(self, case, seed):
        self.case, self.kind = case, case["kind"]
        self.pde = self.srv = None
        self.problems = []

    def __del__(self):
        try:
            if self.srv is not None:
                self.srv.stop()
            if self.pde is not None:
                self.pde.close()
            for p in self.problems:
                p.grid.close()
        except Exception:
            pass


def requests_of(case, seed):
    """The batch's requests: (problem 0 heat or 1 advection, FP type, steps, initial values' seed)."""
    rng = np.random.default_rng([19, case["requests"]])
    return [(int(rng.integers(0, 2)), "f64" if rng.random() < 0.25 else "f32",
             int(rng.integers(max(1, case["steps"] // 2), case["steps"] + 1)), 1000 * seed + k)
            for k in range(case["requests"])]


def serve_problems(case, seed):
    small = dict(N=max(642, case["N"] // 4), n=31)
    return [Problem(case, seed, "heat", degree(case["n"], "heat")), Problem(small, seed + 1, "advect", 2)]


def prepare(case, seed):
    S = State(case, seed)
    kind = S.kind
    if kind == "knn":
        # scattered nodes: every one moved by a seeded fraction of the node distance
        x = nodes(case["N"], seed)
        x += 0.15 * spacing(len(x)) * np.random.default_rng([23, seed]).standard_normal(x.shape)
        S.xyz = x / np.linalg.norm(x, axis=1)[:, None]
        _ctx()
        return S
    if kind == "weights":
        P = Problem(case, seed, case["ops"], case["deg"], case["mixed"]).library()
        S.problems.append(P)
        S.u = torch.from_numpy(smooth_field(P.xyz, 1, seed)).cuda()
        S.out = [torch.empty_like(S.u) for _ in P.ops]
        return S
    if kind == "deriv":
        op_set = op_set_of(case["op"])
        P = Problem(case, seed, op_set, degree(case["n"], op_set)).library()
        S.problems.append(P)
        P.der.computeAllWeightsForAllStencils()
        u = smooth_field(P.xyz, case["T"], seed)
        if case["host"]:
            S.u = u
        else:
            S.u = torch.from_numpy(u).to("cuda", DTYPES[case["dtype"]][1])
            S.out = torch.empty_like(S.u)
        return S
    if kind == "advance":
        op_set = "heat" if case["pde"] == "heat" else "advect"
        P = Problem(case, seed, op_set, degree(case["n"], op_set)).library()
        S.problems.append(P)
        P.der.computeAllWeightsForAllStencils()
        kw = dict(dtype=DTYPES[case["dtype"]][0], ntracers=case["T"])
        if case["pde"] == "heat":
            S.pde = R.HeatSphere(P.grid, P.der, 1.0, **kw)
        elif case["pde"] == "bell":
            S.pde = R.CosineBell(P.grid, P.der, 1.0, math.pi / 2, REVOLUTION, True, **kw)
        else:
            S.pde = R.Advection(P.grid, P.der, *vortex_flow(P.xyz, seed), True, **kw)
        if case["fused"]:
            S.pde.setFusedOperator(True)
        S.u = smooth_field(P.xyz, case["T"], seed)
        S.dt = time_step(case)
        return S
    S.problems = [p.library() for p in serve_problems(case, seed)]
    for p in S.problems:
        p.der.computeAllWeightsForAllStencils()
    S.srv = R.Server(_ctx())
    S.flow = vortex_flow(S.problems[1].xyz, seed)
    S.requests = []
    for which, dtype, steps, s in requests_of(case, seed):
        P, dt = S.problems[which], DTYPES[dtype][0]
        N = len(P.xyz)
        if which == 0:
            S.requests.append((P, R.heat_params(1.0, dt), smooth_field(P.xyz, 1, s), 0.05 / N, steps, None, dtype))
        else:
            prm = R.heat_params(1.0, dt)
            prm.rhs_kind, prm.use_hv = RHS_ADVECTION, 1
            S.requests.append((P, prm, smooth_field(P.xyz, 1, s), 0.3 * spacing(N), steps, S.flow, dtype))
    return S


def run(S):
    case = S.case
    if S.kind == "knn":
        return R.knn_stencils_gpu(_ctx(), S.xyz, case["n"])
    if S.kind == "weights":
        P = S.problems[0]
        P.der.computeAllWeightsForAllStencils()
        if case["back"]:
            return [P.der.getWeights(OPS[o]) for o in P.ops]
        for o, out in zip(P.ops, S.out):
            P.der.applyWeightsForDerivDev(OPS[o], S.u.data_ptr(), out.data_ptr())
        return S.out
    if S.kind == "deriv":
        der, op, dt = S.problems[0].der, OPS[case["op"]], DTYPES[case["dtype"]]
        if case["host"]:
            # an FP32 derivative comes back in doubles: returned as the FP32 values it holds
            d = der.applyWeightsForDeriv(op, S.u, dtype=dt[0])
            return d if case["dtype"] == "f64" else d.astype(dt[2])
        der.applyWeightsForDerivDev(op, S.u.data_ptr(), S.out.data_ptr(), dtype=dt[0], ntracers=case["T"])
        return S.out
    if S.kind == "advance":
        S.pde.fillInitialConditions(S.u)
        S.pde.advance(R.RK4, S.dt, case["steps"], graph=case["graph"])
        u = S.pde.getLocalSolution()
        return u if case["dtype"] == "f64" else u.astype(np.float32)
    ids = [S.srv.submit(P.grid, prm, u0, dt, steps, *(flow or ())) for P, prm, u0, dt, steps, flow, _ in S.requests]
    S.srv.wait_idle()
    return [S.srv.result(i).astype(DTYPES[q[6]][2]) for i, q in zip(ids, S.requests)]


def work(case):
    """Each stencil index, weight, coordinate and value once; 2 flops per multiply-add."""
    N, n, kind = case["N"], case["n"], case["kind"]
    w = 4 if case.get("dtype") == "f32" else 8
    if kind == "knn":
        return {"bytes": N * (24 + 4 * n), "flops": 8 * N * n}
    if kind == "weights":
        K = len(OP_SETS[case["ops"]])
        sizes = MIX if case["mixed"] else ((n, case["deg"]),)
        flops = bytes_ = 0.0
        for s, d in sizes:
            m = s + {0: 1, 1: 4}.get(d, (d + 1) * (d + 2) // 2)
            flops += N / len(sizes) * (2 * m ** 3 / 3 + m * m / 2 + 2 * K * m * m)
            bytes_ += N / len(sizes) * s * (4 + 8 * K)
        return {"bytes": bytes_ + 32 * N, "flops": flops}
    if kind == "deriv":
        return {"bytes": N * n * (4 + w) + 2 * N * case["T"] * (8 if case["host"] else w), "flops": 2 * N * n * case["T"]}
    if kind == "advance":
        K = 1 if case["pde"] == "heat" or case["fused"] else 3
        T = case["T"]
        return {"bytes": N * n * (4 + K * w) + 2 * N * T * 8, "flops": case["steps"] * 4 * T * N * (2 * n * K + 8)}
    q, small = case["requests"], max(642, N // 4)
    return {"bytes": N * n * 8 + small * 31 * 16 + q * 8 * (N + small),
            "flops": q * 0.75 * case["steps"] * 4 * (N * 2 * n + small * 2 * 31 * 3) / 2}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits

def _poly_terms(deg):
    return [(t - b, b) for t in range(deg + 1) for b in range(t + 1)]


def _weights_of(xyz, st, eps, deg, ops):
    """Weights [rows][n] of each operator for stencils of one size and degree:
    Gaussian RBF systems with a polynomial border (none but a constant for
    degree 0, {1, x, y, z} for degree 1, scaled tangent-plane polynomials above)."""
    rows, n = st.shape
    N = len(xyz)
    x = xyz[st.long()]
    c = x[:, 0]
    e2 = (eps * eps)[:, None]
    r2 = ((x[:, :, None, :] - x[:, None, :, :]) ** 2).sum(-1)
    terms = 4 if deg == 1 else len(_poly_terms(deg))
    m = n + terms
    A = torch.zeros((rows, m, m), dtype=torch.float64, device=xyz.device)
    A[:, :n, :n] = torch.exp(-r2 * e2[:, :, None])
    del r2
    lam, th = torch.atan2(c[:, 1], c[:, 0])[:, None], torch.atan2(c[:, 2], torch.hypot(c[:, 0], c[:, 1]))[:, None]
    zero = torch.zeros_like(lam[:, 0])
    east = torch.stack([-torch.sin(lam[:, 0]), torch.cos(lam[:, 0]), zero], dim=1)
    north = torch.stack([-torch.sin(th) * torch.cos(lam), -torch.sin(th) * torch.sin(lam), torch.cos(th)], dim=1)[:, :, 0]
    d = x - c[:, None, :]
    s = torch.sqrt((d * d).sum(-1).amax(1))[:, None]
    if deg == 1:
        A[:, :n, n] = 1.0
        A[:, :n, n + 1:] = x
    else:
        xi, eta = (d * east[:, None]).sum(-1) / s, (d * north[:, None]).sum(-1) / s
        for q, (a, b) in enumerate(_poly_terms(deg)):
            A[:, :n, n + q] = xi ** a * eta ** b
    A[:, n:, :n] = A[:, :n, n:].transpose(1, 2)
    q2 = (d * d).sum(-1)
    phi = torch.exp(-q2 * e2)
    rdr = -2.0 * e2 * phi
    lj, tj = torch.atan2(x[..., 1], x[..., 0]), torch.atan2(x[..., 2], torch.hypot(x[..., 0], x[..., 1]))
    B = torch.zeros((rows, m, len(ops)), dtype=torch.float64, device=xyz.device)
    for k, op in enumerate(ops):
        grad = None  # the tangent vector whose directional derivative this operator is
        if op == "lambda":
            B[:, :n, k] = torch.cos(tj) * torch.sin(lam - lj) * rdr
            grad = east
        elif op == "theta":
            B[:, :n, k] = (torch.cos(tj) * torch.sin(th) * torch.cos(lam - lj) - torch.sin(tj) * torch.cos(th)) * rdr
            grad = north
        elif op == "lsfc":
            rd2 = rdr + 4.0 * e2 * e2 * q2 * phi
            B[:, :n, k] = 0.25 * ((4.0 - q2) * rd2 + (4.0 - 3.0 * q2) * rdr)
            if deg == 1:
                B[:, n + 1:, k] = -2.0 * c
            for q, t in enumerate(_poly_terms(deg) if deg >= 2 else []):
                if t in ((2, 0), (0, 2)):
                    B[:, n + q, k] = 2.0 / s[:, 0] ** 2
        elif op == "hv":
            y, p0, p1 = e2 * q2, torch.ones_like(q2), 4.0 * e2 * q2 - 4.0
            for j in range(2, HV_K + 1):
                p0, p1 = p1, 4.0 * (y - 2.0 * (j - 1) - 1.0) * p1 - 8.0 * (j - 1) * (2.0 * (j - 1)) * p0
            B[:, :n, k] = e2 ** HV_K * p1 * phi
        else:
            ax = "xyz".index(op[0])
            B[:, :n, k] = (c[:, ax, None] * (c[:, None] * x).sum(-1) - x[..., ax]) * rdr
            unit = torch.zeros_like(c)
            unit[:, ax] = 1.0
            grad = unit - c[:, ax, None] * c
        if grad is not None and deg == 1:
            B[:, n + 1:, k] = grad
        if grad is not None and deg >= 2:
            B[:, n + 1, k] = (grad * east).sum(1) / s[:, 0]
            B[:, n + 2, k] = (grad * north).sum(1) / s[:, 0]
    W = torch.linalg.solve(A, B)[:, :n]
    scale = [-HV_GAMMA * float(N) ** -HV_K if op == "hv" else 1.0 for op in ops]
    return W * torch.tensor(scale, dtype=torch.float64, device=xyz.device)


def exact_weights(P):
    """[N][n][operators], zero beyond a stencil's length."""
    N, n = P.st.shape
    xyz, st, eps = (torch.from_numpy(a).cuda() for a in (P.xyz, P.st, P.eps))
    W = torch.zeros((N, n, len(P.ops)), dtype=torch.float64, device="cuda")
    for size, deg in (MIX if P.lens is not None else ((n, P.deg),)):
        rows = torch.arange(N, device="cuda")
        if P.lens is not None:
            rows = rows[torch.from_numpy(P.lens).cuda() == size]
        for part in torch.split(rows, max(1, int(2e8) // (size + 15) ** 2)):
            W[part, :size] = _weights_of(xyz, st[part, :size], eps[part], deg, P.ops)
    return W


def _derivative(W, st, u):
    """sum over each stencil, tracers last."""
    out = torch.empty_like(u)
    for part in torch.split(torch.arange(len(st), device="cuda"), max(1, int(1e8) // (st.shape[1] * u.shape[1]))):
        out[part] = torch.einsum("in,int->it", W[part], u[st[part].long()])
    return out


def _rk4(f, u, dt, steps):
    for _ in range(steps):
        k1 = f(u)
        k2 = f(u + 0.5 * dt * k1)
        k3 = f(u + 0.5 * dt * k2)
        k4 = f(u + dt * k3)
        u = u + dt / 6.0 * (k1 + 2 * k2 + 2 * k3 + k4)
    return u


def _right_hand_side(P, W, flow):
    """f(u) of heat (flow None) or advection in `flow` with hyperviscosity, as one operator."""
    st = torch.from_numpy(P.st).cuda()
    if flow is None:
        L = W[:, :, 0]
    else:
        cu, cv = (torch.from_numpy(a).cuda()[:, None] for a in flow)
        hv, wl, wt = (W[:, :, k] for k in range(3))
        L = hv - cu * wl - cv * wt
    return lambda u: _derivative(L, st, u)


def _bell_flow(xyz):
    """Solid-body rotation at 90 degrees, unit sphere."""
    u0 = 2 * math.pi / REVOLUTION
    lam, th = np.arctan2(xyz[:, 1], xyz[:, 0]), np.arctan2(xyz[:, 2], np.hypot(xyz[:, 0], xyz[:, 1]))
    a = math.pi / 2
    return (u0 * (np.cos(th) * math.cos(a) + np.sin(th) * np.cos(lam) * math.sin(a)), -u0 * np.sin(lam) * math.sin(a))


def exact(case, seed):
    kind = case["kind"]
    if kind == "knn":
        return None

    def host(u, shape):
        return u.cpu().numpy().reshape(shape)

    if kind == "weights":
        P = Problem(case, seed, case["ops"], case["deg"], case["mixed"])
        W = exact_weights(P)
        if case["back"]:
            return [W[:, :, k].contiguous().cpu().numpy() for k in range(len(P.ops))]
        u, st = torch.from_numpy(smooth_field(P.xyz, 1, seed)).cuda()[:, None], torch.from_numpy(P.st).cuda()
        return [_derivative(W[:, :, k], st, u)[:, 0] for k in range(len(P.ops))]
    if kind == "serve":
        out = {}
        problems = serve_problems(case, seed)
        fs = [_right_hand_side(problems[0], exact_weights(problems[0]), None),
              _right_hand_side(problems[1], exact_weights(problems[1]), vortex_flow(problems[1].xyz, seed))]
        for i, (which, _, steps, s) in enumerate(requests_of(case, seed)):
            P = problems[which]
            N = len(P.xyz)
            u = torch.from_numpy(smooth_field(P.xyz, 1, s)).cuda()[:, None]
            out[i] = host(_rk4(fs[which], u, 0.05 / N if which == 0 else 0.3 * spacing(N), steps), N)
        return [out[i] for i in range(len(out))]
    N, T = case["N"], case["T"]
    op_set = op_set_of(case["op"]) if kind == "deriv" else ("heat" if case["pde"] == "heat" else "advect")
    P = Problem(case, seed, op_set, degree(case["n"], op_set))
    W = exact_weights(P)
    u = torch.from_numpy(smooth_field(P.xyz, T, seed)).cuda().reshape(N, T)
    if kind == "deriv":
        d = _derivative(W[:, :, P.ops.index(case["op"])], torch.from_numpy(P.st).cuda(), u)
        return host(d, (N,)) if case["host"] else d.reshape((N, T) if T > 1 else (N,))
    flow = None if case["pde"] == "heat" else (_bell_flow(P.xyz) if case["pde"] == "bell" else vortex_flow(P.xyz, seed))
    return host(_rk4(_right_hand_side(P, W, flow), u, time_step(case), case["steps"]), (N, T) if T > 1 else (N,))
