"""What a program built on this package spends its time in: the cases to time it by.

Four families, each through the public entry points:

* mesh exchange    Selector gathers, Reducer segment sums, a Linsys product
                   and the aggregators, as the forward of a user's module
                   calls them one by one;
* shallow water    the tutorial's explicit time loop through ``compile`` and
                   ``eqn()``, FP64 and FP32, exact and fast arithmetic;
* single systems   ``CG.solve`` and ``GMRES.solve`` on a compiled Linsys;
* batched systems  ``BatchedPCG.solve`` over uneven meshes.
"""
import math

import torch

import easier_gb300 as esr
from easier_gb300 import mesh, workloads
from easier_gb300.numeric import Linsys
from easier_gb300.numeric.batched import BatchedPCG, p1_instance, p1_sides
from easier_gb300.numeric.preconditioner import Jacobi
from easier_gb300.numeric.solver import CG, GMRES

DTYPES = {"f32": torch.float32, "f64": torch.float64}
BYTES = {"f32": 4, "f64": 8}


def listed():
    return [
        # one exchange on a mesh of a thousand cells (a unit test's or a coarse
        # level's size): launches and host work
        dict(name="exchange_small", kind="exchange", n=16, cols=1, dtype="f64", reduce="sum"),
        # the exchange of a three-component state on two million cells, whose
        # rows (12 bytes) are no power of two
        dict(name="exchange_state", kind="exchange", n=700, cols=3, dtype="f32", reduce="sum"),
        # y = A x on the benchmark's P1 grid, as a user's own solver calls it
        dict(name="linsys_apply", kind="linsys", n=1000, dtype="f64"),
        # sums, norms and extrema of a field, as a time loop's monitor takes them
        dict(name="aggregate_field", kind="aggregate", rows=8_000_003, cols=1, dtype="f64"),
        # the tutorial's run: FP64, N = 100, a hump of water at rest
        dict(name="swe_tutorial_f64", kind="swe", n=100, dtype="f64", precision="exact", flow=False, steps=50),
        # FP64 at a size that fills the chip, in the middle of a run
        dict(name="swe_large_f64", kind="swe", n=701, dtype="f64", precision="exact", flow=True, steps=6),
        # FP32 with the default (exact) arithmetic
        dict(name="swe_exact_f32", kind="swe", n=1000, dtype="f32", precision="exact", flow=True, steps=30),
        # the benchmark's headline: N = 2000, FP32, fast arithmetic
        dict(name="swe_fast_f32", kind="swe", n=2000, dtype="f32", precision="fast", flow=True, steps=40),
        # the tutorial's finite-volume Poisson problem, CG
        dict(name="cg_tutorial", kind="cg", system="fv", n=100),
        # the benchmark's P1 Poisson problem, Jacobi-PCG
        dict(name="cg_p1", kind="cg", system="p1", n=1000),
        # ten cycles of GMRES(20) with Jacobi
        dict(name="gmres_p1", kind="gmres", n=200, restart=20, cycles=10),
        # a batch of uneven meshes with a random coefficient field
        dict(name="batch_p1", kind="batch", count=48, nmin=32, nmax=384),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["exchange", "linsys", "aggregate", "swe", "swe", "cg", "gmres", "batch"])
    if kind == "exchange":
        cols = rng.choice([1, 1, 2, 3, 4, 5])
        return dict(kind=kind, n=_log(rng, 8, 700 if cols <= 3 else 300), cols=cols, dtype=rng.choice(["f32", "f64"]),
                    reduce=rng.choice(["sum", "sum", "mean", "amax"]))
    if kind == "linsys":
        return dict(kind=kind, n=_log(rng, 10, 1000), dtype=rng.choice(["f64", "f64", "f32"]))
    if kind == "aggregate":
        cols = rng.choice([1, 1, 1, 2, 3, 5])
        return dict(kind=kind, rows=_log(rng, 100, 8_000_000 // cols), cols=cols, dtype=rng.choice(["f32", "f64"]))
    if kind == "swe":
        dtype, precision = rng.choice([("f64", "exact"), ("f64", "fast"), ("f32", "exact"), ("f32", "fast")])
        return dict(kind=kind, n=_log(rng, 8, 700 if dtype == "f64" else 1000), dtype=dtype, precision=precision,
                    flow=True, steps=rng.randint(2, 6))
    if kind == "cg":
        system = rng.choice(["fv", "p1"])
        return dict(kind=kind, system=system, n=_log(rng, 10, 150 if system == "fv" else 1000))
    if kind == "gmres":
        return dict(kind=kind, n=_log(rng, 20, 300), restart=rng.randint(5, 24), cycles=rng.randint(2, 6))
    lo = rng.randint(16, 64)
    return dict(kind=kind, count=rng.randint(1, 40), nmin=lo, nmax=lo + rng.randint(8, 256))


# ------------------------------------------------------------------ inputs --
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _field(seed, *shape, mean=1.0, dtype=torch.float64):
    """Values of a state field: around one, some per cent apart (mean 0: a
    flux)."""
    return (mean + 0.1 * torch.randn(shape, generator=_generator(seed), dtype=torch.float64, device="cuda")).to(dtype)


class Exchange(esr.Module):
    """Source values to the edges, edge fluxes summed into the cells."""

    def __init__(self, src, dst, nc, reduce):
        super().__init__()
        self.gather = esr.Selector(src)
        self.scatter = esr.Reducer(dst, nc, reduce)
        self.to("cuda")

    def forward(self, x, flux):
        return self.gather(x), self.scatter(flux)


class Operator(esr.Module):
    """A P1 stiffness matrix as a Linsys."""

    def __init__(self, n, dtype):
        super().__init__()
        s = mesh.p1_system(n)
        t = torch.from_numpy
        self.nunk = s.nunk
        self.reducer = esr.Reducer(t(s.row), s.nunk)
        self.selector = esr.Selector(t(s.col))
        self.Av = esr.Tensor(t(s.Av), mode="partition")
        self.Ae = esr.Tensor(t(s.Ae), mode="partition")
        self.A = Linsys(self.Av, self.Ae, self.selector, self.reducer)
        self.to("cuda")
        if dtype != torch.float64:
            self.to(dtype)


def _swe_state(case, seed):
    """Mesh, geometry and state: a Gaussian hump somewhere inside the unit
    square, at rest or (flow) in a large slow eddy."""
    m = mesh.triangular_mesh(case["n"], device="cuda")
    g = mesh.swe_geometry(m)
    u = torch.rand(4, generator=_generator(seed), dtype=torch.float64, device="cuda")
    x0, y0, amp, eddy = (0.3 + 0.4 * u[0]), (0.3 + 0.4 * u[1]), (0.05 + 0.05 * u[2]), (0.1 + 0.1 * u[3])
    h = 1 + amp * torch.exp(-((g.x - x0) ** 2 + (g.y - y0) ** 2) / 0.01)
    if not case["flow"]:
        return m, g, (h, torch.zeros_like(h), torch.zeros_like(h))
    sx, cx, sy, cy = (f(math.pi * a) for a in (g.x, g.y) for f in (torch.sin, torch.cos))
    return m, g, (h, eddy * h * sx * cy, -eddy * h * cx * sy)


def _dt(case):
    return min(5e-4, 0.25 / case["n"])


def _rhs(n, seed):
    """Right hand side of a P1 grid: sixteen sine modes, lumped, on a load
    that is rough at the scale of the grid."""
    x = torch.arange(1, n, dtype=torch.float64, device="cuda") / n
    k = torch.randint(1, 9, (2, 16), generator=_generator(seed), device="cuda").to(torch.float64)
    c = torch.randn(16, generator=_generator(seed + 1), dtype=torch.float64, device="cuda")
    sx, sy = torch.sin(math.pi * k[0][:, None] * x), torch.sin(math.pi * k[1][:, None] * x)
    f = torch.einsum("m,mj,mi->ji", c, sy, sx).reshape(-1)
    return f * _field(seed + 2, f.shape[0]) / (n * n)


def _poisson(case, seed):
    """(module, right hand side) of a case's Poisson problem."""
    if case.get("system") == "fv":
        m = mesh.triangular_mesh(case["n"], device="cuda")
        a = mesh.poisson_fv(m)
        b = a.b * _field(seed, a.b.shape[0])
        return workloads.Poisson(m.src, m.dst, m.nc, b, a.Ac, a.Af, device="cuda"), b
    b = _rhs(case["n"], seed)
    return workloads.P1Poisson(case["n"], b=b, device="cuda"), b


def _batch(case, seed):
    """Systems of uneven sides; fields and right hand sides from the seed."""
    return [p1_instance(i, int(n), seed) for i, n in enumerate(p1_sides(case["count"], case["nmin"], case["nmax"]))]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "exchange":
        m = mesh.triangular_mesh(case["n"], device="cuda")
        dtype = DTYPES[case["dtype"]]
        mod = Exchange(m.src, m.dst, m.nc, case["reduce"])
        esr.compile([mod], "cuda")
        tail = () if case["cols"] == 1 else (case["cols"],)
        return dict(kind=kind, mod=mod, x=_field(seed, m.nc, *tail, dtype=dtype),
                    flux=_field(seed + 1, m.ne, *tail, mean=0.0, dtype=dtype))
    if kind == "linsys":
        dtype = DTYPES[case["dtype"]]
        mod = Operator(case["n"], dtype)
        esr.compile([mod], "cuda")
        return dict(kind=kind, mod=mod, x=_field(seed, mod.nunk, dtype=dtype))
    if kind == "aggregate":
        tail = () if case["cols"] == 1 else (case["cols"],)
        return dict(kind=kind, x=_field(seed, case["rows"], *tail, dtype=DTYPES[case["dtype"]]))
    if kind == "swe":
        m, g, (h, uh, vh) = _swe_state(case, seed)
        geom = dict(sx=g.sx, sy=g.sy, alpha=g.alpha, area=g.area, x=g.x, y=g.y, bsx=g.bsx, bsy=g.bsy)
        eqn = workloads.ShallowWaterEquation(m.src, m.dst, m.bcells, geom, h, dt=_dt(case), uh=uh, vh=vh, device="cuda")
        if case["dtype"] == "f32":
            eqn.to(torch.float32)
        esr.compile([eqn], "cuda", precision=case["precision"])
        return dict(kind=kind, eqn=eqn, steps=case["steps"])
    if kind in ("cg", "gmres"):
        mod, _ = _poisson(case, seed)
        jacobi = None if case.get("system") == "fv" else Jacobi(mod.A)
        if kind == "cg":
            sol, args = CG(mod.A, mod.b, mod.x, M=jacobi), dict(rtol=1e-8)
        else:
            sol = GMRES(mod.A, mod.b, mod.x, M=jacobi, restart=case["restart"])
            args = dict(rtol=1e-12, maxiter=case["cycles"])
        esr.compile([mod, sol], "cuda")
        sol.solve(rtol=1.0, maxiter=1)  # the plan, which the solver keeps between calls
        return dict(kind=kind, mod=mod, sol=sol, args=args)
    eng = BatchedPCG(_batch(case, seed), jacobi=True, precision="df64")
    eng.autotune()
    x0 = torch.zeros(eng.pack.n, dtype=torch.float64, device="cuda")
    return dict(kind=kind, eng=eng, x0=x0, args=dict(rtol=1e-8))


def run(state):
    kind = state["kind"]
    if kind == "exchange":
        return state["mod"](state["x"], state["flux"])
    if kind == "linsys":
        return state["mod"].A(state["x"])
    if kind == "aggregate":
        x = state["x"]
        return esr.sum(x), esr.norm(x), esr.max(x), esr.min(x)
    if kind == "swe":
        eqn = state["eqn"]
        for _ in range(state["steps"]):
            eqn()
        return eqn.h.collect(), eqn.uh.collect(), eqn.vh.collect()
    if kind in ("cg", "gmres"):
        state["mod"].x[:] = 0.0
        state["sol"].solve(**state["args"])
        return state["mod"].x.data
    eng = state["eng"]
    eng.reset(state["x0"])
    eng.solve(**state["args"])
    return eng.solution()


# -------------------------------------------------------------------- work --
def _mesh_sizes(n):
    nc, ne, _, _ = mesh.mesh_sizes(n)
    return nc, ne


def _p1_sizes(n):
    """Unknowns and off-diagonal couplings of the P1 grid that are not zero
    (the four axis neighbours)."""
    m = n - 1
    return m * m, 4 * m * (m - 1)


def _solver(n, nnz, iters, vectors, touches):
    """`iters` iterations (what these systems take to 1e-8, by their side),
    each: the matrix (8-byte values, 4-byte columns) and diagonal once,
    `touches` vector reads and writes; 2 flops per multiply-add."""
    return {"bytes": iters * (12 * nnz + 8 * n * (1 + touches)), "flops": iters * 2 * (nnz + n * (1 + vectors))}


def work(case):
    kind = case["kind"]
    if kind == "exchange":
        nc, ne = _mesh_sizes(case["n"])
        row = BYTES[case["dtype"]] * case["cols"]
        return {"bytes": 8 * ne + 4 * nc + 2 * nc * row + 2 * ne * row, "flops": ne * case["cols"]}
    if kind == "linsys":
        s = BYTES[case["dtype"]]
        n = (case["n"] - 1) ** 2
        nnz = 6 * n
        return {"bytes": nnz * (4 + s) + n * (4 + 3 * s), "flops": 2 * (nnz + n)}
    if kind == "aggregate":
        n = case["rows"] * case["cols"]
        return {"bytes": 4 * n * BYTES[case["dtype"]], "flops": 5 * n}
    if kind == "swe":
        # a step: the state in and out, and per face its normal, weight and
        # neighbour; 28 operations and 2 divisions a face and stage
        nc, ne = _mesh_sizes(case["n"])
        s = BYTES[case["dtype"]]
        return {"bytes": case["steps"] * (nc * 7 * s + ne * (4 + 3 * s)), "flops": case["steps"] * 4 * (30 * ne + 12 * nc)}
    if kind == "cg":
        if case["system"] == "fv":
            n, nnz = _mesh_sizes(case["n"])
            return _solver(n, nnz, 6.8 * case["n"], 5, 10)
        n, nnz = _p1_sizes(case["n"])
        return _solver(n, nnz, 2.7 * case["n"], 6, 11)
    if kind == "gmres":
        n, nnz = _p1_sizes(case["n"])
        r = case["restart"]
        per = _solver(n, nnz, r + 1, 1, 4)
        basis = n * r * (r + 1) // 2
        return {"bytes": case["cycles"] * (per["bytes"] + 8 * basis), "flops": case["cycles"] * (per["flops"] + 4 * basis)}
    each = [_solver(*_p1_sizes(int(k)), 3.8 * int(k), 6, 11) for k in p1_sides(case["count"], case["nmin"], case["nmax"])]
    return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}


# ------------------------------------------------------------- 64-bit values --
def _exact_exchange(case, seed):
    m = mesh.triangular_mesh(case["n"], device="cuda")
    tail = () if case["cols"] == 1 else (case["cols"],)
    dtype = DTYPES[case["dtype"]]
    x = _field(seed, m.nc, *tail, dtype=dtype).double()
    flux = _field(seed + 1, m.ne, *tail, mean=0.0, dtype=dtype).double()
    at = m.dst if case["cols"] == 1 else m.dst[:, None].expand(-1, case["cols"])
    y = torch.zeros_like(x).scatter_reduce_(0, at, flux, case["reduce"], include_self=False)
    return x[m.src], y


def _apply(row, col, Ae, Av, x):
    return (x * Av).index_add_(0, row, x[col] * Ae)


def _exact_linsys(case, seed):
    s = mesh.p1_system(case["n"])
    row, col, Ae, Av = (torch.from_numpy(a).cuda() for a in (s.row, s.col, s.Ae, s.Av))
    dtype = DTYPES[case["dtype"]]
    x = _field(seed, s.nunk, dtype=dtype).double()
    return _apply(row, col, Ae.to(dtype).double(), Av.to(dtype).double(), x)


def _exact_swe(case, seed):
    m, g, state = _swe_state(case, seed)
    dtype, dt = DTYPES[case["dtype"]], _dt(case)
    sx, sy, alpha, bsx, bsy, area = (a.to(dtype).double() for a in (g.sx, g.sy, g.alpha, g.bsx, g.bsy, g.area))

    def delta(h, u, v):
        hf, uf, vf = ((1 - alpha) * a[m.src] + alpha * a[m.dst] for a in (h, u, v))
        flow, half = uf * sx + vf * sy, 0.5 * hf * hf
        wall = 0.5 * h[m.bcells] ** 2
        out = [torch.zeros_like(h) for _ in range(3)]
        out[0].index_add_(0, m.dst, flow)
        out[1].index_add_(0, m.dst, uf / hf * flow + half * sx).index_add_(0, m.bcells, wall * bsx)
        out[2].index_add_(0, m.dst, vf / hf * flow + half * sy).index_add_(0, m.bcells, wall * bsy)
        return [-a / area for a in out]

    s = [a.to(dtype).double() for a in state]
    for _ in range(case["steps"]):
        k, total = delta(*s), None
        for c in (0.5 * dt, 0.5 * dt, dt, None):
            total = k if total is None else [a + b for a, b in zip(total, k)]
            if c is not None:
                k = delta(*[a + c * b for a, b in zip(s, k)])
        s = [a + dt / 6 * b for a, b in zip(s, total)]
    return tuple(s)


def _exact_cg(row, col, Ae, Av, b, jacobi, rtol):
    inv = 1 / Av if jacobi else torch.ones_like(Av)
    x, r = torch.zeros_like(b), b.clone()
    p = z = inv * r
    rz, tol = r @ z, rtol * float(b.norm())
    while True:
        q = _apply(row, col, Ae, Av, p)
        a = rz / (p @ q)
        x, r = x + a * p, r - a * q
        if float(r.norm()) <= tol:
            return x
        z = inv * r
        new = r @ z
        p, rz = z + new / rz * p, new


def _p1_arrays(s):
    row, col, Ae, Av = (torch.as_tensor(a).cuda() for a in (s.row, s.col, s.Ae, s.Av))
    keep = Ae != 0
    return row[keep], col[keep], Ae[keep], Av


def _exact_solve(case, seed):
    if case.get("system") == "fv":
        m = mesh.triangular_mesh(case["n"], device="cuda")
        a = mesh.poisson_fv(m)
        return _exact_cg(m.src, m.dst, a.Af, a.Ac, a.b * _field(seed, a.b.shape[0]), False, 1e-8)
    return _exact_cg(*_p1_arrays(mesh.p1_system(case["n"])), _rhs(case["n"], seed), True, 1e-8)


def _exact_gmres(case, seed):
    row, col, Ae, Av = _p1_arrays(mesh.p1_system(case["n"]))
    b, R = _rhs(case["n"], seed), case["restart"]
    x = torch.zeros_like(b)
    for _ in range(case["cycles"]):
        r = b - _apply(row, col, Ae, Av, x)
        beta = r.norm()
        V, H = [r / beta], torch.zeros((R + 1, R), dtype=torch.float64, device="cuda")
        for j in range(R):
            w = _apply(row, col, Ae, Av, V[j] / Av)
            for i in range(j + 1):
                H[i, j] = V[i] @ w
                w = w - H[i, j] * V[i]
            H[j + 1, j] = w.norm()
            V.append(w / H[j + 1, j])
        e = torch.zeros((R + 1, 1), dtype=torch.float64)
        e[0] = beta.cpu()
        y = torch.linalg.lstsq(H.cpu(), e).solution.cuda()[:, 0]
        x = x + (torch.stack(V[:R], 1) @ y) / Av
    return x


def _exact_batch(case, seed):
    out = []
    for s in _batch(case, seed):
        x = _exact_cg(*_p1_arrays(s), torch.as_tensor(s.b).cuda(), True, 1e-8)
        out.append(torch.cat([x, x.new_zeros(-s.n % 256)]))
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "exchange":
        return _exact_exchange(case, seed)
    if kind == "linsys":
        return _exact_linsys(case, seed)
    if kind == "aggregate":
        tail = () if case["cols"] == 1 else (case["cols"],)
        x = _field(seed, case["rows"], *tail, dtype=DTYPES[case["dtype"]]).double()
        return (x.sum(0, keepdim=True), x.square().sum(0, keepdim=True).sqrt(), x.amax(0, keepdim=True),
                x.amin(0, keepdim=True))
    if kind == "swe":
        return _exact_swe(case, seed)
    if kind == "cg":
        return _exact_solve(case, seed)
    if kind == "gmres":
        return _exact_gmres(case, seed)
    return _exact_batch(case, seed)
