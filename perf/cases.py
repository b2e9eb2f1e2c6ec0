"""Performance cases: the solves that a user of this library has it do, timed whole.

Every case goes through the package's public calls (``solve``, ``adjoint_grad``,
``spmv``, ``block_dot``, ``block_axpy``, ``nrm2``) with the matrix, the
right-hand side and the solution resident on the GPU, as a program that solves
in a loop keeps them. Systems are those of ``solver_cpp_b200/matrices.py``
(Poisson, log-normal diffusion, upwind convection-diffusion, on boxes of any
edge) and a weighted graph Laplacian for matrices that are no stencil.

The right-hand side is b = A x* for a known x* (a smooth field with noise on
top), so x* is the solution in 64 bits. Solves run to a relative residual of
1e-12, the tolerance the package's gradient workloads use (1e-11 for the
mixed-precision methods, whose FP64 check of the true residual rounds near
1e-12 on the largest systems): the solution then agrees with x* to about
1e-10 whatever order a reduction adds its terms in.
"""
import math

import numpy as np
import torch

import solver_cpp_b200 as ks

TOL = 1e-12
TOL_MIXED = 1e-11
MAXLOOP = 20000


def _c(name, kind, problem, nx, ny=1, nz=1, **kw):
    d = dict(kind=kind, problem=problem, nx=nx, ny=ny, nz=nz, **kw)
    return dict(name=name, **d) if name else d


def listed():
    return [
        # the smallest system of the configurations: a 2D Poisson solve of a few
        # thousand rows, one launch, bound by latency
        _c("cg_poisson_64x64", "solve", "poisson", 64, 64, method="CG"),
        # a 2D heterogeneous problem on an odd grid: no edge is a multiple of a
        # vector width
        _c("cg_varcoef_333x333", "solve", "varcoef", 333, 333, method="CG", sigma=1.0),
        # the 3D Poisson configuration (2.1M rows)
        _c("cg_poisson_128", "solve", "poisson", 128, 128, 128, method="CG"),
        # the largest configuration in plain FP64 (4.1M rows, log-normal diffusion)
        _c("cg_varcoef_160", "solve", "varcoef", 160, 160, 160, method="CG", sigma=1.5),
        # a matrix that is no stencil (a mesh graph, as read from a Matrix Market
        # file): the CSR path
        _c("cg_graph_250k", "solve", "graph", 250007, method="CG", degree=14, band=6000),
        # the nonsymmetric configuration: BiCG reads A and A^T
        _c("bicg_convdiff_128", "solve", "convdiff", 128, 128, 128, method="BICG"),
        # the same system with the restarted method most callers take
        _c("gmres30_convdiff_128", "solve", "convdiff", 128, 128, 128, method="GMRES", restart=30),
        # the k-skip method of the reference on an ordinary 3D grid
        _c("kskipcg2_poisson_100", "solve", "poisson", 100, 100, 100, method="KSKIPCG", kskip=2),
        # the mixed-precision headline: FP64 outer CG, 20 FP32 inner iterations
        _c("vpcg_fp32_varcoef_160", "solve", "varcoef", 160, 160, 160, method="VPCG", inner="fp32", sigma=1.5),
        # the same with BF16 matrix values inside, on an odd grid of ordinary size
        _c("vpcg_bf16_varcoef_99", "solve", "varcoef", 99, 99, 99, method="VPCG", inner="bf16", sigma=1.5),
        # forward solve and gradients with respect to b and every matrix value
        _c("adjoint_cg_varcoef_512", "adjoint", "varcoef", 512, 512, method="CG", sigma=1.0),
        # a caller's own Arnoldi step on the primitives: product, projections on
        # k basis vectors, orthogonalisation, norm
        _c("arnoldi24_convdiff_117", "arnoldi", "convdiff", 117, 117, 117, k=24),
    ]


def _edge(rng, lo, hi):
    """A grid edge, spread over the logarithm; odd as often as even."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    """A box whose edges differ by up to a quarter."""
    e = _edge(rng, lo, hi)
    return [max(4, int(round(e * rng.uniform(0.85, 1.1)))) if rng.random() < 0.5 else e for _ in range(3)]


def draw(rng):
    kind = rng.choice(["cg2d", "cg3d", "cr3d", "graph", "bicg", "gmres", "gcr", "kskip", "vpcg", "vpcg", "adjoint",
                       "arnoldi"])
    if kind == "cg2d":
        nx, ny = _edge(rng, 32, 620), _edge(rng, 32, 620)
        return _c("", "solve", rng.choice(["poisson", "varcoef"]), nx, ny, method="CG", sigma=1.0)
    if kind == "cg3d":
        nx, ny, nz = _box(rng, 16, 148)
        return _c("", "solve", rng.choice(["poisson", "varcoef"]), nx, ny, nz, method="CG", sigma=1.0)
    if kind == "cr3d":
        nx, ny, nz = _box(rng, 20, 130)
        return _c("", "solve", "poisson", nx, ny, nz, method="CR")
    if kind == "graph":
        n = _edge(rng, 5000, 600000)
        return _c("", "solve", "graph", n, method="CG", degree=rng.randrange(6, 28), band=max(64, n // rng.randrange(6, 60)))
    if kind == "bicg":
        nx, ny, nz = _box(rng, 16, 128)
        return _c("", "solve", "convdiff", nx, ny, nz, method="BICG")
    if kind in ("gmres", "gcr"):
        nx, ny, nz = _box(rng, 16, 116)
        return _c("", "solve", "convdiff", nx, ny, nz, method=kind.upper(), restart=rng.randrange(20, 51))
    if kind == "kskip":
        nx, ny, nz = _box(rng, 24, 116)
        return _c("", "solve", "poisson", nx, ny, nz, method="KSKIPCG", kskip=2)
    if kind == "vpcg":
        nx, ny, nz = _box(rng, 24, 144)
        return _c("", "solve", "varcoef", nx, ny, nz, method="VPCG", inner=rng.choice(["fp32", "fp32", "bf16"]), sigma=1.5)
    if kind == "adjoint":
        nx, ny = _edge(rng, 64, 500), _edge(rng, 64, 500)
        return _c("", "adjoint", "varcoef", nx, ny, method="CG", sigma=1.0)
    nx, ny, nz = _box(rng, 24, 116)
    return _c("", "arnoldi", "convdiff", nx, ny, nz, k=rng.randrange(4, 41))


# ---------------------------------------------------------------- systems
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * (int(seed) % (1 << 40)) + salt)
    return g


def _field(case, seed, salt):
    """A smooth field that vanishes on the boundary, with noise of 1e-3."""
    g = _gen(seed, salt)
    dims = [d for d in (case["nx"], case["ny"], case["nz"]) if d > 1]
    amp = torch.rand(3, generator=g, device="cuda", dtype=torch.float64) + 0.5
    if case["problem"] == "graph":
        t = torch.arange(dims[0], device="cuda", dtype=torch.float64) / dims[0]
        x = sum(amp[m] * torch.cos(2 * math.pi * (m + 1) * t) for m in range(3))
    else:
        x = None
        for d in dims:  # x fastest: the first edge is the last axis
            t = torch.arange(1, d + 1, device="cuda", dtype=torch.float64) / (d + 1)
            m = torch.stack([torch.sin(math.pi * (k + 1) * t) for k in range(3)])
            x = m if x is None else m.reshape(3, d, *([1] * (x.dim() - 1))) * x.unsqueeze(1)
        x = (amp.reshape(3, *([1] * (x.dim() - 1))) * x).sum(0).reshape(-1)
    noise = torch.rand(x.numel(), generator=g, device="cuda", dtype=torch.float64) - 0.5
    return x + 2e-3 * noise


class _Stencil:
    """5- or 7-point matrix on a box, rows i = ix + nx (iy + ny iz): tables of
    its coefficients by diagonal, ascending offsets."""

    def __init__(self, case, seed):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        self.n = n = nx * ny * nz
        i = torch.arange(n, device="cuda")
        axes = [(1, i % nx, nx), (nx, (i // nx) % ny, ny)] + ([(nx * ny, i // (nx * ny), nz)] if nz > 1 else [])
        dim = len(axes)
        faces = {}
        if case["problem"] == "poisson":
            one = torch.ones(n, device="cuda", dtype=torch.float64)
            diag = 2.0 * dim * one
            for off, _, _ in axes:
                faces[-off] = faces[off] = -one
        elif case["problem"] == "varcoef":  # ln kappa ~ N(0, sigma^2) per cell, harmonic-mean faces
            kap = torch.exp(case["sigma"] * torch.randn(n, generator=_gen(seed, 1), device="cuda", dtype=torch.float64))
            diag = torch.zeros(n, device="cuda", dtype=torch.float64)
            for off, c, e in axes:
                nb = torch.roll(kap, -off)
                up = torch.where(c < e - 1, 2.0 * kap * nb / (kap + nb), kap)
                lo = torch.where(c > 0, torch.roll(up, off), kap)
                faces[off], faces[-off] = -up, -lo
                diag = diag + up + lo
        else:  # first-order upwind, cell Peclet number 0.5, h = 1
            one = torch.ones(n, device="cuda", dtype=torch.float64)
            diag = torch.zeros(n, device="cuda", dtype=torch.float64)
            for (off, _, _), v in zip(axes, (1.0, 0.5, 0.25)):
                faces[-off], faces[off] = -(1.0 + v) * one, -one
                diag = diag + (2.0 + v)
        table = [(0, diag, torch.ones(n, device="cuda", dtype=torch.bool))]
        for off, c, e in axes:
            table += [(off, faces[off], c < e - 1), (-off, faces[-off], c > 0)]
        table.sort(key=lambda t: t[0])
        self.offs = [t[0] for t in table]
        self.keep = torch.stack([t[2] for t in table], 1)
        self.vals = torch.stack([t[1] for t in table], 1)

    def csr(self):
        ptr = torch.zeros(self.n + 1, device="cuda", dtype=torch.int32)
        ptr[1:] = torch.cumsum(self.keep.sum(1), 0)
        col = torch.arange(self.n, device="cuda", dtype=torch.int32)[:, None] + torch.tensor(
            self.offs, device="cuda", dtype=torch.int32)
        return ks.CSR(ptr.cpu().numpy(), col[self.keep].cpu().numpy(), self.vals[self.keep].cpu().numpy())

    def product(self, x, trans=False):
        """A x or A^T x."""
        y = torch.zeros_like(x)
        for d, off in enumerate(self.offs):
            v = torch.where(self.keep[:, d], self.vals[:, d], torch.zeros((), device="cuda", dtype=torch.float64))
            y += torch.roll(v * x, off) if trans else v * torch.roll(x, -off)
        return y

    def entries(self):
        """Row and column of every nonzero, in CSR order."""
        i = torch.arange(self.n, device="cuda")[:, None]
        cols = (i + torch.tensor(self.offs, device="cuda"))[self.keep]
        return i.expand(self.n, len(self.offs))[self.keep], cols


class _Graph:
    """Weighted Laplacian of a random mesh-like graph (neighbours within
    `band`, log-normal weights) plus a mass term: SPD, unstructured rows."""

    def __init__(self, case, seed):
        self.n = n = case["nx"]
        r = np.random.default_rng([int(seed) % (1 << 40), 7])
        m = case["degree"] // 2
        i = np.repeat(np.arange(n, dtype=np.int64), m)
        j = i + 1 + (r.random(n * m) ** 2 * case["band"]).astype(np.int64)
        i, j = i[j < n], j[j < n]
        key = np.unique(i * n + j)
        i, j = key // n, key % n
        w = np.exp(0.5 * r.standard_normal(key.shape[0]))
        rows, cols, vals = np.concatenate([i, j]), np.concatenate([j, i]), np.concatenate([-w, -w])
        deg = np.bincount(rows, weights=-vals, minlength=n)
        d = np.arange(n, dtype=np.int64)
        rows, cols, vals = np.concatenate([rows, d]), np.concatenate([cols, d]), np.concatenate([vals, deg + 0.01])
        order = np.argsort(rows * n + cols, kind="stable")
        self.rows, self.cols, self.vals = rows[order], cols[order], vals[order]

    def csr(self):
        ptr = np.zeros(self.n + 1, dtype=np.int32)
        ptr[1:] = np.cumsum(np.bincount(self.rows, minlength=self.n))
        return ks.CSR(ptr, self.cols.astype(np.int32), self.vals)

    def product(self, x):
        y = np.bincount(self.rows, weights=self.vals * x.cpu().numpy()[self.cols], minlength=self.n)
        return torch.from_numpy(y).cuda()


def _system(case, seed):
    return (_Graph if case["problem"] == "graph" else _Stencil)(case, seed)


# ---------------------------------------------------------------- the calls
def _params(case):
    p = dict(E=TOL_MIXED if "inner" in case else TOL, L=MAXLOOP)
    if "restart" in case:
        p["R"] = case["restart"]
    if "kskip" in case:
        p["K"] = case["kskip"]
    if "inner" in case:
        p.update(inner="CG", l=20, e=1e-30, inner_precision=case["inner"])
    return p


def _wrap(ctx, t):
    return ks.Vector(ctx, n=t.numel(), wrap_ptr=t.data_ptr())


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.kind = case["kind"]
    a = _system(case, seed)
    s.ctx = ks.Context(torch.cuda.current_device())
    s.mat = s.ctx.matrix(a.csr(), transpose=case.get("method") == "BICG" or s.kind == "adjoint",
                         fp32=case.get("inner") == "fp32", bf16=case.get("inner") == "bf16")
    if s.kind == "arnoldi":
        k, n = case["k"], a.n
        s.k, s.n = k, n
        s.V = torch.randn(k, n, generator=_gen(seed, 2), device="cuda", dtype=torch.float64) / math.sqrt(n)
        s.v = s.V[k - 1].clone()  # a row of V need not lie on 16 bytes, as a library vector does
        s.w = torch.empty(n, device="cuda", dtype=torch.float64)
        s.h = torch.empty(k, device="cuda", dtype=torch.float64)
        s.Vv, s.vv, s.wv = _wrap(s.ctx, s.V), _wrap(s.ctx, s.v), _wrap(s.ctx, s.w)
    else:
        s.method, s.params = case["method"], _params(case)
        s.b = a.product(_field(case, seed, 3))
        s.x = torch.empty_like(s.b)
        s.bv, s.xv = _wrap(s.ctx, s.b), _wrap(s.ctx, s.x)
        if s.kind == "adjoint":
            s.g = a.product(_field(case, seed, 4), trans=True)
            s.gb, s.gv = torch.empty_like(s.b), torch.empty(s.mat.nnz, device="cuda", dtype=torch.float64)
            s.gvec, s.gbv, s.gvv = _wrap(s.ctx, s.g), _wrap(s.ctx, s.gb), _wrap(s.ctx, s.gv)
    torch.cuda.synchronize()  # the context works on its own stream
    return s


def run(s):
    if s.kind == "arnoldi":
        ks.spmv(s.mat, s.vv, s.wv)
        ks.block_dot(s.Vv, s.n, s.k, s.wv, out_device_ptr=s.h.data_ptr())
        ks.block_axpy(s.Vv, s.n, s.k, s.h.data_ptr(), s.wv)
        return {"norm": ks.nrm2(s.wv), "h": s.h, "w": s.w}
    ks.solve(s.ctx, s.mat, s.method, s.bv, x=s.xv, **s.params)
    if s.kind == "adjoint":
        ks.adjoint_grad(s.ctx, s.mat, s.method, s.xv, s.gvec, s.gbv, s.gvv, **s.params)
        return {"x": s.x, "grad_b": s.gb, "grad_val": s.gv}
    return {"x": s.x}


def exact(case, seed):
    if case["kind"] == "arnoldi":
        a, k = _system(case, seed), case["k"]
        V = torch.randn(k, a.n, generator=_gen(seed, 2), device="cuda", dtype=torch.float64) / math.sqrt(a.n)
        w = a.product(V[k - 1])
        h = (V * w).sum(1)
        w = w - (h[:, None] * V).sum(0)
        return {"norm": w.square().sum().sqrt(), "h": h, "w": w}
    x = _field(case, seed, 3)
    if case["kind"] == "adjoint":
        lam = _field(case, seed, 4)
        rows, cols = _system(case, seed).entries()
        return {"x": x, "grad_b": lam, "grad_val": -lam[rows] * x[cols]}
    return {"x": x}


# ---------------------------------------------------------------- least work
def _iterations(case):
    """About how many iterations the method takes (a VP method: inner ones)."""
    e = max(case["nx"], case["ny"], case["nz"])
    if case["problem"] == "graph":
        return 160
    if case["problem"] == "convdiff":
        return (4.9 if "restart" in case else 4.0) * e
    if case["problem"] == "poisson":
        return (4.1 if case["nz"] > 1 else 3.4) * e
    if "inner" in case:
        return 66.0 * e
    return (29.0 if case["sigma"] > 1.2 else 10.0) * e


def work(case):
    """Bytes: every product reads the distinct matrix values once and its input
    and writes its output; a restarted method reads its basis twice per step.
    Everything else could stay on chip."""
    n = case["nx"] * case["ny"] * case["nz"]
    dim = 3 if case["nz"] > 1 else 2
    if case["problem"] == "graph":
        nnz, value = n * (case["degree"] + 1), 12
        distinct = nnz
    else:
        nnz, value = n * (2 * dim + 1), 8
        distinct = nnz if case["problem"] == "convdiff" else n * (dim + 1)
    if case["kind"] == "arnoldi":
        k = case["k"]
        return {"bytes": value * distinct + 8.0 * n * (2 * k + 4), "flops": 2.0 * nnz + 4.0 * n * k + 2.0 * n}
    its = _iterations(case)
    if "inner" in case:
        value = 4 if case["inner"] == "fp32" else 2
        return {"bytes": its * (value * distinct + 8.0 * n), "flops": its * (2.0 * nnz + 10.0 * n)}
    products = {"BICG": 2, "KSKIPCG": 2}.get(case["method"], 1) * (2 if case["kind"] == "adjoint" else 1)
    basis = case.get("restart", 0)
    return {"bytes": its * (products * (value * distinct + 16.0 * n) + 8.0 * n * basis),
            "flops": its * (products * 2.0 * nnz + 10.0 * n + 2.0 * n * basis)}
