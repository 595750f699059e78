"""The work that programs have this library do, as measurable cases.

Each case goes through the public Python entry points (lineal_gb300 and
lineal_gb300.autograd) the way a user's program does.  The kinds:

  product    one sparse product y = A x: assembled CSR in FP64 or FP32, or a
             matrix-free diffusion stencil
  jacobi_cg  Jacobi-preconditioned CG on the lookup stencil (constant-
             coefficient Poisson, FP64)
  ssor_cg    SSOR-preconditioned CG on an assembled operator, FP64
  bicgstab   Jacobi-preconditioned BiCGStab on an upwind convection-diffusion
             matrix (nonsymmetric, FP64)
  amg        AMG-preconditioned CG with a hierarchy that the program keeps:
             FP64 throughout, or a float cycle under float-vector CG with
             FP64 reliable updates
  once       a system that is solved once: assembly, AMG setup and solve
  batch      many small uneven convection-diffusion systems in one call
  multi      blocked AMG-CG on many right-hand sides
  adjoint    a differentiable solve, forward and backward

The conductivities are lognormal per cell, the right-hand sides uniform in
[-1, 1], the velocities uniform in [-20, 20].
"""

import math
import random

import numpy as np
import torch

import lineal_gb300 as g
from lineal_gb300 import autograd

# relative residual of the iterative solves; 1e-10 where high contrast leaves FP64 no more
RTOL, RTOL_CONTRAST = 1e-11, 1e-10


def listed():
    return [
        # a tiny operator inside a host loop: launch and call latency
        dict(name="product_small", kind="product", op="csr27", dtype="f64", n0=12, n1=11, n2=10),
        # one product of a large assembled 27-point operator on an uneven grid
        dict(name="product_csr27", kind="product", op="csr27", dtype="f64", n0=200, n1=181, n2=150),
        # the plain method at its usual small size: 64^3 Poisson, matrix-free, Jacobi-CG
        dict(name="jacobi_cg_64", kind="jacobi_cg", n0=64, n1=64, n2=64),
        # a smoother as the whole preconditioner, on a grid with odd edges
        dict(name="ssor_cg_odd", kind="ssor_cg", points=27, n0=61, n1=67, n2=71, sigma=1.5),
        # a nonsymmetric transport problem
        dict(name="bicgstab_transport", kind="bicgstab", n0=72, n1=75, n2=70),
        # the plain FP64 method at scale: 27 points, 256^3, lognormal sigma = 1.5
        dict(name="amg_f64_256", kind="amg", points=27, cycle="f64", smallest_last=True,
             n0=256, n1=256, n2=256, sigma=1.5, rtol=1e-10),
        # a mid-sized mixed solve on odd edges, where the finest level is a general matrix
        dict(name="amg_f32_odd", kind="amg", points=27, cycle="f32", smallest_last=False,
             n0=121, n1=117, n2=125, sigma=1.5, rtol=RTOL),
        # the precision form: 7 points, 256^3, high contrast, to 1e-10
        dict(name="amg_f32_contrast_256", kind="amg", points=7, cycle="f32", smallest_last=False,
             n0=256, n1=256, n2=256, sigma=3.0, rtol=RTOL_CONTRAST),
        # one system from its conductivities to its solution, setup included
        dict(name="once_27pt", kind="once", points=27, cycle="f32", n0=96, n1=100, n2=104,
             sigma=1.5),
        # a batch of small uneven systems
        dict(name="batch_192", kind="batch", systems=192, lo=12, hi=48, mix=3),
        # 128^3 Poisson with 32 right-hand sides
        dict(name="multi_32", kind="multi", rhs=32, cycle="f32", n0=128, n1=128, n2=128,
             sigma=0.0),
        # a gradient step on log-conductivities
        dict(name="adjoint_72", kind="adjoint", mixed=True, n0=72, n1=66, n2=70, sigma=1.0),
    ]


def _edges(rng, lo, hi):
    """three edges around a common size, spread over the logarithm; at times all even"""
    e = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    dims = [max(lo, min(hi, round(e * rng.uniform(0.85, 1.15)))) for _ in range(3)]
    if rng.random() < 0.5:
        dims = [d + (d & 1) for d in dims]
    return dict(zip(("n0", "n1", "n2"), dims))


def draw(rng):
    kind = rng.choice(["product", "product", "jacobi_cg", "ssor_cg", "bicgstab", "amg", "amg",
                       "once", "batch", "multi", "adjoint"])
    if kind == "product":
        op = rng.choice(["csr27", "csr7", "lookup", "value"])
        dtype = rng.choice(["f64", "f32"]) if op.startswith("csr") else "f64"
        return dict(kind=kind, op=op, dtype=dtype, **_edges(rng, 8, 200))
    if kind == "jacobi_cg":
        return dict(kind=kind, **_edges(rng, 12, 96))
    if kind == "ssor_cg":
        return dict(kind=kind, points=rng.choice([7, 27]), sigma=rng.choice([0.5, 1.5]),
                    **_edges(rng, 12, 84))
    if kind == "bicgstab":
        return dict(kind=kind, **_edges(rng, 12, 90))
    if kind == "amg":
        sigma = rng.choice([0.5, 1.5, 3.0])
        return dict(kind=kind, points=rng.choice([7, 27]), cycle=rng.choice(["f64", "f32"]),
                    smallest_last=rng.random() < 0.3, sigma=sigma,
                    rtol=RTOL_CONTRAST if sigma > 2 else RTOL, **_edges(rng, 16, 160))
    if kind == "once":
        return dict(kind=kind, points=rng.choice([7, 27]), cycle=rng.choice(["f64", "f32"]),
                    sigma=rng.choice([0.5, 1.5]), **_edges(rng, 16, 110))
    if kind == "batch":
        lo = rng.randint(8, 24)
        return dict(kind=kind, systems=round(math.exp(rng.uniform(math.log(4), math.log(190)))),
                    lo=lo, hi=rng.randint(lo, 48), mix=rng.randint(0, 1 << 20))
    if kind == "multi":
        return dict(kind=kind, rhs=rng.randint(2, 32), cycle=rng.choice(["f64", "f32"]),
                    sigma=rng.choice([0.0, 1.0]), **_edges(rng, 16, 96))
    return dict(kind=kind, mixed=rng.random() < 0.5, sigma=1.0, **_edges(rng, 16, 80))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _dims(case):
    return case["n0"], case["n1"], case["n2"]


def _rng(seed):
    r = torch.Generator(device="cuda")
    r.manual_seed(int(seed))
    return r


def _uniform(r, *shape, scale=1.0):
    return scale * (2.0 * torch.rand(*shape, generator=r, device="cuda", dtype=torch.float64) - 1.0)


def _conductivities(r, dims, sigma):
    n = dims[0] * dims[1] * dims[2]
    return torch.exp(sigma * torch.randn(n, generator=r, device="cuda", dtype=torch.float64))


def _grid_colours(dims, points):
    """parity colours of a 27-point operator, red-black ones of a 7-point one"""
    i, j, k = (torch.arange(d, device="cuda", dtype=torch.int32) for d in dims)
    i, j, k = i[:, None, None], j[None, :, None], k[None, None, :]
    c = (i % 2) * 4 + (j % 2) * 2 + (k % 2) if points == 27 else (i + j + k) % 2
    return c.expand(*dims).reshape(-1).contiguous()


def _structured(dims, points):
    """whether a program would colour the finest level by its grid: the
    red-black colours always serve, the parity colours need even edges to
    balance"""
    return points == 7 or all(d % 2 == 0 for d in dims)


def _matrix(dims, points, k, storage=g.F64):
    return (g.gen_27pt if points == 27 else g.gen_7pt)(dims, k, storage)


def _finest_colouring(a, dims, points):
    if not _structured(dims, points):
        return None
    return g.Colouring.from_array(a, _grid_colours(dims, points), 8 if points == 27 else 2)


def _convdiff_coeffs(v):
    """|a_ij| toward -d and +d on each axis, D = 1, unit spacing, upwind"""
    return [(1.0 + max(c, 0.0), 1.0 + max(-c, 0.0)) for c in v]


def _convdiff_csr(dims, v):
    """the assembled upwind operator: rows in natural order, sorted columns"""
    n0, n1, n2 = dims
    n = n0 * n1 * n2
    co = _convdiff_coeffs(v)
    idx = torch.arange(n, device="cuda").reshape(dims)
    strides = (n1 * n2, n2, 1)
    cols, vals, masks = [], [], []

    def entry(axis, side):
        m = torch.ones(dims, dtype=torch.bool, device="cuda")
        m.select(axis, 0 if side < 0 else dims[axis] - 1).fill_(False)
        cols.append(idx + side * strides[axis])
        masks.append(m)
        vals.append(-co[axis][0 if side < 0 else 1])

    for axis in range(3):
        entry(axis, -1)
    cols.append(idx)
    masks.append(torch.ones(dims, dtype=torch.bool, device="cuda"))
    vals.append(sum(x for pair in co for x in pair))
    for axis in (2, 1, 0):
        entry(axis, 1)
    mask = torch.stack(masks, -1).reshape(n, 7)
    col = torch.stack(cols, -1).reshape(n, 7)[mask].to(torch.int32)
    val = torch.tensor(vals, dtype=torch.float64, device="cuda").expand(n, 7)[mask].contiguous()
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(mask.sum(1), 0, out=rowptr[1:])
    return rowptr, col, val


def _batch_edges(case):
    r = random.Random(case["mix"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["systems"])]


def _velocities(seed, count):
    r = np.random.default_rng(seed)
    return [tuple(float(c) for c in r.uniform(-20.0, 20.0, 3)) for _ in range(count)]


def _amg_kw(case, dims, points):
    """how a program runs the float cycle: float-vector CG under FP64 reliable
    updates; on high contrast with the flexible beta and earlier updates"""
    if case["cycle"] == "f64":
        return {}
    if case["sigma"] > 2:
        return dict(refine=2, inner_rtol=1e-2, flexible=True)
    return dict(refine=2, inner_rtol=1e-4)


def _bump(dims):
    axes = [torch.arange(d, device="cuda", dtype=torch.float64) / d - 0.5 for d in dims]
    r2 = axes[0][:, None, None] ** 2 + axes[1][None, :, None] ** 2 + axes[2][None, None, :] ** 2
    return torch.exp(-40.0 * r2).reshape(-1)


def prepare(case, seed):
    kind = case["kind"]
    r = _rng(seed)
    if kind == "batch":
        edges = _batch_edges(case)
        systems = [((e,) * 3, v) for e, v in zip(edges, _velocities(seed, len(edges)))]
        return dict(case=case, systems=systems, b=_uniform(r, sum(e ** 3 for e in edges)))
    dims = _dims(case)
    n = dims[0] * dims[1] * dims[2]
    s = dict(case=case, dims=dims)
    if kind == "product":
        x = _uniform(r, n)
        if case["op"] == "lookup":
            mat = torch.randint(0, 4, (n,), generator=r, device="cuda").to(torch.uint8)
            s["a"] = g.StencilMatrix.lookup(g.BoxInfo(dims, dims), None, (0.5, 1.0, 2.0, 3.0), mat)
            s["mat"] = mat
        elif case["op"] == "value":
            s["k"] = _conductivities(r, dims, 1.5)
            s["a"] = g.StencilMatrix.value(g.BoxInfo(dims, dims), None, s["k"])
        else:
            s["k"] = _conductivities(r, dims, 1.5)
            s["a"] = _matrix(dims, 27 if case["op"] == "csr27" else 7, s["k"],
                             g.F64 if case["dtype"] == "f64" else g.F32)
        s["x"] = x if case["dtype"] == "f64" else x.to(torch.float32)
    elif kind == "jacobi_cg":
        mat = torch.ones(n, dtype=torch.uint8, device="cuda")
        s["a"] = g.StencilMatrix.lookup(g.BoxInfo(dims, dims), None, (0.0, 1.0, 0.0, 0.0), mat,
                                        0.0, 0.0)
        s["b"] = _uniform(r, n)
    elif kind == "ssor_cg":
        s["k"] = _conductivities(r, dims, case["sigma"])
        s["b"] = _uniform(r, n)
        s["a"] = _matrix(dims, case["points"], s["k"])
        s["colouring"] = g.Colouring.jp(s["a"])
    elif kind == "bicgstab":
        s["v"] = _velocities(seed, 1)[0]
        s["a"] = g.CsrMatrix.from_device(*_convdiff_csr(dims, s["v"]), symmetric=False)
        s["b"] = _uniform(r, n)
    elif kind == "amg":
        s["k"] = _conductivities(r, dims, case["sigma"])
        s["b"] = _uniform(r, n)
        s["a"] = _matrix(dims, case["points"], s["k"])
        s["h"] = g.HierarchyWright(cycle_f32=case["cycle"] == "f32",
                                   coarse_smallest_last=case["smallest_last"]).instantiate(
            s["a"], finest_colouring=_finest_colouring(s["a"], dims, case["points"]))
    elif kind == "once":
        s["k"] = _conductivities(r, dims, case["sigma"])
        s["b"] = _uniform(r, n)
    elif kind == "multi":
        s["k"] = _conductivities(r, dims, case["sigma"])
        s["b"] = _uniform(r, n, case["rhs"])
        s["a"] = _matrix(dims, 7, s["k"])
        s["h"] = g.HierarchyWright(cycle_f32=case["cycle"] == "f32").instantiate(
            s["a"], finest_colouring=_finest_colouring(s["a"], dims, 7))
    else:
        s["theta"] = (case["sigma"] * torch.randn(n, generator=r, device="cuda",
                                                  dtype=torch.float64)).requires_grad_()
        s["b"] = _bump(dims).mul_(1.0 + torch.rand((), generator=r, device="cuda",
                                                   dtype=torch.float64)).requires_grad_()
        s["target"] = _uniform(r, n, scale=0.1)
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "product":
        return (g.spmv if case["dtype"] == "f64" else g.spmv_f32)(state["a"], state["x"])
    if kind == "jacobi_cg":
        return g.pcg(state["a"], state["b"], precon=g.PRECON_JACOBI, rtol=RTOL,
                     maxit=5000).x
    if kind == "ssor_cg":
        return g.pcg(state["a"], state["b"], precon=g.PRECON_SSOR, colouring=state["colouring"],
                     rtol=RTOL, maxit=2000).x
    if kind == "bicgstab":
        return g.pbicgstab(state["a"], state["b"], precon=g.PRECON_JACOBI, rtol=RTOL,
                           maxit=2000).x
    if kind == "amg":
        return g.pcg(state["a"], state["b"], precon=g.PRECON_AMG, amg=state["h"],
                     rtol=case["rtol"], maxit=1000,
                     **_amg_kw(case, state["dims"], case["points"])).x
    if kind == "once":
        dims = state["dims"]
        a = _matrix(dims, case["points"], state["k"])
        h = g.HierarchyWright(cycle_f32=case["cycle"] == "f32").instantiate(
            a, finest_colouring=_finest_colouring(a, dims, case["points"]))
        return g.pcg(a, state["b"], precon=g.PRECON_AMG, amg=h, rtol=RTOL, maxit=1000,
                     **_amg_kw(case, dims, case["points"])).x
    if kind == "batch":
        return g.batch_convdiff_bicgstab(state["systems"], state["b"], rtol=RTOL, maxit=2000).x
    if kind == "multi":
        return g.pcg_multi(state["a"], state["h"], state["b"], rtol=RTOL)[0]
    x = autograd.diffusion7_solve(state["theta"], state["b"], state["dims"],
                                  autograd.SolveOptions(rtol=RTOL, mixed=case["mixed"]))
    loss = 0.5 * ((x - state["target"]) ** 2).sum()
    gtheta, gb = torch.autograd.grad(loss, (state["theta"], state["b"]))
    return dict(x=x.detach(), theta_grad=gtheta, b_grad=gb)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _nnz(dims, points):
    if points == 27:
        return math.prod(3 * d - 2 for d in dims)
    n = math.prod(dims)
    return n + 2 * sum(n // d * (d - 1) for d in dims)


def work(case):
    """Bytes and operations of one pass.  For the iterative solves: the
    iterations that the method takes at this size (round figures), each with
    the operator's passes (one product; an AMG cycle or SSOR application: two
    more, as a sweep from zero and the residual after it need each half of the
    matrix once; the coarse levels a third more) and five vector passes."""
    kind = case["kind"]
    if kind == "batch":
        rows = sum(e ** 3 for e in _batch_edges(case))
        it = 60
        return dict(bytes=16.0 * rows, flops=2.0 * rows * it * (2 * 7 + 12))
    dims = _dims(case)
    n = math.prod(dims)
    if kind == "product":
        w = 8 if case["dtype"] == "f64" else 4
        if case["op"] == "lookup":
            return dict(bytes=n * (1 + 16), flops=14.0 * n)
        if case["op"] == "value":
            return dict(bytes=n * 24, flops=14.0 * n)
        nnz = _nnz(dims, 27 if case["op"] == "csr27" else 7)
        return dict(bytes=nnz * (w + 4) + n * (8 + 2 * w), flops=2.0 * nnz)
    edge = n ** (1 / 3)
    if kind == "jacobi_cg":
        it = 5.6 * edge
        return dict(bytes=it * n * (1 + 8 * 6), flops=it * n * (14 + 12))
    if kind == "bicgstab":
        it = 0.9 * edge
        nnz = _nnz(dims, 7)
        return dict(bytes=it * (2 * nnz * 12 + n * 8 * 10), flops=it * (4.0 * nnz + 24 * n))
    w = 8
    points = 7 if kind in ("multi", "adjoint") else case["points"]
    nnz = _nnz(dims, points)
    if kind == "ssor_cg":
        it = 1.1 * edge
        return dict(bytes=it * (3 * nnz * 12 + n * 8 * 5), flops=it * (6.0 * nnz + 12 * n))
    rhs = case.get("rhs", 1)
    w = 8 if case.get("cycle") == "f64" or (kind == "adjoint" and not case["mixed"]) else 4
    it = 36 if kind == "multi" else (120 if case["sigma"] > 2 else 60)
    solves = 2 if kind == "adjoint" else 1
    passes = solves * it * (1 + 2 * 4 / 3)
    return dict(bytes=passes * nnz * w + solves * it * n * w * 5 * rhs,
                flops=rhs * (passes * 2.0 * nnz + solves * it * 12.0 * n))


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain torch
# ---------------------------------------------------------------------------
class _Diffusion:
    """The 7- or 27-point diffusion operator, matrix-free: harmonic-mean face
    coefficients weighted 1, 1/2, 1/4 for face, edge and corner neighbours,
    2 k on both axis-0 faces."""

    def __init__(self, dims, k, points):
        self.dims = dims
        k = k.reshape(dims)
        self.border = torch.zeros_like(k)
        self.border[0] += 2.0 * k[0]
        self.border[-1] += 2.0 * k[-1]
        self.pairs = []
        self.diag = self.border.clone()
        for dz in (0, 1):
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    steps = abs(dz) + abs(dy) + abs(dx)
                    if (dz, dy, dx) <= (0, 0, 0) or (points == 7 and steps > 1):
                        continue
                    lo = tuple(slice(max(0, -o), d - max(0, o)) for o, d in zip((dz, dy, dx), dims))
                    hi = tuple(slice(max(0, o), d - max(0, -o)) for o, d in zip((dz, dy, dx), dims))
                    a, b = k[lo], k[hi]
                    c = 2.0 * a * b / (a + b) * 0.5 ** (steps - 1)
                    self.pairs.append((lo, hi, c))
                    self.diag[lo] += c
                    self.diag[hi] += c

    def __call__(self, x):
        extra = (1,) * (x.dim() - 3)
        y = self.border.reshape(self.dims + extra) * x
        for lo, hi, c in self.pairs:
            f = c.reshape(c.shape + extra) * (x[lo] - x[hi])
            y[lo] += f
            y[hi] -= f
        return y


def _cg(apply, diag, b, tol, maxit):
    """Jacobi-CG on the leading three axes, the columns of a fourth by themselves"""
    axes = (0, 1, 2)
    dot = lambda u, v: (u * v).sum(axes, keepdim=True)  # noqa: E731
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / diag
    p = z.clone()
    rho = dot(r, z)
    stop = tol * tol * dot(b, b)
    for it in range(maxit):
        q = apply(p)
        pq = dot(p, q)
        alpha = torch.where(pq > 0, rho / pq, torch.zeros_like(rho))
        x += alpha * p
        r -= alpha * q
        z = r / diag
        new = dot(r, z)
        p = z + torch.where(rho > 0, new / rho, torch.zeros_like(rho)) * p
        rho = new
        if it % 16 == 15 and bool((dot(r, r) <= stop).all()):
            break
    return x


def _solve(op, b):
    """A^-1 b: CG, and two corrections from the recomputed residual"""
    diag = op.diag.reshape(op.dims + (1,) * (b.dim() - 3))
    x = _cg(op, diag, b, 1e-13, 20000)
    for _ in range(2):
        x += _cg(op, diag, b - op(x), 1e-4, 20000)
    return x


def _convdiff_apply(dims, co, x):
    """the upwind operator on (systems, n0 + 2, n1 + 2, n2 + 2) blocks whose
    padding is zero; co[axis][side] per system"""
    y = sum(c for pair in co for c in pair) * x
    for axis in range(3):
        y[(slice(None),) * (axis + 1) + (slice(1, None),)] -= co[axis][0] * x.narrow(
            axis + 1, 0, x.shape[axis + 1] - 1)
        y[(slice(None),) * (axis + 1) + (slice(0, -1),)] -= co[axis][1] * x.narrow(
            axis + 1, 1, x.shape[axis + 1] - 1)
    return y


def _convdiff_solve(edges, vs, bs):
    """BiCGStab on systems padded to one size, each with its own scalars; a
    second run on the recomputed residual"""
    e = [max(d[a] for d in edges) for a in range(3)]
    shape = (len(edges), e[0], e[1], e[2])
    b = torch.zeros(shape, dtype=torch.float64, device="cuda")
    mask = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for s, (d, v) in enumerate(zip(edges, bs)):
        b[s, :d[0], :d[1], :d[2]] = v.reshape(d)
        mask[s, :d[0], :d[1], :d[2]] = 1.0
    table = torch.tensor([_convdiff_coeffs(v) for v in vs], dtype=torch.float64, device="cuda")
    co = [[table[:, a, side].reshape(-1, 1, 1, 1) for side in (0, 1)] for a in range(3)]
    dg = sum(c for pair in co for c in pair)
    apply = lambda x: _convdiff_apply(e, co, x) * mask  # noqa: E731
    dot = lambda u, v: (u * v).sum((1, 2, 3), keepdim=True)  # noqa: E731
    safe = lambda u, v: torch.where(v != 0, u / v, torch.zeros_like(u))  # noqa: E731
    x = torch.zeros_like(b)
    for tol in (1e-13, 1e-4, 1e-4):
        r = b - apply(x)
        r0, p = r.clone(), r.clone()
        rho = dot(r, r0)
        stop = tol * tol * dot(r, r)
        live = torch.ones_like(rho)
        for it in range(3000):
            z = p / dg
            v = apply(z)
            alpha = safe(rho, dot(r0, v)) * live
            x += alpha * z
            r = r - alpha * v
            z = r / dg
            t = apply(z)
            omega = safe(dot(t, r), dot(t, t)) * live
            x += omega * z
            r = r - omega * t
            new = dot(r, r0)
            beta = safe(new, rho) * safe(alpha, omega)
            rho = new
            p = r + beta * (p - omega * v)
            live = (dot(r, r) > stop).to(torch.float64)
            if it % 8 == 7 and not bool(live.any()):
                break
    return [x[s, :d[0], :d[1], :d[2]].reshape(-1) for s, d in enumerate(edges)]


def exact(case, seed):
    kind = case["kind"]
    r = _rng(seed)
    if kind == "batch":
        edges = [(e,) * 3 for e in _batch_edges(case)]
        b = _uniform(r, sum(e[0] ** 3 for e in edges))
        return torch.cat(_convdiff_solve(edges, _velocities(seed, len(edges)),
                                         b.split([e[0] ** 3 for e in edges])))
    dims = _dims(case)
    n = math.prod(dims)
    if kind == "bicgstab":
        return _convdiff_solve([dims], _velocities(seed, 1), [_uniform(r, n)])[0]
    if kind == "jacobi_cg":
        op = _Diffusion(dims, torch.ones(n, dtype=torch.float64, device="cuda"), 7)
        return _solve(op, _uniform(r, n).reshape(dims)).reshape(-1)
    if kind == "product":
        x = _uniform(r, n)
        if case["op"] == "lookup":
            mat = torch.randint(0, 4, (n,), generator=r, device="cuda")
            k = torch.tensor([0.5, 1.0, 2.0, 3.0], dtype=torch.float64, device="cuda")[mat]
        else:
            k = _conductivities(r, dims, 1.5)
        if case["dtype"] == "f32":
            x = x.to(torch.float32).to(torch.float64)
        op = _Diffusion(dims, k, 27 if case["op"] == "csr27" else 7)
        return op(x.reshape(dims)).reshape(-1)
    if kind == "adjoint":
        theta = case["sigma"] * torch.randn(n, generator=r, device="cuda", dtype=torch.float64)
        b = _bump(dims).mul_(1.0 + torch.rand((), generator=r, device="cuda", dtype=torch.float64))
        target = _uniform(r, n, scale=0.1)
        op = _Diffusion(dims, torch.exp(theta), 7)
        x = _solve(op, b.reshape(dims))
        lam = _solve(op, x - target.reshape(dims))
        theta.requires_grad_()
        s = -(lam * _Diffusion(dims, torch.exp(theta), 7)(x)).sum()
        return dict(x=x.reshape(-1), theta_grad=torch.autograd.grad(s, theta)[0],
                    b_grad=lam.reshape(-1))
    if n > 4_000_000:  # CG by plain torch would take too long
        return None
    k = _conductivities(r, dims, case["sigma"])
    if kind == "multi":
        b = _uniform(r, n, case["rhs"]).reshape(dims + (case["rhs"],))
        return _solve(_Diffusion(dims, k, 7), b).reshape(n, case["rhs"])
    op = _Diffusion(dims, k, case["points"])
    return _solve(op, _uniform(r, n).reshape(dims)).reshape(-1)
