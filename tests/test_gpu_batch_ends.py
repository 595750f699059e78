"""Where a batched BiCGStab ends in the middle of an iteration: the half step
that was taken is in x, and a residual counts as 0 exactly when the sum of its
squares is."""

import ctypes
from fractions import Fraction

import numpy as np
import pytest

import oracle as lo

pytestmark = pytest.mark.gpu


def _batch(cuda, systems, b, x0=None, **kw):
    """Through the C ABI, which leaves x and the statuses of failed systems."""
    import torch

    arr = (cuda._ConvDiffSystem * len(systems))()
    for s, (dims, v) in zip(arr, systems):
        s.dims[:] = dims
        s.v[:] = v
    n = len(systems)
    bt = torch.from_numpy(b).cuda()
    x = torch.zeros_like(bt) if x0 is None else torch.from_numpy(x0).cuda()
    it, rel, st = np.zeros(n, dtype=np.int64), np.zeros(n), np.zeros(n, dtype=np.int32)
    p = lambda a: ctypes.c_void_p(a.data_ptr() if hasattr(a, "data_ptr") else a.ctypes.data)
    cuda.lib().lgx_batch_convdiff_bicgstab(n, arr, p(bt), p(x), kw.get("rtol", 1e-8),
                                           kw.get("maxit", 10), 8, 1.0, cuda._stream(), p(it),
                                           p(rel), p(st))
    return x.cpu().numpy(), it, rel, st


def _dense(dims, v):
    import oracle as lo

    a = lo.gen_convdiff(dims, v)
    d = np.zeros((a.n, a.n))
    for i in range(a.n):
        for k in range(a.rowptr[i], a.rowptr[i + 1]):
            d[i, a.col[k]] = a.val[k]
    return d


@pytest.mark.parametrize("dims,v", [((3, 1, 1), (19.0, 0.0, 0.0)),
                                    ((5, 2, 1), (20.0, 20.0, 0.0))])
def test_overflow_in_the_middle(cuda, dims, v):
    """b as large as its norm allows, chosen so that the square of the omega step's
    product overflows: status 2 with the alpha step in x."""
    a = lo.gen_convdiff(dims, v)
    d = np.zeros((a.n, a.n))
    d[np.repeat(np.arange(a.n), np.diff(a.rowptr)), a.col] = a.val
    a, d = d, np.diag(d)
    rng = np.random.default_rng(1)
    for _ in range(2000):
        b = rng.uniform(-1, 1, len(d))
        b /= np.linalg.norm(b)
        z = b / d
        w = a @ z
        alpha = 1.0 / (b @ w)
        t = a @ ((b - alpha * w) / d)
        if t @ t > 1.2 and 1.0 < np.abs(alpha) < 1e3:
            break
    else:
        raise AssertionError("no such right-hand side")
    scale = np.sqrt(0.9) * 2.0**512  # ||b||^2 = 0.9 2^1024, t.t beyond the largest double
    x, it, _, st = _batch(cuda, [(dims, v)], b * scale)
    assert st[0] == 2 and it[0] == 0
    # 1 / (b.w) amplifies the rounding of b.w by alpha
    np.testing.assert_allclose(x, alpha * z * scale, rtol=1e-14 * max(1.0, np.abs(alpha)) * 8)


def _fma(a, b, c):
    return float(Fraction(a) * Fraction(b) + Fraction(c))


def test_residual_of_zero(cuda):
    """Two cells with right-hand sides of about 2^-534: residuals after the alpha
    step on both sides of 2^-537.5, whose square is half the smallest double (the
    step simulated in exact arithmetic with its roundings)."""
    dims, v = (2, 1, 1), (4.0, 0.0, 0.0)  # rows (10, -1), (-5, 10)
    s = 1.0 / 10.0
    rng = np.random.default_rng(0)
    zero, live = [], []
    while len(zero) < 16 or len(live) < 16:
        b = [float(t) for t in rng.uniform(-1, 1, 2) * 2.0 ** rng.uniform(-537, -530)]
        w = [_fma(-s, b[1], b[0]), _fma(-s * 5.0, b[0], b[1])]
        rho = _fma(b[0], b[0], 0.0) + _fma(b[1], b[1], 0.0)
        den = _fma(b[0], w[0], 0.0) + _fma(b[1], w[1], 0.0)
        if rho == 0.0 or den == 0.0:
            continue
        r = [_fma(-(rho / den), w[k], b[k]) for k in (0, 1)]
        top, ss = max(map(abs, r)), sum(_fma(t, t, 0.0) for t in r)
        if ss == 0.0 and top >= 2.0**-538:
            zero.append((b, rho / den * s))
        elif ss > 0.0 and top < 2.0**-537.4:
            live.append((b, rho / den * s))
    zero, live = zero[:16], live[:16]
    b = np.array([b for b, _ in zero + live])
    alpha_step = np.array([[_fma(t, a, 0.0) for t in b] for b, a in zero + live])
    x, it, rel, st = _batch(cuda, [(dims, v)] * 32, b.ravel(), rtol=1e-300, maxit=1)
    assert (st[:16] == 0).all() and (it[:16] == 1).all() and (rel[:16] == 0.0).all()
    taken = (x.reshape(32, 2) == alpha_step).all(axis=1)
    assert taken[:16].all()
    # a residual that is not 0 goes on to the omega step
    assert ((st[16:] != 0) | ~taken[16:]).all()
