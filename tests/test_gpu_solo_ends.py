"""One-launch CG and BiCGStab (graphs on) against the loop that looks at every
iteration (graphs off): the same ends for every tolerance, also negative and
not a number, and the same errors on systems that break down or overflow."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _outcome(cuda, fn, m, b, **kw):
    try:
        r = fn(m, b, **kw)
    except cuda.LinealError as e:
        return str(e)
    return r.iterations, r.history, r.x.cpu().numpy()


def _same(got, want):
    """Errors and iterations alike; values up to the grouping of the sums."""
    if isinstance(got, str) or isinstance(want, str):
        return got == want
    return got[0] == want[0] and all(
        np.allclose(g, w, rtol=1e-6, equal_nan=True,
                    atol=1e-9 * np.abs(w[np.isfinite(w)]).max(initial=0))
        for g, w in zip(got[1:], want[1:]))


@pytest.mark.parametrize("rtol", [-1.0, -1e-300, 0.0, 1e-200, 0.5, 1.0, 3.0, float("inf"),
                                  float("-inf"), float("nan")])
@pytest.mark.parametrize("precon", ["none", "jacobi"])
@pytest.mark.parametrize("method", ["pcg", "pbicgstab"])
def test_tolerances(cuda, method, precon, rtol):
    dims = (12, 11, 10)
    n = int(np.prod(dims))
    rng = np.random.default_rng(5)
    m = cuda.gen_7pt(dims, np.exp(rng.standard_normal(n)))
    b = rng.uniform(-1, 1, n)
    pc = cuda.PRECON_JACOBI if precon == "jacobi" else cuda.PRECON_NONE
    for maxit in (0, 1, 6):
        got, want = (_outcome(cuda, getattr(cuda, method), m, b, precon=pc, rtol=rtol,
                              maxit=maxit, use_graphs=g) for g in (True, False))
        assert _same(got, want), (maxit, got[:2], want[:2])
        if rtol < 0:
            assert got[0] == maxit


@pytest.mark.parametrize("n", [1, 2, 3, 4, 7])
def test_ends_as_stepwise(cuda, n):
    """Small integers, mostly indefinite or nonsymmetric, some right-hand sides
    close to where squares overflow: exact solutions, zero denominators,
    infinities; residuals recomputed every iteration, every second one or never."""
    rng = np.random.default_rng(n)
    for k in range(60):
        d = rng.integers(-2, 3, (n, n)).astype(float)
        if k % 2:
            d = d + d.T
        d[np.diag_indices(n)] = rng.choice([-2.0, -1.0, 1.0, 2.0], n) * (1e-160 if k % 7 == 6 else 1)
        r, c = np.nonzero(d)
        rowptr = np.zeros(n + 1, dtype=np.int64)
        np.cumsum(np.bincount(r, minlength=n), out=rowptr[1:])
        m = cuda.CsrMatrix.from_host(rowptr, c.astype(np.int32), d[r, c], symmetric=bool(k % 2))
        b = rng.integers(-2, 3, n).astype(float) * 2.0 ** (0 if k % 3 else 507 + k % 4)
        for fn in (cuda.pcg, cuda.pbicgstab):
            for pc in (cuda.PRECON_NONE, cuda.PRECON_JACOBI):
                for rere in (0, 1, 2):
                    got, want = (_outcome(cuda, fn, m, b, precon=pc, rtol=1e-14, maxit=12,
                                          rere_period=rere, use_graphs=g) for g in (True, False))
                    assert _same(got, want), (k, fn.__name__, pc, rere, got, want)


@pytest.mark.parametrize("n", [2, 20000])
def test_overflow_of_the_half_residual(cuda, n):
    """BiCGStab where the residual after the alpha step has a norm whose square
    overflows, and the products of the omega step and the next residual do not: two
    coupled rows, alone and among uncoupled ones of many CTAs."""
    rng = np.random.default_rng(2)
    at = n // 2 - 1
    length = np.ones(n, dtype=np.int64)
    length[at:at + 2] = 2
    rowptr = np.concatenate([[0], np.cumsum(length)])
    col = np.sort(np.concatenate([np.arange(n), [at, at + 1]])).astype(np.int32)
    col[at:at + 4] = [at, at + 1, at, at + 1]
    found = 0
    while found < 10:
        a = rng.uniform(-1, 1, (2, 2))
        r0 = rng.uniform(-1, 1, 2)
        r0 /= np.linalg.norm(r0)
        v = a @ r0
        half = r0 - v / (r0 @ v)
        t = a @ half
        end = half - (t @ half) / (t @ t) * t
        if half @ half < 4.0 or end @ end > 0.5 or np.abs(v @ r0) < 0.01 or t @ t < 0.01:
            continue
        found += 1
        val, b = np.ones(n + 2), np.zeros(n)
        val[at:at + 4] = a.ravel() * 2.0**-20
        b[at:at + 2] = r0 * 2.0**511.7
        m = cuda.CsrMatrix.from_host(rowptr, col, val, symmetric=False)
        got, want = (_outcome(cuda, cuda.pbicgstab, m, b, maxit=1, rtol=1e-14,
                              precon=cuda.PRECON_NONE, use_graphs=g) for g in (True, False))
        assert want == "lineal_gb300 status 5: non-finite value in iteration 1"
        assert got == want
