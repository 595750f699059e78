"""Which systems the one-launch solvers take, by the number of launches, and
their results on full grids of CTAs: one CTA per SM, two per SM, and the sizes
from which the launches of the step-by-step loop are the better way."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(cuda, method, m, b, **kw):
    kw = dict(dict(precon=cuda.PRECON_JACOBI, rtol=-1.0, maxit=5, rere_period=3), **kw)
    m.diagonal()  # kept by the matrix
    before = cuda.kernel_launches()
    r = getattr(cuda, method)(m, b, **kw)
    return r, cuda.kernel_launches() - before


def _banded(cuda, n, per_row, long_rows=0, long_len=0):
    """`per_row` entries in each row; the first `long_rows` rows also couple to
    every row of a stretch of `long_len` (symmetric)."""
    half = (per_row - 1) // 2
    i = np.arange(n)
    rows, cols = [i], [i]
    for o in (1 + np.arange(half) * 37) % (n // 2 - 1) + 1:
        rows += [i, (i + o) % n]
        cols += [(i + o) % n, i]
    for q in range(long_rows):
        far = n // 2 + (q * 97 + np.arange(long_len)) % (n // 2 - 1)
        rows += [np.full(long_len, q), far]
        cols += [far, np.full(long_len, q)]
    key = np.unique(np.concatenate(rows).astype(np.int64) * n + np.concatenate(cols))
    r, c = key // n, key % n
    count = np.bincount(r, minlength=n)
    rowptr = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(count, out=rowptr[1:])
    v = np.where(r == c, count[r] + 0.5, -1.0)
    return cuda.CsrMatrix.from_host(rowptr, c.astype(np.int32), v, symmetric=True)


# 90 x 30 x 29 = 78,300 rows: every SM has a CTA; 610,000 rows: two per SM;
# 1,500,000 rows are the last, 1,500,100 the first of the other way
@pytest.mark.parametrize("method", ["pcg", "pbicgstab"])
@pytest.mark.parametrize("dims,one", [((90, 30, 29), True), ((100, 100, 61), True),
                                      ((100, 100, 150), True), ((100, 7, 2143), False)])
def test_full_grids(cuda, method, dims, one):
    n = int(np.prod(dims))
    rng = np.random.default_rng(3)
    mat = rng.integers(0, 4, n).astype(np.uint8)
    m = cuda.StencilMatrix.lookup(cuda.BoxInfo(dims, dims), None, (0.5, 1.0, 2.0, 3.0), mat, 0.0,
                                  0.0)
    b = rng.uniform(-1, 1, n)
    got, launches = _solve(cuda, method, m, b)
    want, _ = _solve(cuda, method, m, b, use_graphs=False)
    assert (launches <= 2) == one
    assert got.iterations == want.iterations == 5
    np.testing.assert_allclose(got.history, want.history, rtol=1e-9)
    scale = np.abs(want.x.cpu().numpy()).max()
    np.testing.assert_allclose(got.x.cpu().numpy(), want.x.cpu().numpy(), rtol=1e-8,
                               atol=1e-10 * scale)


def test_entries_decide(cuda):
    b = np.random.default_rng(4).uniform(-1, 1, 4000)
    # short rows, and rows long enough that a thread's chain outlasts the launches
    for per_row, one in ((7, True), (61, True), (1201, False)):
        assert (_solve(cuda, "pcg", _banded(cuda, 4000, per_row), b)[1] <= 2) == one, per_row
    # a few rows far longer than the rest: their CTA would keep all others waiting
    m = _banded(cuda, 4000, 5, 3, 1500)
    got, launches = _solve(cuda, "pcg", m, b)
    assert launches > 2
    want, _ = _solve(cuda, "pcg", m, b, use_graphs=False)
    np.testing.assert_allclose(got.history, want.history, rtol=1e-9)
    # 27 points, up to 1.5M rows: 29.8M and 37.3M entries
    for d, one in ((104, True), (112, False)):
        m = cuda.gen_27pt((d, d, d), np.ones(d**3))
        b = np.random.default_rng(4).uniform(-1, 1, d**3)
        assert (_solve(cuda, "pcg", m, b)[1] <= 2) == one, d
