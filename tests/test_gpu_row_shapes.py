"""Row launches at the edges of their shapes: few tiles in one-warp CTAs with
rounds of 8, 16 or 32 gathers, long launches in four-warp CTAs; products and
sweeps bit for bit against the oracle."""

import numpy as np
import pytest

import oracle as lo

pytestmark = pytest.mark.gpu


def _banded(n, longest, seed):
    """A symmetric pattern with rows of 1 to `longest` entries (bands at a
    spread of offsets, some rows cut to their diagonal)."""
    rng = np.random.default_rng(seed)
    half = (longest - 1) // 2
    offs = np.unique(np.concatenate([[1], (np.arange(1, half) * 7919) % max(n // 2, 2) + 2]))
    offs = offs[:half] if half else offs[:0]
    keep = rng.random(n) > 0.1
    rows = [np.arange(n)]
    cols = [np.arange(n)]
    for o in offs:
        i = np.arange(n - o)
        i = i[keep[i] & keep[i + o]]
        rows += [i, i + o]
        cols += [i + o, i]
    r, c = np.concatenate(rows), np.concatenate(cols)
    order = np.lexsort((c, r))
    r, c = r[order], c[order]
    v = rng.uniform(-1, 1, len(r))
    v[r == c] = longest + 1.0
    rowptr = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=rowptr[1:])
    return lo.Csr(rowptr, c.astype(np.int32), v, symmetric=False)


# 8 tiles per SM of 32 rows (152 SMs): 38912 rows; both sides of it, and the
# sides of a tile
@pytest.mark.parametrize("n", [1, 31, 33, 38912, 38913])
@pytest.mark.parametrize("longest", [1, 7, 9, 17, 33, 41])
def test_row_shapes_bitexact(cuda, n, longest):
    ref = _banded(n, longest, 7)
    m = cuda.CsrMatrix.from_host(ref.rowptr, ref.col, ref.val, symmetric=False)
    rng = np.random.default_rng(8)
    x, b = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    np.testing.assert_array_equal(cuda.spmv(m, x).cpu().numpy(), lo.spmv(ref, x))
    np.testing.assert_array_equal(cuda.residual(m, b, x, with_norm=False).cpu().numpy(),
                                  lo.residual(ref, b, x))
    colours, nc = lo.colour_jp(ref, 5)
    col = cuda.Colouring.from_array(m, colours, nc)
    order = lo.colour_order(colours, nc)
    for x_in in (x, None):
        want = lo.sor_sweep(ref, b, x_in=x_in, relax=0.9, forward=True, order=order)
        got = cuda.sor_sweep(m, col, b, x_in, relax=0.9).cpu().numpy()
        np.testing.assert_array_equal(got, want)
