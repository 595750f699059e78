"""The colour order at the edges of its counting sort (256 rows a round, 1024
rows a block, at most 64 colours; above that one pass per colour), with empty
colours: sweeps bit for bit against the oracle's in the same order."""

import numpy as np
import pytest

import oracle as lo

pytestmark = pytest.mark.gpu


def _coloured(n, ncolours, seed):
    """Random colours (some empty) and a symmetric band matrix that couples
    only rows of different colours."""
    rng = np.random.default_rng(seed)
    used = rng.permutation(ncolours)[: max(1, ncolours - ncolours // 4)]
    colours = used[rng.integers(0, len(used), n)].astype(np.int32)
    rows, cols = [np.arange(n)], [np.arange(n)]
    for off in (1, 3, 300):
        i = np.arange(max(n - off, 0))
        i = i[colours[i] != colours[i + off]]
        rows += [i, i + off]
        cols += [i + off, i]
    r, c = np.concatenate(rows), np.concatenate(cols)
    order = np.lexsort((c, r))
    r, c = r[order], c[order]
    v = rng.uniform(-1, 1, len(r))
    v[r == c] = 8.0
    rowptr = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=rowptr[1:])
    return lo.Csr(rowptr, c.astype(np.int32), v, symmetric=False), colours


@pytest.mark.parametrize("n", [1, 255, 257, 1024, 1025, 5000])
@pytest.mark.parametrize("ncolours", [1, 2, 63, 64, 65])
def test_colour_order(cuda, n, ncolours):
    ref, colours = _coloured(n, ncolours, 11)
    m = cuda.CsrMatrix.from_host(ref.rowptr, ref.col, ref.val, symmetric=False)
    col = cuda.Colouring.from_array(m, colours, ncolours)
    rng = np.random.default_rng(12)
    b, x = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    order = lo.colour_order(colours, ncolours)
    for forward in (True, False):
        want = lo.sor_sweep(ref, b, x_in=x, relax=0.9, forward=forward, order=order)
        got = cuda.sor_sweep(m, col, b, x, relax=0.9, forward=forward).cpu().numpy()
        np.testing.assert_array_equal(got, want)
    colours[n // 2] = ncolours
    with pytest.raises(cuda.LinealError):
        cuda.Colouring.from_array(m, colours, ncolours)


def _pattern(kind):
    """A clique of 70 rows within 300 (more than 64 colours, rows of 1 and of 70
    entries), or random rows with a few one-sided
    couplings."""
    rng = np.random.default_rng(21)
    if kind == "clique":
        n, member = 300, np.zeros(300, dtype=bool)
        member[rng.permutation(300)[:70]] = True
        dense = np.outer(member, member) | np.eye(300, dtype=bool)
    else:
        n = 1500
        upper = np.triu(rng.random((n, n)) < 0.005, 1)
        dense = upper | upper.T | np.eye(n, dtype=bool)
        one_sided = rng.integers(0, n, (2, 3))
        dense[one_sided[0], one_sided[1]] = True
    r, c = np.nonzero(dense)
    rowptr = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=rowptr[1:])
    return lo.Csr(rowptr, c.astype(np.int32), np.ones(len(r)), symmetric=False), dense


@pytest.mark.parametrize("kind,seed", [("clique", 1), ("clique", 2), ("unsymmetric", 1),
                                       ("unsymmetric", 2), ("unsymmetric", 4)])
def test_jp_patterns(cuda, kind, seed):
    ref, dense = _pattern(kind)
    m = cuda.CsrMatrix.from_host(ref.rowptr, ref.col, ref.val, symmetric=False)
    want, nc = lo.colour_jp(ref, seed)
    same = want[:, None] == want[None, :]
    np.fill_diagonal(same, False)
    if (same & dense).any():  # a one-sided neighbour took the colour in the same round
        with pytest.raises(cuda.LinealError):
            cuda.Colouring.jp(m, seed=seed)
        return
    got, gnc = cuda.Colouring.jp(m, seed=seed).export()
    assert gnc == nc
    np.testing.assert_array_equal(got.cpu().numpy(), want)
