"""Rows of natural-order levels with the lanes along their entries: V-cycles bit
for bit against the engine configuration that gives every row a lane, and the
FP64 ones against the oracle; rows of 1 to 41 entries, one row longer than the
rest of its tile, sizes around a tile of 32 rows and around eight tiles per SM
(beyond them long rows run in eight-warp CTAs)."""

import functools

import numpy as np
import pytest

import oracle as lo

pytestmark = pytest.mark.gpu

PARAMS = dict(min_coarsen_size=16, partition_size=512)


@functools.lru_cache(maxsize=1)
def _matrix(n, longest, seed, wide=0):
    """Symmetric M-matrix of bands at a spread of offsets, some rows cut to
    their diagonal; row n / 2 coupled to `wide` others."""
    rng = np.random.default_rng(seed)
    half = (longest - 1) // 2
    offs = np.unique(np.concatenate([[1], np.arange(1, half) * 37 % max(n // 2, 2) + 2]))[:half]
    keep = rng.random(n) > 0.1
    rows, cols = [np.arange(n)], [np.arange(n)]
    for o in offs:
        i = np.arange(max(n - o, 0))
        i = i[keep[i] & keep[i + o]]
        rows += [i, i + o]
        cols += [i + o, i]
    if wide:
        far = np.setdiff1d(rng.choice(n, wide, replace=False), [n // 2])
        rows += [np.full(len(far), n // 2), far]
        cols += [far, np.full(len(far), n // 2)]
    r, c = np.concatenate(rows), np.concatenate(cols)
    key = np.unique(r.astype(np.int64) * n + c)
    r, c = key // n, key % n
    v = -(1.0 + ((np.minimum(r, c) * 31 + np.maximum(r, c)) % 17) / 17.0)
    off = np.where(r == c, 0.0, v)
    v[r == c] = 0.05 - np.bincount(r, off, n)[r[r == c]]
    rowptr = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=rowptr[1:])
    return lo.Csr(rowptr, c.astype(np.int32), v, symmetric=True)


@pytest.mark.parametrize("form", ["fp64", "f32", "coarse_f32"])
@pytest.mark.parametrize("n,longest,wide", [(31, 5, 0), (33, 9, 0), (640, 41, 0), (3000, 33, 900),
                                            (20000, 19, 0), (90000, 7, 0), (90000, 21, 0),
                                            (500000, 23, 0)])
def test_spread_rows_vcycle(cuda, n, longest, wide, form):
    ref = _matrix(n, longest, 31, wide)
    m = cuda.CsrMatrix.from_host(ref.rowptr, ref.col, ref.val, symmetric=True)
    kw = dict(PARAMS, **{"fp64": {}, "f32": dict(cycle_f32=True),
                         "coarse_f32": dict(coarse_f32=True)}[form])
    b = np.random.default_rng(2).uniform(-1, 1, n)
    before = cuda.row_engine()
    try:
        got = {}
        for config in (3, 4):
            cuda.row_engine(config)
            got[config] = cuda.HierarchyWright(**kw).instantiate(m).vcycle(b).cpu().numpy()
    finally:
        cuda.row_engine(before)
    np.testing.assert_array_equal(got[3], got[4])
    if form == "fp64":
        want = lo.Amg(ref, smoother_parts=0, **PARAMS).vcycle(b)
        assert np.abs(got[3] - want).max() <= 1e-11 * np.abs(want).max()
