"""Half rows of the finest level (sweeps from zero, residuals after them): grid
kernels, staged and unstaged, against the general matrix's rows in the same
colour order, and V-cycles against the oracle; blocks whose tiles straddle
colours, grids of one cell per colour, relax other than 1."""

import numpy as np
import pytest

import oracle as lo

pytestmark = pytest.mark.gpu

PARAMS = dict(min_coarsen_size=16, partition_size=512)


def _colours(dims, points):
    i, j, k = np.meshgrid(*[np.arange(d) for d in dims], indexing="ij")
    c = (i % 2) * 4 + (j % 2) * 2 + (k % 2) if points == 27 else (i + j + k) % 2
    return c.ravel().astype(np.int32), 8 if points == 27 else 2


# blocks of 1 (27) cells per colour, of odd size, below / at / above a tile of
# 256 rows, of many tiles
@pytest.mark.parametrize("points,dims", [(27, (2, 2, 4)), (27, (6, 10, 14)), (27, (16, 16, 8)),
                                         (27, (16, 16, 10)), (27, (32, 40, 36)), (7, (1, 3, 4)),
                                         (7, (5, 7, 10)), (7, (8, 8, 8)), (7, (33, 20, 34))])
@pytest.mark.parametrize("form", ["fp64", "f32", "coarse_f32"])
@pytest.mark.parametrize("relax", [1.0, 0.8])
def test_half_rows_vcycle(cuda, points, dims, form, relax):
    n = int(np.prod(dims))
    k = np.exp(np.random.default_rng(9).standard_normal(n))
    m = (cuda.gen_27pt if points == 27 else cuda.gen_7pt)(dims, k)
    colours, nc = _colours(dims, points)
    kw = dict(PARAMS, smoother_relax=relax,
              **{"fp64": {}, "f32": dict(cycle_f32=True), "coarse_f32": dict(coarse_f32=True)}[form])
    hs = [cuda.HierarchyWright(grid27=g, **kw).instantiate(
        m, finest_colouring=cuda.Colouring.from_array(m, colours, nc)) for g in (True, False)]
    assert hs[0].grid27_active() and not hs[1].grid27_active()
    b = np.random.default_rng(2).uniform(-1, 1, n)
    grid, general = (h.vcycle(b).cpu().numpy() for h in hs)
    np.testing.assert_array_equal(grid, general)
    if form == "fp64":
        ref = (lo.gen_27pt if points == 27 else lo.gen_7pt)(dims, k)
        oh = lo.Amg(ref, finest_colours=colours, ncolours=nc, smoother_parts=0,
                    smoother_relax=relax, **PARAMS)
        want = oh.vcycle(b)
        assert np.abs(grid - want).max() <= 1e-11 * np.abs(want).max()
