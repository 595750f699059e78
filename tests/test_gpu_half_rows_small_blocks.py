"""Half rows of small parity-coloured grids: with fewer than 256 rows per colour
a tile of the residual spans several colours, and one in its middle can need
value planes that neither its first nor its last colour needs.  Blocks on both
sides of where that begins and ends, against the general rows bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# rows per colour: 64, 65, 75, 80, 85, 86, 128, 129, 140, 150, 170, 171, 192, 193, 196, 204, 205
DIMS = [(8, 8, 8), (10, 26, 2), (10, 10, 6), (8, 8, 10), (10, 34, 2), (4, 86, 2), (8, 8, 16),
        (6, 86, 2), (8, 10, 14), (10, 10, 12), (10, 4, 34), (6, 6, 38), (8, 8, 24), (2, 2, 386),
        (8, 14, 14), (8, 6, 34), (10, 82, 2)]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("form", ["fp64", "f32"])
def test_tiles_over_several_colours(cuda, dims, form):
    n = int(np.prod(dims))
    m = cuda.gen_27pt(dims, np.exp(np.random.default_rng(9).standard_normal(n)))
    i, j, k = np.meshgrid(*[np.arange(d) for d in dims], indexing="ij")
    colours = ((i % 2) * 4 + (j % 2) * 2 + (k % 2)).ravel().astype(np.int32)
    hs = [cuda.HierarchyWright(grid27=g, min_coarsen_size=16, partition_size=512,
                               cycle_f32=form == "f32").instantiate(
        m, finest_colouring=cuda.Colouring.from_array(m, colours, 8)) for g in (True, False)]
    assert hs[0].grid27_active() and not hs[1].grid27_active()
    b = np.random.default_rng(2).uniform(-1, 1, n)
    grid, general = (h.vcycle(b).cpu().numpy() for h in hs)
    np.testing.assert_array_equal(grid, general)
