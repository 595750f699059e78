"""Blocked solves at every width of the column groups (four, two or one
columns per lane; 4 to 32 lanes per row): a column's solution does not depend
on how many others share the pass, bit for bit, and solves its system."""

import numpy as np
import pytest

import oracle as lo

pytestmark = pytest.mark.gpu

PARAMS = dict(min_coarsen_size=64, partition_size=512)


# (10, 9, 8): a general finest matrix in natural order; with the red-black
# colouring: a finest level in colour order
@pytest.mark.parametrize("red_black", [False, True])
@pytest.mark.parametrize("cycle_f32", [False, True])
def test_columns_do_not_depend_on_the_width(cuda, cycle_f32, red_black):
    dims = (10, 9, 8)
    n = int(np.prod(dims))
    k = np.exp(np.random.default_rng(3).standard_normal(n))
    m, ref = cuda.gen_7pt(dims, k), lo.gen_7pt(dims, k)
    col = None
    if red_black:
        i, j, l = np.meshgrid(*[np.arange(d) for d in dims], indexing="ij")
        col = cuda.Colouring.from_array(m, ((i + j + l) % 2).ravel().astype(np.int32), 2)
    h = cuda.HierarchyWright(cycle_f32=cycle_f32, **PARAMS).instantiate(m, finest_colouring=col)
    b = np.random.default_rng(4).uniform(-1, 1, (n, 32))
    full = cuda.pcg_multi(m, h, b, rtol=1e-8)[0].cpu().numpy()
    for c in range(32):
        r = b[:, c] - lo.spmv(ref, np.ascontiguousarray(full[:, c]))
        assert np.linalg.norm(r) <= 1.01e-8 * np.linalg.norm(b[:, c])
    for width in (1, 2, 3, 4, 5, 6, 8, 12, 15, 16, 17, 20, 30, 31):
        part = cuda.pcg_multi(m, h, np.ascontiguousarray(b[:, :width]), rtol=1e-8)[0]
        np.testing.assert_array_equal(part.cpu().numpy(), full[:, :width])
