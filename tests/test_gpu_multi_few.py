"""Blocked solves around the line below which a launch takes a column per lane
(80000 lanes): a column's solution does not depend on how many others share
the pass, bit for bit, on either side, and solves its system."""

import numpy as np
import pytest

import oracle as lo

pytestmark = pytest.mark.gpu


# 2500 and 2501 rows with 32 columns are the two sides of the finest level's products
@pytest.mark.parametrize("dims", [(3, 3, 3), (4, 25, 25), (1, 41, 61), (20, 19, 18)])
@pytest.mark.parametrize("points", [7, 27])
@pytest.mark.parametrize("cycle_f32", [False, True])
def test_few_rows(cuda, dims, points, cycle_f32):
    n = int(np.prod(dims))
    k = np.exp(np.random.default_rng(3).standard_normal(n))
    m, ref = ((cuda.gen_7pt(dims, k), lo.gen_7pt(dims, k)) if points == 7 else
              (cuda.gen_27pt(dims, k), lo.gen_27pt(dims, k)))
    h = cuda.HierarchyWright(cycle_f32=cycle_f32, min_coarsen_size=16,
                             partition_size=512).instantiate(m)
    b = np.random.default_rng(4).uniform(-1, 1, (n, 32))
    full = cuda.pcg_multi(m, h, b, rtol=1e-8)[0].cpu().numpy()
    for c in range(32):
        r = b[:, c] - lo.spmv(ref, np.ascontiguousarray(full[:, c]))
        assert np.linalg.norm(r) <= 1.01e-8 * np.linalg.norm(b[:, c])
    for width in (1, 3, 8, 9, 31):
        part = cuda.pcg_multi(m, h, np.ascontiguousarray(b[:, :width]), rtol=1e-8)[0]
        np.testing.assert_array_equal(part.cpu().numpy(), full[:, :width])
