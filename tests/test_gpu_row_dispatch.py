"""Which shape of the row engine (warps per CTA, stages, register cap) products and
sweeps take on both sides of the dispatch's lines, by kernel names."""

import re

import numpy as np
import pytest

from test_gpu_tune_scope import _kernels, records  # noqa: F401

pytestmark = pytest.mark.gpu


def _matrix(cuda, points, dims, storage=0):
    n = int(np.prod(dims))
    return (cuda.gen_27pt if points == 27 else cuda.gen_7pt)(dims, np.ones(n), storage)


def _shapes(run, op):
    """(warps, stages, cap) of the launches of `op`, without repeats, in order."""
    found = []
    for name in _kernels(run):
        m = re.search(r"k_wrows<.*lgx::" + op + r"<.*>, (\d+), (\d+), (\d+)>", name)
        if m and tuple(map(int, m.groups())) not in found:
            found.append(tuple(map(int, m.groups())))
    return found


@pytest.mark.parametrize("points", [7, 27])
@pytest.mark.parametrize("dims", [(20, 20, 18), (33, 32, 31), (50, 50, 51)])
def test_jacobi_in_four_warps(cuda, records, points, dims):  # noqa: F811
    m = _matrix(cuda, points, dims)
    x = np.ones(m.row_num())
    assert _shapes(lambda: cuda.jacobi_sweep(m, x, x), "JacobiOp") == [(4, 1, 0)]
