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


SMALL8, SMALL32, FOUR, SHORT = (1, 1, 20), (1, 1, 10), (4, 1, 0), (4, 1, 6)


# rows on both sides of 2, 8, 20 and 256 tiles per SM
@pytest.mark.parametrize("kind,points,dims,shape", [
    ("f64", 7, (8, 16, 304), SMALL8), ("f64", 7, (8, 17, 304), FOUR),
    ("f64", 7, (20, 16, 304), FOUR), ("f64", 7, (20, 17, 304), SHORT),
    ("f64", 27, (8, 16, 304), SMALL32), ("f64", 27, (8, 17, 304), FOUR),
    ("f32", 7, (2, 16, 304), SMALL8), ("f32", 7, (3, 16, 304), FOUR),
    ("f32", 7, (256, 16, 304), FOUR), ("f32", 7, (256, 17, 304), SHORT),
    ("f32", 27, (8, 16, 304), SMALL32), ("f32", 27, (8, 17, 304), FOUR),
    ("mixed", 7, (8, 16, 304), SMALL8), ("mixed", 7, (8, 17, 304), FOUR),
    ("mixed", 7, (256, 17, 304), FOUR)])
def test_product_shapes(cuda, records, kind, points, dims, shape):  # noqa: F811
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("the lines are in tiles per SM")
    m = _matrix(cuda, points, dims, 0 if kind == "f64" else 1)
    x = torch.ones(m.row_num(), dtype=torch.float32 if kind == "f32" else torch.float64,
                   device="cuda")
    run = (lambda: cuda.spmv_f32(m, x)) if kind == "f32" else (lambda: cuda.spmv(m, x))
    assert _shapes(run, "SpmvOp") == [shape]


BRANCH = (4, 1, 5)


# rows per colour on both sides of 6, 8 and 20 tiles per SM
@pytest.mark.parametrize("dtype,points,dims,shape", [
    ("float64", 7, (12, 16, 304), SMALL8), ("float64", 7, (12, 17, 304), BRANCH),
    ("float64", 7, (40, 16, 304), BRANCH), ("float64", 7, (40, 17, 304), FOUR),
    ("float32", 7, (16, 16, 304), SMALL8), ("float32", 7, (16, 17, 304), BRANCH),
    ("float32", 7, (40, 16, 304), BRANCH), ("float32", 7, (40, 17, 304), FOUR),
    ("float64", 27, (64, 16, 304), SMALL32), ("float64", 27, (64, 18, 304), FOUR),
    ("float32", 27, (64, 16, 304), SMALL32), ("float32", 27, (64, 18, 304), BRANCH),
    ("float32", 27, (160, 16, 304), BRANCH), ("float32", 27, (160, 18, 304), FOUR)])
def test_sweep_shapes(cuda, records, dtype, points, dims, shape):  # noqa: F811
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("the lines are in tiles per SM")
    i, j, k = np.meshgrid(*[np.arange(d) for d in dims], indexing="ij")
    c = (i % 2) * 4 + (j % 2) * 2 + k % 2 if points == 27 else (i + j + k) % 2
    m = _matrix(cuda, points, dims)
    col = cuda.Colouring.from_array(m, c.ravel().astype(np.int32), 8 if points == 27 else 2)
    x = torch.ones(m.row_num(), dtype=getattr(torch, dtype), device="cuda")
    assert _shapes(lambda: cuda.sor_sweep_permuted(col, x, x.clone()), "SorOp") == [shape]
