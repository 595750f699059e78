"""One V-cycle whose output overlaps its right-hand side: the same vector, and
views of one buffer a few entries apart, equal the cycle on separate vectors bit
for bit, for every order that the finest level's vectors can have."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PARAMS = dict(min_coarsen_size=64, partition_size=512)


@pytest.mark.parametrize("form", ["fp64", "f32", "bf16", "given colouring", "stencil",
                                  "one level"])
def test_output_over_input(cuda, form):
    import torch

    dims = (12, 10, 14)
    n = int(np.prod(dims))
    k = np.exp(np.random.default_rng(3).standard_normal(n))
    kw = {"f32": dict(cycle_f32=True), "bf16": dict(cycle_f32=True, cycle_bf16=True),
          "one level": dict(max_level_num=1)}.get(form, {})
    col = None
    if form == "stencil":
        m = cuda.StencilMatrix.value(cuda.BoxInfo(dims, dims), None, k, 0.0, 0.0)
    else:
        m = cuda.gen_7pt(dims, k)
    if form == "given colouring":
        col = cuda.Colouring.jp(m)
    h = cuda.HierarchyWright(**PARAMS, **kw).instantiate(m, finest_colouring=col)
    b = torch.from_numpy(np.random.default_rng(4).uniform(-1, 1, n)).cuda()
    want = h.vcycle(b)
    for shift in (0, 5, -5):
        buf = torch.zeros(n + 10, dtype=torch.float64, device="cuda")
        src, dst = buf[5:5 + n], buf[5 + shift:5 + shift + n]
        src.copy_(b)
        h.vcycle(src, out=dst)
        assert torch.equal(dst, want), shift
