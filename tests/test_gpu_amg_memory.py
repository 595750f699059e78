"""Hierarchies where device memory is scarce: what fits in colour order (about 21
bytes per finest entry at this size) is set up and solves although the rows with
their halves would take 36, with the same V-cycle bit for bit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch

    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    return torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("form", ["fp64", "coarse_f32", "f32"])
def test_setup_with_little_memory(cuda, form):
    import torch

    dims = (100, 100, 100)
    n = int(np.prod(dims))
    m = cuda.gen_27pt(dims, np.exp(np.random.default_rng(3).standard_normal(n)))
    kw = dict(coarse_f32=form == "coarse_f32", cycle_f32=form == "f32")
    b = torch.from_numpy(np.random.default_rng(4).uniform(-1, 1, n)).cuda()
    out = torch.empty_like(b)
    want = cuda.HierarchyWright(**kw).instantiate(m).vcycle(b).clone()
    # 28 bytes an entry: the hierarchy, its set-up and 8 vectors of a solve
    ballast = torch.empty(max(_free() - 28 * m.non_zero_num(), 0), dtype=torch.uint8,
                          device="cuda")
    try:
        h = cuda.HierarchyWright(**kw).instantiate(m)
        h.vcycle(b, out=out)
        res = cuda.pcg(m, b, precon=cuda.PRECON_AMG, amg=h, rtol=1e-6, maxit=100,
                       flexible=form == "f32")
    finally:
        del ballast
        torch.cuda.empty_cache()
    assert torch.equal(out, want)
    assert res.rel_residual <= 1e-6
