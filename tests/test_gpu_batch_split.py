"""The batched BiCGStab's ways to spread a system: a CTA (up to 4096 rows), a
cluster of 16 CTAs (few larger systems) or of 8 (many), with the own rows'
vectors in shared or global memory; each system within the oracle's iterations
and its residual verified in FP64."""

import numpy as np
import pytest

import oracle as lo

pytestmark = pytest.mark.gpu

CASES = {
    # 4096 rows stay with a CTA, 4097 rows (a prime times 17) go to a cluster
    "edge": [(16, 16, 16), (17, 241, 1), (1, 1, 4097), (5, 5, 5)],
    "cluster16": [(33, 31, 29), (21, 20, 20), (3, 2, 1)],
    # more large systems than clusters of 16 fit at a time
    "cluster8": [(21, 20, 20)] * 40 + [(9, 8, 7)] * 30,
    # slices of more rows than shared memory holds vectors for
    "large": [(70, 61, 53), (64, 33, 65)],
}


@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("relax", [1.0, 0.9])
def test_batch_spread(cuda, case, relax):
    rng = np.random.default_rng(5)
    systems = [(d, tuple(float(c) for c in rng.uniform(-20.0, 20.0, 3))) for d in CASES[case]]
    bs = [rng.uniform(-1, 1, int(np.prod(d))) for d, _ in systems]
    res = cuda.batch_convdiff_bicgstab(systems, np.concatenate(bs), rtol=1e-8, maxit=1000,
                                       relax=relax)
    assert (res.status == 0).all(), res.status
    x, off = res.x.cpu().numpy(), 0
    for s, ((dims, v), b) in enumerate(zip(systems, bs)):
        xs = x[off:off + b.size]
        off += b.size
        a = lo.gen_convdiff(dims, v)
        assert np.linalg.norm(b - lo.spmv(a, xs)) <= 1.1e-8 * np.linalg.norm(b), (s, dims)
        if s < 4:
            _, it, _ = lo.pbicgstab(a, b, precon=lo.PRECON_JACOBI, relax=relax, rtol=1e-8,
                                    maxit=1000)
            assert abs(int(res.iterations[s]) - it) <= max(1, int(0.05 * it + 0.999)), (s, dims)
