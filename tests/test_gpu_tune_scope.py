"""What the autotuner's choices reach, by the names of the kernels that run: a
hierarchy's choice for its finest product stays with that hierarchy, and a level
that is tuned to the process-wide configuration runs what an untuned one runs."""

import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PARAMS = dict(min_coarsen_size=64, partition_size=512, max_partitions=1 << 30)


def _kernels(run):
    """Names of the library's kernels that `run` launches, in order."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        run()
        torch.cuda.synchronize()
    return [name for _, name in sorted((e.time_range.start, e.name) for e in p.events()
                                       if "lgx::" in e.name)]


@pytest.fixture
def records(cuda):
    """The profiler starts up in its first uses in a process, which record nothing."""
    import torch

    x = torch.zeros(64, dtype=torch.float64, device="cuda")
    if not any(_kernels(lambda: cuda.dot(x, x)) for _ in range(3)):
        pytest.skip("no kernel records on this machine")


def _matrix(cuda, dims):
    n = int(np.prod(dims))
    return cuda.gen_27pt(dims, np.exp(np.random.default_rng(5).standard_normal(n)))


def test_product_choice_stays_with_its_hierarchy(cuda, records):
    """With CTA tiles as the process-wide configuration the tuner chooses another."""
    before = cuda.row_engine()
    try:
        cuda.row_engine(0)
        m = _matrix(cuda, (60, 61, 62))
        x = np.random.default_rng(2).uniform(-1, 1, m.row_num())
        product = lambda: _kernels(lambda: cuda.spmv(m, x))
        untuned = product()
        h, other = (cuda.HierarchyWright(cycle_f32=True, **PARAMS).instantiate(m)
                    for _ in range(2))
        outer = [e for e in h.autotune(reps=3) if e["value_bytes"] == 8]
        assert len(outer) == 1 and outer[0]["config"] != 0
        assert product() == untuned

        def solve(amg):
            names = _kernels(lambda: cuda.pcg(m, x, precon=cuda.PRECON_AMG, amg=amg, rtol=1e-3,
                                              maxit=2, flexible=True))
            return {k for k in names if "SpmvOp<double, double>" in k}

        assert solve(other) == set(untuned)
        assert solve(h) and solve(h) != set(untuned)
        # a choice of the matrix's own outlives the hierarchy's, in any order
        m.autotune(reps=3)
        own = product()
        h.autotune(reps=1)
        assert product() == own
        h.autotune_reset()
        assert product() == own
        assert solve(h) == solve(other) == set(own)
    finally:
        cuda.row_engine(before)


def test_default_choice_runs_the_default(cuda, records):
    """The tuner times the process-wide configuration (3) as it runs untuned: the
    first warp-tile launches of the finest level's sweeps are the untuned ones
    (1.06M rows of 27 entries: more than eight tiles per SM and colour)."""
    assert cuda.row_engine() == 3
    dims = (101, 102, 103)
    m = _matrix(cuda, dims)
    h = cuda.HierarchyWright(**PARAMS).instantiate(m)
    b = np.random.default_rng(2).uniform(-1, 1, m.row_num())
    shape = lambda names: [re.search(r"k_wrows<.*>", k).group() for k in names
                           if "k_wrows<" in k and "lgx::SorOp<double, double>" in k]
    # the last backward sweep of a cycle is the finest level's
    untuned = shape(_kernels(lambda: h.vcycle(b)))[-2]
    tuned = shape(_kernels(lambda: h.autotune(reps=1)))
    assert tuned[0] == untuned
