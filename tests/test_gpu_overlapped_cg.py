"""Preconditioned CG with the host half an iteration behind (graphs on) against
the loop that looks at every iteration's end (graphs off): the same iterates,
histories and errors, bit for bit, also where the solve ends in the middle."""

import numpy as np
import pytest

import oracle as lo

pytestmark = pytest.mark.gpu


def _outcome(cuda, *args, **kw):
    try:
        r = cuda.pcg(*args, **kw)
    except cuda.LinealError as e:
        return str(e)
    return r.iterations, r.rel_residual, r.history.tolist(), r.x.cpu().numpy().tobytes()


@pytest.mark.parametrize("precon", ["ssor", "amg"])
@pytest.mark.parametrize("flexible", [False, True])
@pytest.mark.parametrize("stop", [dict(), dict(maxit=1), dict(maxit=9), dict(rtol=0.5),
                                  dict(rere_period=0), dict(rere_period=1)])
def test_overlapped_matches_stepwise(cuda, precon, flexible, stop):
    dims = (9, 14, 11)
    n = int(np.prod(dims))
    rng = np.random.default_rng(5)
    a = cuda.gen_7pt(dims, np.exp(rng.standard_normal(n)))
    kw = dict(dict(rtol=1e-10, maxit=500, flexible=flexible), **stop)
    if precon == "ssor":
        kw.update(precon=cuda.PRECON_SSOR, colouring=cuda.Colouring.jp(a))
    else:
        kw.update(precon=cuda.PRECON_AMG, amg=cuda.HierarchyWright(
            min_coarsen_size=16, partition_size=128).instantiate(a))
    b = rng.uniform(-1, 1, n)
    want = _outcome(cuda, a, b, use_graphs=False, **kw)
    assert _outcome(cuda, a, b, use_graphs=True, **kw) == want
    assert not isinstance(want, str)


@pytest.mark.parametrize("n", [1, 2, 3, 4])
def test_overlapped_ends_as_stepwise(cuda, n):
    """Small symmetric systems of small integers, mostly indefinite: exact
    solutions, zero rho, zero denominators and overflow within a few steps."""
    rng = np.random.default_rng(n)
    ends = set()
    for k in range(60):
        d = rng.integers(-2, 3, (n, n)).astype(float)
        d = d + d.T
        d[np.diag_indices(n)] = rng.choice([-2.0, -1.0, 1.0, 2.0], n) * (1e-160 if k % 7 == 6 else 1)
        r, c = np.nonzero(d)
        rowptr = np.zeros(n + 1, dtype=np.int64)
        np.cumsum(np.bincount(r, minlength=n), out=rowptr[1:])
        m = cuda.CsrMatrix.from_host(rowptr, c.astype(np.int32), d[r, c], symmetric=True)
        b = rng.integers(-2, 3, n).astype(float)
        kw = dict(precon=cuda.PRECON_SSOR, rtol=1e-14, maxit=12)
        want = _outcome(cuda, m, b, use_graphs=False, **kw)
        assert _outcome(cuda, m, b, use_graphs=True, **kw) == want
        ends.add(want if isinstance(want, str) else "done")
    assert "done" in ends
