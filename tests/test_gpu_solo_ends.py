"""One-launch CG and BiCGStab (graphs on) against the loop that looks at every
iteration (graphs off): the same ends for every tolerance, also negative and
not a number."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _outcome(cuda, fn, m, b, **kw):
    try:
        r = fn(m, b, **kw)
    except cuda.LinealError as e:
        return str(e)
    return r.iterations, r.history, r.x.cpu().numpy()


def _same(got, want):
    """Errors and iterations alike; values up to the grouping of the sums."""
    if isinstance(got, str) or isinstance(want, str):
        return got == want
    return got[0] == want[0] and all(
        np.allclose(g, w, rtol=1e-6, atol=1e-9 * np.abs(w).max(initial=0), equal_nan=True)
        for g, w in zip(got[1:], want[1:]))


@pytest.mark.parametrize("rtol", [-1.0, -1e-300, 0.0, 1e-200, 0.5, 1.0, 3.0, float("inf"),
                                  float("-inf"), float("nan")])
@pytest.mark.parametrize("precon", ["none", "jacobi"])
@pytest.mark.parametrize("method", ["pcg", "pbicgstab"])
def test_tolerances(cuda, method, precon, rtol):
    dims = (12, 11, 10)
    n = int(np.prod(dims))
    rng = np.random.default_rng(5)
    m = cuda.gen_7pt(dims, np.exp(rng.standard_normal(n)))
    b = rng.uniform(-1, 1, n)
    pc = cuda.PRECON_JACOBI if precon == "jacobi" else cuda.PRECON_NONE
    for maxit in (0, 1, 6):
        got, want = (_outcome(cuda, getattr(cuda, method), m, b, precon=pc, rtol=rtol,
                              maxit=maxit, use_graphs=g) for g in (True, False))
        assert _same(got, want), (maxit, got[:2], want[:2])
        if rtol < 0:
            assert got[0] == maxit
