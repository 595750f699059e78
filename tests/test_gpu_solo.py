"""CG and BiCGStab in one launch (no preconditioner, Jacobi): against the
oracle's solves over the operators and sizes that the grid of CTAs splits
differently, with the solver object's iteration by iteration as the other path;
stopping, recomputed residuals and error cases as there."""

import numpy as np
import pytest

import oracle as lo

pytestmark = pytest.mark.gpu


def _operator(cuda, kind, dims, seed=3):
    n = int(np.prod(dims))
    rng = np.random.default_rng(seed)
    k = np.exp(0.5 * rng.standard_normal(n))
    if kind == "lookup":
        mat, coeffs = rng.integers(0, 4, n).astype(np.uint8), (0.5, 1.0, 2.0, 3.0)
        m = cuda.StencilMatrix.lookup(cuda.BoxInfo(dims, dims), None, coeffs, mat, 0.0, 0.0)
        return m, lo.Stencil(dims, mat=mat, coeffs=coeffs, sol_start=0, sol_end=0).to_csr()[0]
    if kind == "value":
        m = cuda.StencilMatrix.value(cuda.BoxInfo(dims, dims), None, k, 0.0, 0.0)
        return m, lo.Stencil(dims, k=k, sol_start=0, sol_end=0).to_csr()[0]
    if kind == "convdiff":
        ref = lo.gen_convdiff(dims, (6.0, -3.0, 2.0))
        return cuda.CsrMatrix.from_host(ref.rowptr, ref.col, ref.val, symmetric=False), ref
    gen, ogen = (cuda.gen_27pt, lo.gen_27pt) if kind == "csr27" else (cuda.gen_7pt, lo.gen_7pt)
    return gen(dims, k), ogen(dims, k)


# one CTA (up to 1023 rows), the edges of a CTA's rows, many CTAs
DIMS = [(1, 1, 2), (9, 8, 7), (8, 8, 16), (31, 33, 1), (41, 37, 29)]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("kind", ["lookup", "value", "csr7", "csr27", "convdiff"])
@pytest.mark.parametrize("method", ["cg", "bicgstab"])
@pytest.mark.parametrize("precon,relax", [("jacobi", 1.0), ("jacobi", 0.8), ("none", 1.0)])
def test_solo_matches_oracle(cuda, dims, kind, method, precon, relax):
    if method == "cg" and kind == "convdiff":
        pytest.skip("nonsymmetric")
    m, ref = _operator(cuda, kind, dims)
    b = np.random.default_rng(4).uniform(-1, 1, ref.n)
    fn, ofn = (cuda.pcg, lo.pcg) if method == "cg" else (cuda.pbicgstab, lo.pbicgstab)
    pc, opc = ((cuda.PRECON_JACOBI, lo.PRECON_JACOBI) if precon == "jacobi"
               else (cuda.PRECON_NONE, lo.PRECON_NONE))
    res = fn(m, b, precon=pc, relax=relax, rtol=1e-9, maxit=2000)
    _, it, hist = ofn(ref, b, precon=opc, relax=relax, rtol=1e-9, maxit=2000)
    x = res.x.cpu().numpy()
    assert res.rel_residual <= 1e-9
    assert np.linalg.norm(b - lo.spmv(ref, x)) <= 1.01e-9 * np.linalg.norm(b)
    # rounding moves BiCGStab's path more than CG's
    slack = 0.05 if method == "cg" else 0.15
    assert abs(res.iterations - it) <= max(2, slack * it + 1)
    assert len(res.history) == res.iterations + 1
    head = min(4, it, res.iterations) + 1
    np.testing.assert_allclose(res.history[:head], hist[:head], rtol=1e-8,
                               atol=1e-9 * hist[0])


def test_solo_initial_guess_limits_and_errors(cuda):
    dims = (12, 11, 10)
    m, ref = _operator(cuda, "csr7", dims)
    b = np.random.default_rng(5).uniform(-1, 1, ref.n)
    full = cuda.pcg(m, b, precon=cuda.PRECON_JACOBI, rtol=1e-10, maxit=2000)
    # a start at the solution needs no iteration to its own tolerance
    again = cuda.pcg(m, b, x0=full.x, precon=cuda.PRECON_JACOBI, rtol=1.0, maxit=10)
    assert again.iterations == 0
    np.testing.assert_array_equal(again.x.cpu().numpy(), full.x.cpu().numpy())
    # maxit is exact, and the launches' path (use_graphs=0) takes the same steps
    for maxit in (0, 1, 9, 17):
        a = cuda.pcg(m, b, precon=cuda.PRECON_JACOBI, rtol=1e-12, maxit=maxit)
        e = cuda.pcg(m, b, precon=cuda.PRECON_JACOBI, rtol=1e-12, maxit=maxit, use_graphs=False)
        assert a.iterations == e.iterations == maxit
        np.testing.assert_allclose(a.history, e.history, rtol=1e-9)
        np.testing.assert_allclose(a.x.cpu().numpy(), e.x.cpu().numpy(), rtol=1e-9, atol=1e-12)
    # zero right-hand side: solved at once
    zero = cuda.pcg(m, np.zeros(ref.n), precon=cuda.PRECON_JACOBI)
    assert zero.iterations == 0 and not zero.x.any()
    for bad in (np.inf, np.nan):
        c = b.copy()
        c[7] = bad
        for fn in (cuda.pcg, cuda.pbicgstab):
            with pytest.raises(cuda.LinealError, match="non-finite initial residual"):
                fn(m, c, precon=cuda.PRECON_JACOBI)
    # r.Ar = 0 with r != 0: both paths end with the same status
    ind = lo.Csr(np.array([0, 2, 4]), np.array([0, 1, 0, 1], dtype=np.int32),
                 np.array([1.0, 0.0, 0.0, -1.0]))
    im = cuda.CsrMatrix.from_host(ind.rowptr, ind.col, ind.val)
    status = []
    for graphs in (True, False):
        with pytest.raises(cuda.LinealError) as err:
            cuda.pcg(im, np.array([1.0, 1.0]), precon=cuda.PRECON_NONE, use_graphs=graphs)
        status.append(err.value.status)
    assert status[0] == status[1]
