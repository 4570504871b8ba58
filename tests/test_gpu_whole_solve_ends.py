"""How the whole-solve kernels end other than by convergence, at the sizes that take
them: non-positive curvature, right-hand sides and guesses that are not finite, an
exact breakdown of the Arnoldi process. Each as the multi-kernel solve ends."""
import numpy as np
import pytest
import scipy.sparse as sp

pytestmark = pytest.mark.gpu


def matrix(S):
    from cfdrs_b200.sparse import CsrMatrix
    return CsrMatrix.from_scipy(sp.csr_matrix(S))


def tri(n, d):
    return sp.diags([-np.ones(n - 1), np.broadcast_to(d, n), -np.ones(n - 1)], [-1, 0, 1], shape=(n, n)).tolil()


def both(cf, A, b, x0, solve):
    """Outcome with the whole-solve kernels on and off; the launches tell that both ran."""
    from cfdrs_b200.device import device_matrix
    ctx = device_matrix(A).ctx
    out = []
    try:
        for whole in (True, False):
            ctx.set_cluster_solve(whole)
            x = x0.copy()
            rep = solve(A, b, x)
            out.append((x, rep, ctx.kernel_stats()["launches"]))
    finally:
        ctx.set_cluster_solve(True)
    (x1, r1, l1), (x2, r2, l2) = out
    assert l1 <= 4
    assert r1.termination == r2.termination and r1.iterations == r2.iterations
    return out


# a few rows, the cluster's largest, beyond it (the grid)
CG_SIZES = [300, 16384, 70000, 200003]
GMRES_SIZES = [300, 10000, 40000]


@pytest.mark.parametrize("n", CG_SIZES)
@pytest.mark.parametrize("pre", ["none", "jacobi"])
def test_cg_non_positive_curvature(cuda, n, pre):
    import cfdrs_b200 as cf
    cfg = cf.IterativeSolverConfig(0.0, 1e-12, 100)
    T = tri(n, 4.0)
    k = 2 * n // 3
    T[k, k] = -40.0
    A = matrix(T)
    b = np.zeros(n)
    b[k] = 1.0  # the first direction is the negative entry's

    def solve(A, b, x):
        return cf.cg(A, b, x, cfg) if pre == "none" else cf.cg_preconditioned(A, b, cf.JacobiPreconditioner(A), x, cfg)
    (x1, r1, _), (x2, _, _) = both(cf, A, b, np.zeros(n), solve)
    if pre == "none":
        assert r1.termination == cf.Termination.NON_POSITIVE_CURVATURE and r1.iterations == 0
    np.testing.assert_array_equal(x1, x2)


@pytest.mark.parametrize("n", CG_SIZES)
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("where", ["rhs", "guess"])
def test_cg_not_finite(cuda, n, bad, where):
    import cfdrs_b200 as cf
    cfg = cf.IterativeSolverConfig(0.0, 1e-12, 100)
    A = matrix(tri(n, 4.0))
    b, x0 = np.ones(n), np.zeros(n)
    (b if where == "rhs" else x0)[n - 5] = bad
    (x1, r1, _), (x2, _, _) = both(cf, A, b, x0, lambda A, b, x: cf.cg(A, b, x, cfg))
    assert r1.termination == cf.Termination.BREAKDOWN and r1.iterations == 0
    np.testing.assert_array_equal(x1, x0)
    np.testing.assert_array_equal(x2, x0)


@pytest.mark.parametrize("n", CG_SIZES)
def test_cg_exact_in_one_step(cuda, n):
    """The first residual after a step is exactly zero: Converged, with no division by it."""
    import cfdrs_b200 as cf
    A = matrix(2.0 * sp.identity(n))
    cfg = cf.IterativeSolverConfig(0.0, 0.0, 100)
    (x1, r1, _), _ = both(cf, A, np.ones(n), np.zeros(n), lambda A, b, x: cf.cg(A, b, x, cfg))
    assert r1.termination == cf.Termination.CONVERGED and r1.iterations == 1
    np.testing.assert_array_equal(x1, 0.5)


@pytest.mark.parametrize("n", GMRES_SIZES)
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("where", ["rhs", "guess"])
def test_gmres_not_finite(cuda, n, bad, where):
    import cfdrs_b200 as cf
    cfg = cf.IterativeSolverConfig(0.0, 1e-12, 100)
    A = matrix(tri(n, 4.0))
    b, x0 = np.ones(n), np.zeros(n)
    (b if where == "rhs" else x0)[n - 5] = bad
    (x1, r1, _), (x2, _, _) = both(cf, A, b, x0, lambda A, b, x: cf.gmres(A, b, x, cfg))
    assert r1.termination == cf.Termination.BREAKDOWN and r1.iterations == 0
    np.testing.assert_array_equal(x1, x0)
    np.testing.assert_array_equal(x2, x0)


@pytest.mark.parametrize("n", GMRES_SIZES)
@pytest.mark.parametrize("pre", ["none", "jacobi"])
def test_gmres_exact_breakdown(cuda, n, pre):
    """A power of two times the identity and a unit vector: the second Arnoldi vector
    is exactly zero (hn == 0), and the solution is exact."""
    import cfdrs_b200 as cf
    cfg = cf.IterativeSolverConfig(0.0, 1e-12, 100)
    A = matrix(4.0 * sp.identity(n))
    b = np.zeros(n)
    b[n // 2] = 8.0

    def solve(A, b, x):
        return cf.gmres(A, b, x, cfg) if pre == "none" else cf.gmres_preconditioned(A, b, cf.JacobiPreconditioner(A), x, cfg)
    (x1, r1, _), (x2, _, _) = both(cf, A, b, np.zeros(n), solve)
    assert r1.termination == cf.Termination.CONVERGED and r1.iterations == 1
    np.testing.assert_array_equal(x1, b / 4.0)
    np.testing.assert_array_equal(x2, b / 4.0)


@pytest.mark.parametrize("n", GMRES_SIZES)
def test_gmres_singular(cuda, n):
    """A nilpotent shift: the process breaks down without a solution, and the budget ends it."""
    import cfdrs_b200 as cf
    cfg = cf.IterativeSolverConfig(0.0, 1e-12, 12)
    A = matrix(sp.diags([np.ones(n - 1)], [1], shape=(n, n)))
    b = np.zeros(n)
    b[n - 1] = 1.0  # outside the range; A b = e_(n-2)
    (x1, r1, _), (x2, _, _) = both(cf, A, b, np.zeros(n), lambda A, b, x: cf.gmres(A, b, x, cfg, restart=8))
    assert r1.termination == cf.Termination.MAX_ITERATIONS and r1.iterations == 12
    np.testing.assert_array_equal(x1, x2)
