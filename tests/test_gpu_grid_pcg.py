"""CG / Jacobi-PCG on one cooperative grid against the multi-kernel solve: just
beyond a cluster, one to eight rows a thread, ragged last blocks, far couplings
(every row with entries in another CTA), rows longer than a register batch, a
system too large for the grid, budgets that end inside and between launches."""
import numpy as np
import pytest

from test_gpu_cluster_pcg import RTOL, banded

pytestmark = pytest.mark.gpu


def solve_both(cf, A, b, pre, x0, budget=2000, rtol=RTOL):
    from cfdrs_b200.device import device_matrix
    ctx = device_matrix(A).ctx
    cfg = cf.IterativeSolverConfig(0.0, rtol, budget)
    got = []
    try:
        for whole in (True, False):
            ctx.set_cluster_solve(whole)
            x = x0.copy()
            rep = (cf.cg_preconditioned(A, b, cf.JacobiPreconditioner(A), x, cfg) if pre == "jacobi"
                   else cf.cg(A, b, x, cfg))
            got.append((x, rep, ctx.kernel_stats()["launches"]))
    finally:
        ctx.set_cluster_solve(True)
    return got


@pytest.mark.parametrize("n,offsets", [
    (40961, (1, 300)), (65537, (1, 256)), (75776, (1, 50)), (75777, (1, 38000)), (151553, (1, 411)),
    (227329, (1, 20)), (303105, (1, 550)), (380000, (1, 616)), (450001, (1,)), (100003, (1, 2, 3, 4)),
])
@pytest.mark.parametrize("pre", ["jacobi", "none"])
def test_row_splits(cuda, n, offsets, pre):
    import cfdrs_b200 as cf
    A, kappa = banded(n, offsets)
    b = np.random.default_rng(n).uniform(-1, 1, n)
    (x1, r1, l1), (x2, r2, l2) = solve_both(cf, A, b, pre, np.linspace(-1.0, 1.0, n))
    assert l1 <= 4 and l2 > 3 * r2.iterations
    assert r1.termination == r2.termination == cf.Termination.CONVERGED
    assert abs(r1.iterations - r2.iterations) <= 1
    # residuals at most RTOL ||r0|| each: the solutions differ by at most 2 RTOL ||r0|| / lambda_min
    assert np.linalg.norm(x1 - x2) <= 2 * RTOL * r2.initial_residual_norm / 0.5
    # at the solution: no iteration
    (x3, r3, _), (_, r4, _) = solve_both(cf, A, b, pre, x2, rtol=1.0)
    assert r3.termination == r4.termination == cf.Termination.INITIAL_RESIDUAL and np.array_equal(x3, x2)


@pytest.mark.parametrize("budget", [1, 159, 160, 161, 320, 500])
def test_budget(cuda, budget):
    import cfdrs_b200 as cf
    from cfdrs_b200 import problems as P
    A, b = P.poisson_2d_dirichlet(260, 250, seed=3)
    (x1, r1, _), (x2, r2, _) = solve_both(cf, A, b, "jacobi", np.zeros_like(b), budget=budget)
    assert r1.termination == r2.termination == cf.Termination.MAX_ITERATIONS
    assert r1.iterations == r2.iterations == budget
    # the iterates agree to the rounding of the reductions, far below the error of either
    assert np.linalg.norm(x1 - x2) <= 1e-8 * np.linalg.norm(x2)


def test_larger_than_the_grid(cuda):
    import cfdrs_b200 as cf
    from cfdrs_b200.device import device_matrix
    A, _ = banded(700000, (1,))
    b = np.random.default_rng(1).uniform(-1, 1, A.nrows)
    x = np.zeros_like(b)
    rep = cf.cg(A, b, x, cf.IterativeSolverConfig(0.0, 1e-8, 500))
    assert rep.termination == cf.Termination.CONVERGED
    assert device_matrix(A).ctx.kernel_stats()["launches"] > 3 * rep.iterations
