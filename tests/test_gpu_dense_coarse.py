"""The dense coarsest solve (a one-level hierarchy is nothing else): rows of odd
and even lengths, the sizes where the number of warps a row changes, and the
FP32 inverse of the mixed-precision cycle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 33, 254, 257, 1026, 2047, 2048, 2049, 2052])
def test_one_level_cycle_is_the_inverse(cuda, n):
    import cfdrs_b200 as cf
    from helpers import tridiag
    A = tridiag(n, -1.0, 3.0, -0.5)
    amg = cf.AlgebraicMultigrid(A, cf.AMGConfig(max_levels=1, coarse_solve=cf.CoarseSolve.DENSE))
    r = np.random.default_rng(n).uniform(-1, 1, n)
    want = np.linalg.solve(A.to_scipy().toarray(), r)
    # condition number below (3 + 1.5) / (3 - 1.5) = 3 in the maximum norm
    tol = 8 * (n + 8) * np.finfo(np.float64).eps
    assert np.linalg.norm(amg.apply_to(r) - want) <= tol * np.linalg.norm(want)

    S = tridiag(n, -1.0, 3.0, -1.0)
    amg = cf.AlgebraicMultigrid(S, cf.AMGConfig(max_levels=1, coarse_solve=cf.CoarseSolve.DENSE))
    x = np.zeros(n)
    rep = cf.cg_preconditioned(S, r, amg, x, cf.IterativeSolverConfig(0.0, 1e-10, 200),
                               precision=cf.Precision.FP32_REFINE)
    # an FP32 inverse contracts by about n eps32 a step: a few steps reach 1e-10
    assert rep.termination == cf.Termination.CONVERGED and rep.iterations <= 20
    assert np.linalg.norm(S.to_scipy() @ x - r) <= 1.01e-10 * max(np.linalg.norm(r), 1.0)
