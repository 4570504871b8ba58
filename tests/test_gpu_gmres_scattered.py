"""Plain and Jacobi GMRES of systems that fit a cluster but whose columns are
scattered over its CTAs: the separate kernels beyond the line, the cluster below
it, the same outcome as with the cluster forms off."""
import numpy as np
import pytest

from test_gpu_cg_scattered import scattered
from test_gpu_cluster_gmres import RTOL, solve_both

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,half,whole", [(2000, 10, True), (10000, 10, True), (14000, 10, False), (3000, 50, False)])
@pytest.mark.parametrize("pre", ["none", "jacobi"])
def test_scattered_columns(cuda, n, half, whole, pre):
    import cfdrs_b200 as cf
    A = scattered(n, half, seed=n)
    b = np.random.default_rng(1).uniform(-1, 1, n)
    (x1, r1, l1), (x2, r2, l2) = solve_both(cf, A, b, cf.JacobiPreconditioner(A) if pre == "jacobi" else None, 8)
    assert (l1 == 1) == whole and l2 > 10
    assert r1.termination == r2.termination == cf.Termination.CONVERGED
    assert abs(r1.iterations - r2.iterations) <= 1
    # residuals at most RTOL ||b|| each, the smallest eigenvalue at least 0.5
    assert np.linalg.norm(x1 - x2) <= 2 * RTOL * np.linalg.norm(b) / 0.5
