"""CG of systems that fit a cluster but whose columns are scattered over its CTAs
runs on the grid form, with the multi-kernel solve's outcome; stencils, whose
neighbouring rows share their remote entries, stay with the cluster."""
import numpy as np
import pytest

from test_gpu_cluster_pcg import banded
from test_gpu_grid_pcg import solve_both

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def scattered(n, half, seed):
    """Symmetric, `half` random off-diagonals -1 a row and their transposes; dominant by 0.5."""
    import scipy.sparse as sp
    from cfdrs_b200.sparse import CsrMatrix
    j = np.random.default_rng(seed).integers(0, n, n * half)
    S = sp.csr_matrix((np.ones(n * half), (np.repeat(np.arange(n), half), j)), shape=(n, n))
    S = S + S.T
    S.setdiag(0.0)
    S.eliminate_zeros()
    d = np.asarray(S.sum(1)).ravel() + 0.5
    return CsrMatrix.from_scipy((sp.diags(d) - S).tocsr())


@pytest.mark.parametrize("n,half,launches", [(300, 2, 1), (1000, 10, 2), (2000, 5, 2), (8000, 10, 2), (16000, 3, 2)])
@pytest.mark.parametrize("pre", ["jacobi", "none"])
def test_scattered_columns(cuda, n, half, launches, pre):
    import cfdrs_b200 as cf
    A = scattered(n, half, seed=n)
    b = np.random.default_rng(1).uniform(-1, 1, n)
    (x1, r1, l1), (x2, r2, l2) = solve_both(cf, A, b, pre, np.zeros(n))
    assert l1 == launches and l2 > 3 * r2.iterations
    assert r1.termination == r2.termination == cf.Termination.CONVERGED
    assert abs(r1.iterations - r2.iterations) <= 1
    # residuals at most RTOL ||b|| each, the smallest eigenvalue at least 0.5
    assert np.linalg.norm(x1 - x2) <= 2 * RTOL * np.linalg.norm(b) / 0.5


@pytest.mark.parametrize("n,offsets", [(16384, (1, 4097)), (12000, (1, 2, 3, 4, 6000))])
def test_stencils_stay(cuda, n, offsets):
    import cfdrs_b200 as cf
    A, _ = banded(n, offsets)
    (_, _, l1), _ = solve_both(cf, A, np.ones(n), "jacobi", np.zeros(n))
    assert l1 == 1
