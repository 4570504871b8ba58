"""The whole-solve CG / Jacobi-PCG cluster launch against the multi-kernel
solve where its row split changes: one to eight rows a thread, blocks that end
inside a warp, rows longer than a register batch, and rows without entries of
their own CTA."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def banded(n, offsets):
    """Symmetric, diagonal 2 k + 0.5 for k off-diagonal pairs of -1: kappa <= (4 k + 0.5) / 0.5."""
    import scipy.sparse as sp
    from cfdrs_b200.sparse import CsrMatrix
    d = [sp.diags([-np.ones(n - o), -np.ones(n - o)], [-o, o], shape=(n, n)) for o in offsets if o < n]
    k = len(d)
    return CsrMatrix.from_scipy((sum(d) + sp.identity(n) * (2 * k + 0.5)).tocsr()), (4 * k + 0.5) / 0.5


@pytest.mark.parametrize("n,offsets", [
    (5, (1,)), (1023, (1, 7)), (1025, (1, 511)), (8192, (1, 90)), (8193, (1, 90)), (16384, (1, 4097)), (16385, (1, 128)),
    (24577, (1, 155)), (32768, (1, 181)), (32770, (1, 2)), (40961, (1,)), (12000, (1, 2, 3, 4, 6000)),
])
@pytest.mark.parametrize("pre", ["jacobi", "none"])
def test_row_splits(cuda, n, offsets, pre):
    import cfdrs_b200 as cf
    from cfdrs_b200.device import device_matrix
    A, kappa = banded(n, offsets)
    b = np.random.default_rng(n).uniform(-1, 1, n)
    ctx = device_matrix(A).ctx
    cfg = cf.IterativeSolverConfig(0.0, RTOL, 2000)
    got = []
    try:
        for cluster in (True, False):
            ctx.set_cluster_solve(cluster)
            x = np.linspace(-1.0, 1.0, n)  # a warm start
            rep = (cf.cg_preconditioned(A, b, cf.JacobiPreconditioner(A), x, cfg) if pre == "jacobi"
                   else cf.cg(A, b, x, cfg))
            got.append((x, rep, ctx.kernel_stats()["launches"]))
    finally:
        ctx.set_cluster_solve(True)
    (x1, r1, l1), (x2, r2, l2) = got
    assert l1 == 1 and l2 > 10
    assert r1.termination == r2.termination == cf.Termination.CONVERGED
    assert abs(r1.iterations - r2.iterations) <= 1
    # residuals at most RTOL ||r0|| each: the solutions differ by at most 2 RTOL ||r0|| / lambda_min
    assert np.linalg.norm(x1 - x2) <= 2 * RTOL * r2.initial_residual_norm / 0.5
