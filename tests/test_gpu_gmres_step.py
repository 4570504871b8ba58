"""The one-cluster Arnoldi step (FP64 and FP32, rows from fewer than the
cluster's CTAs to the last size it takes, bases past one pull of the shares)
against the step of separate kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-10


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("n,diag,restart", [
    (5, 2.2, 8), (31, 2.2, 8), (513, 2.2, 16), (1000, 2.02, 256), (4099, 2.2, 64), (16384, 2.2, 32), (16385, 2.2, 32),
])
def test_step_matches_separate_kernels(cuda, n, diag, restart, fp32):
    import cfdrs_b200 as cf
    from cfdrs_b200.device import context
    from helpers import tridiag
    A = tridiag(n, -1.0, diag, -1.0)
    b = np.random.default_rng(n).uniform(-1, 1, n)
    npr = n // 3
    pre = cf.BlockDiagonalPreconditioner(A, n - npr, npr)
    prec = cf.Precision.FP32_REFINE if fp32 else cf.Precision.FP64
    ctx, out = context(), []
    try:
        for on in (True, False):
            ctx.set_cluster_solve(on)
            x = np.zeros(n)
            rep = cf.gmres_preconditioned(A, b, pre, x, cf.IterativeSolverConfig(0.0, RTOL, 5000), restart=restart,
                                          precision=prec)
            assert rep.termination == cf.Termination.CONVERGED
            out.append((x, rep, ctx.kernel_stats()["launches"]))
    finally:
        ctx.set_cluster_solve(True)
    (x1, r1, l1), (x2, r2, l2) = out
    assert l1 < 0.7 * l2 if n <= 16384 else l1 > 0.9 * l2, (l1, l2)
    # both residuals are at most RTOL ||b|| and kappa is below (diag + 2) / (diag - 2)
    kappa = (diag + 2) / (diag - 2)
    assert np.linalg.norm(x1 - x2) <= 2 * kappa * RTOL * np.linalg.norm(x2)
    assert abs(r1.iterations - r2.iterations) <= (0.1 * r2.iterations + 2 if fp32 else 1)
