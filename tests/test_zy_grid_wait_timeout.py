"""The grid CG's bounded wait without a GPU fault: on directions that no CTA has
published every CTA's wait runs out, the call reports CFD_ERR_TIMEOUT, and the
context solves on the same kernel afterwards."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_grid_wait_runs_out_and_context_stays_usable(cuda):
    import cfdrs_b200 as cf
    from cfdrs_b200 import _lib
    from cfdrs_b200 import problems as P
    from cfdrs_b200.device import context
    ctx = context(0)
    L = _lib.load()
    for tries in (1, 1000):
        assert L.cfd_selftest_grid_wait_timeout(ctx.h, tries) == 4  # CFD_ERR_TIMEOUT
        assert b"bounded wait ran out" in L.cfd_last_error()
    A, b = P.poisson_2d_dirichlet(260, 250, seed=1)
    x = np.zeros_like(b)
    rep = cf.cg(A, b, x, cf.IterativeSolverConfig(0.0, 1e-8, 5000))
    assert rep.termination == cf.Termination.CONVERGED
    assert np.linalg.norm(A.to_scipy() @ x - b) <= 1e-7 * np.linalg.norm(b)
    assert L.cfd_selftest_grid_wait_timeout(ctx.h, 0) == 2  # CFD_ERR_CONFIG: no wait at all
