"""GMRES of small systems as one thread-block-cluster launch against the
multi-kernel GMRES: the same step count to one and the same solution, at the
sizes where the row split changes (one CTA, levels run by CTA 0 alone, uneven
blocks, the largest pressure system) and for the V-cycle's options."""
import numpy as np
import pytest

from helpers import tridiag

pytestmark = pytest.mark.gpu

RTOL = 1e-12


def solve_both(cf, A, b, pre, restart=30, budget=4000, rtol=RTOL):
    from cfdrs_b200.device import device_matrix
    ctx = device_matrix(A).ctx
    out = []
    try:
        for cluster in (True, False):
            ctx.set_cluster_solve(cluster)
            x = np.zeros_like(b)
            cfg = cf.IterativeSolverConfig(0.0, rtol, budget)
            rep = (cf.gmres(A, b, x, cfg, restart=restart) if pre is None
                   else cf.gmres_preconditioned(A, b, pre, x, cfg, restart=restart))
            out.append((x, rep, ctx.kernel_stats()["launches"]))
    finally:
        ctx.set_cluster_solve(True)
    return out


def check(cf, A, b, pre, kappa, **kw):
    (x1, r1, l1), (x2, r2, l2) = solve_both(cf, A, b, pre, **kw)
    assert l1 == 1 and l2 > 10
    assert r1.termination == r2.termination == cf.Termination.CONVERGED
    assert abs(r1.iterations - r2.iterations) <= 1
    # both residuals are at most RTOL ||b||, so the solutions differ by at most 2 kappa RTOL
    assert np.linalg.norm(x1 - x2) <= 2 * kappa * RTOL * np.linalg.norm(x2)
    assert abs(r1.initial_residual_norm - r2.initial_residual_norm) <= 1e-13 * r2.initial_residual_norm


def poisson_kappa(nx, ny):
    s = [np.sin(np.pi / (2 * (n + 1))) ** 2 for n in (nx, ny)]
    return (2 - sum(s)) / sum(s)


@pytest.mark.parametrize("nx,ny", [(2, 3), (16, 8), (43, 3), (27, 19), (47, 35), (101, 98)])
def test_pressure_amg_sizes(cuda, nx, ny):
    import cfdrs_b200 as cf
    from cfdrs_b200 import problems as P
    A, b = P.poisson_2d_dirichlet(nx, ny, seed=1)
    check(cf, A, b, cf.AlgebraicMultigrid(A, cf.AMGConfig()), poisson_kappa(nx, ny))


@pytest.mark.parametrize("cfg", [
    dict(pre_smooth_iterations=1, post_smooth_iterations=1, relaxation_factor=2 / 3),
    dict(pre_smooth_iterations=0, post_smooth_iterations=2, relaxation_factor=2 / 3),
    dict(pre_smooth_iterations=3, post_smooth_iterations=0, relaxation_factor=2 / 3, coarse_sweeps=0),
    dict(coarse_sweeps=1), dict(max_levels=1, coarse_sweeps=5, relaxation_factor=2 / 3),
    dict(coarse_solve=1, min_coarse_size=20), dict(coarse_solve=1, min_coarse_size=500),
])
def test_vcycle_options(cuda, cfg):
    import cfdrs_b200 as cf
    from cfdrs_b200 import problems as P
    cfg = dict(cfg)
    if "coarse_solve" in cfg:
        cfg["coarse_solve"] = cf.CoarseSolve(cfg["coarse_solve"])
    A, b = P.poisson_2d_dirichlet(45, 37, seed=2)
    check(cf, A, b, cf.AlgebraicMultigrid(A, cf.AMGConfig(**cfg)), poisson_kappa(45, 37))


@pytest.mark.parametrize("n", [1, 31, 128, 129, 512, 513, 3001])
@pytest.mark.parametrize("pre", ["none", "jacobi"])
def test_plain_sizes(cuda, n, pre):
    import cfdrs_b200 as cf
    A = tridiag(n, lo=-1.3, d=3.0, hi=-0.7)
    b = np.random.default_rng(n).uniform(-1, 1, n)
    (x1, r1, l1), (x2, r2, _) = solve_both(cf, A, b, cf.JacobiPreconditioner(A) if pre == "jacobi" else None, 8)
    assert l1 == 1 and r1.termination == r2.termination and abs(r1.iterations - r2.iterations) <= 1
    # strictly diagonally dominant by 1 with norm at most 5: kappa <= 5
    assert np.linalg.norm(x1 - x2) <= 2 * 5 * RTOL * np.linalg.norm(x2)


def test_budget_over_several_launches(cuda):
    """A solve that cannot converge runs out its budget over bounded launches."""
    import cfdrs_b200 as cf
    n = 2000
    A = tridiag(n, lo=-1.0, d=2.0, hi=-1.0)
    b = np.random.default_rng(0).uniform(-1, 1, n)
    (x1, r1, l1), (x2, r2, _) = solve_both(cf, A, b, None, restart=8, budget=9000)
    assert r1.termination == r2.termination == cf.Termination.MAX_ITERATIONS
    assert r1.iterations == r2.iterations == 9000 and l1 == 3
    assert np.linalg.norm(x1 - x2) <= 1e-6 * np.linalg.norm(x2)
