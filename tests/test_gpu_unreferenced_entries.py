"""A vector entry that no row has a column for stays out of every row: a dead cell
(an empty row and column) whose initial guess is NaN leaves the solution of the
other cells alone, in each kernel that reads rows in padded batches (the cluster
and grid CG, the cluster GMRES, both batched Krylov kernels). The dead cell is
row 0, and the first rows of the other blocks of a split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RTOL = 1e-10


def dead_cells(n, offset, dead):
    """Diagonal 4.5, off-diagonals -1 at distances 1 and offset; the dead rows and columns empty."""
    import scipy.sparse as sp
    from cfdrs_b200.sparse import CsrMatrix
    A = sum(sp.diags([-np.ones(n - o), -np.ones(n - o)], [-o, o], shape=(n, n)) for o in (1, offset))
    A = (A + 4.5 * sp.identity(n)).tocsr()
    keep = np.ones(n)
    keep[dead] = 0.0
    A = sp.diags(keep) @ A @ sp.diags(keep)
    A = A.tocsr()
    A.eliminate_zeros()
    b = np.random.default_rng(n).uniform(-1, 1, n) * keep
    x0 = np.where(keep > 0, 0.0, np.nan)
    return CsrMatrix.from_scipy(A), b, x0, keep > 0


def check(A, b, x, live):
    assert np.all(np.isnan(x[~live]))
    S = A.to_scipy()
    r = S[live][:, live] @ x[live] - b[live]
    # the recurrence's residual is at RTOL; the true one is off by rounding, kappa <= 8.5 / 0.5
    assert np.linalg.norm(r) <= 2 * RTOL * np.linalg.norm(b)


@pytest.mark.parametrize("n,blocks", [(500, 2), (16384, 16), (40000, 16), (70000, 148), (300001, 148)])
@pytest.mark.parametrize("pre", ["jacobi", "none"])
def test_cg(cuda, n, blocks, pre):
    import cfdrs_b200 as cf
    rows = -(-n // blocks)
    A, b, x, live = dead_cells(n, 90, np.arange(0, n, rows))
    cfg = cf.IterativeSolverConfig(0.0, RTOL, 500)
    rep = (cf.cg_preconditioned(A, b, cf.JacobiPreconditioner(A), x, cfg) if pre == "jacobi" else cf.cg(A, b, x, cfg))
    assert rep.termination == cf.Termination.CONVERGED
    check(A, b, x, live)


@pytest.mark.parametrize("n,blocks", [(500, 8), (3000, 16), (40000, 16)])
@pytest.mark.parametrize("pre", ["jacobi", "none"])
def test_gmres(cuda, n, blocks, pre):
    import cfdrs_b200 as cf
    rows = -(-n // blocks)
    A, b, x, live = dead_cells(n, 90, np.arange(0, n, rows))
    cfg = cf.IterativeSolverConfig(0.0, RTOL, 500)
    rep = (cf.gmres_preconditioned(A, b, cf.JacobiPreconditioner(A), x, cfg) if pre == "jacobi"
           else cf.gmres(A, b, x, cfg))
    assert rep.termination == cf.Termination.CONVERGED
    check(A, b, x, live)


@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
@pytest.mark.parametrize("form", ["jacobi_cg", "cg", "bicgstab"])
def test_batch(cuda, form, precision):
    import cfdrs_b200 as cf
    from cfdrs_b200.batch import LS_BICGSTAB, LS_CG, LS_PATHS, NetworkBatch
    prec = cf.Precision.FP64 if precision == "fp64" else cf.Precision.FP32_REFINE
    parts = [dead_cells(n, 7, [0]) for n in (300, 1000, 1600)]
    nb = NetworkBatch([p[0] for p in parts])
    b, x0 = (np.concatenate([p[k] for p in parts]) for k in (1, 2))
    if form == "jacobi_cg":
        x, rep = nb.solve(b, x0, config=cf.IterativeSolverConfig(0.0, RTOL, 500), precision=prec)
        assert np.all(rep.termination == int(cf.Termination.CONVERGED))
    else:
        x, rep = nb.solve_linear_systems(b, x0, tolerance=RTOL, method=LS_CG if form == "cg" else LS_BICGSTAB,
                                         precision=prec)
        assert all(LS_PATHS[p] == "krylov" for p in rep.path)
    for (A, bs, _, live), xs in zip(parts, nb.split(x)):
        assert np.all(np.isnan(xs[~live]))
        # row-equilibrated residuals at RTOL (relative or absolute), rows of at most 4.5: 4.5 RTOL, doubled for rounding
        r = A.to_scipy()[live][:, live] @ xs[live] - bs[live]
        assert np.linalg.norm(r) <= 2 * 4.5 * RTOL * max(1.0, np.linalg.norm(bs))
