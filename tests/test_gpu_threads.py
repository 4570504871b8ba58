"""Solves from two threads with a context each. The whole-solve kernels and the
dense inverse are shared by all contexts of the process: solves of different
sizes must not take each other's launch limits away, and give what they give alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def in_threads(jobs):
    """Runs the jobs side by side; the first exception of any is raised here."""
    errors = []

    def guard(job):
        try:
            job()
        except Exception as e:  # noqa: BLE001 (raised below)
            errors.append(e)
    threads = [threading.Thread(target=guard, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def repeated(ctx, A, b, solve, more):
    """Solves on a context of their own while more(count) holds, each the bits of the first."""
    from cfdrs_b200.device import DeviceCsr
    d = DeviceCsr(A, ctx)
    first, count = None, 0
    while more(count):
        x = np.zeros_like(b)
        solve(d, b, x)
        first = x if first is None else first
        np.testing.assert_array_equal(x, first)
        count += 1


@pytest.mark.parametrize("solver,small,large,count", [
    ("gmres", (9, 8), (70, 61), 4000), ("cg", (9, 8), (200, 170), 4000), ("cg", (230, 240), (600, 500), 2000),
])
def test_two_contexts(cuda, solver, small, large, count):
    """A small system again and again beside `count` solves of a large one, which
    needs more shared memory than a kernel has without asking (a budget of one
    iteration: what may go wrong is the launch)."""
    import cfdrs_b200 as cf
    from cfdrs_b200 import problems as P
    from cfdrs_b200.device import Context
    cfg = cf.IterativeSolverConfig(0.0, 1e-8, 1)
    solve = {"gmres": lambda d, b, x: cf.gmres(d, b, x, cfg), "cg": lambda d, b, x: cf.cg(d, b, x, cfg)}[solver]
    done = threading.Event()

    def beside():
        try:
            repeated(Context(0), *P.poisson_2d_dirichlet(*large, seed=1), solve, lambda k: k < count)
        finally:
            done.set()
    in_threads([beside, lambda: repeated(Context(0), *P.poisson_2d_dirichlet(*small, seed=1), solve,
                                         lambda k: k == 0 or not done.is_set())])


def test_two_contexts_dense_inverse(cuda):
    import cfdrs_b200 as cf
    from cfdrs_b200 import problems as P
    from cfdrs_b200.device import Context
    cfg = cf.AMGConfig(max_levels=1, coarse_solve=cf.CoarseSolve.DENSE)
    contexts = [Context(0) for _ in range(2)]

    def job(ctx, nx, ny):
        A, b = P.poisson_2d_dirichlet(nx, ny, seed=1)
        amg = cf.AlgebraicMultigrid(A, cfg, ctx=ctx)
        want = amg.apply_to(b)
        for _ in range(30):
            amg.recompute(A)
            np.testing.assert_array_equal(amg.apply_to(b), want)
    in_threads([lambda: job(contexts[0], 14, 13), lambda: job(contexts[1], 24, 25)])
