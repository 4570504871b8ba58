"""A batch makes a system's elimination plan when it first solves it directly: a
batch whose larger systems fall back only later, some of them at a time, ends with
the bits of one that solved all of them directly at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [0, 40])  # beside 40 further systems the new plans' slots go up one by one
def test_plans_made_in_steps(cuda, more):
    from cfdrs_b200 import problems as P
    from cfdrs_b200.batch import LS_CG, LS_PATHS, NetworkBatch
    rng = np.random.default_rng(5)
    systems = [P.random_network(n, rng) for n in (20, 100, 256, 257, 300, 700, 1500, 280) + (30,) * more]
    mats, b = [A for A, _ in systems], np.concatenate([q for _, q in systems])
    whole = NetworkBatch(mats)
    steps = NetworkBatch(mats)
    # one CG iteration: every system beyond 256 rows falls back
    want, rep = whole.solve_linear_systems(b, tolerance=1e-10, max_iterations=1, method=LS_CG)
    assert [LS_PATHS[p] for p in rep.path] == ["direct"] * 3 + ["krylov_fallback"] * 5 + ["direct"] * more
    # at the solution the Krylov solves end at once, and only the small systems are solved directly
    guess = want.copy()
    x, rep = steps.solve_linear_systems(b, guess, tolerance=1e-6, max_iterations=1, method=LS_CG)
    assert [LS_PATHS[p] for p in rep.path] == ["direct"] * 3 + ["krylov"] * 5 + ["direct"] * more
    # two of the others moved off their solutions, then all
    for k in (4, 6):
        guess[steps.sys_row[k]:steps.sys_row[k + 1]] = 0.0
    x, rep = steps.solve_linear_systems(b, guess, tolerance=1e-6, max_iterations=1, method=LS_CG)
    assert [LS_PATHS[p] for p in rep.path[3:8]] == ["krylov", "krylov_fallback", "krylov", "krylov_fallback", "krylov"]
    for k in (0, 1, 2, 4, 6):
        np.testing.assert_array_equal(steps.split(x)[k], whole.split(want)[k])
    x, rep = steps.solve_linear_systems(b, tolerance=1e-10, max_iterations=1, method=LS_CG)
    np.testing.assert_array_equal(x, want)
