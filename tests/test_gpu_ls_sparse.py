"""Direct solves of the 1-D cascade by sparse elimination, against numpy's dense
LU, over the patterns that decide a plan: paths, stars, trees with loops,
grids, one-sided couplings, isolated nodes, missing diagonals, repeated entries,
nearly full matrices (no plan) and matrices that need row exchanges (the guard).

Tolerance: both solve in FP64; the difference is bounded by a modest multiple of
kappa eps (64 n^1/2 for the elimination's growth and the residual's rounding).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def from_entries(n, entries):
    """CsrMatrix of (i, j, v) entries in the given order within each row, repeats kept."""
    from cfdrs_b200.sparse import CsrMatrix
    rows = [[] for _ in range(n)]
    for i, j, v in entries:
        rows[i].append((j, v))
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    col = np.array([j for r in rows for j, _ in r], dtype=np.int32)
    val = np.array([v for r in rows for _, v in r], dtype=np.float64)
    return CsrMatrix(rp, col, val, (n, n))


def laplacian(n, edges, rng, shift=1e-3):
    d = np.full(n, shift)
    ent = []
    for i, j in edges:
        if i == j:
            continue
        g = rng.uniform(0.1, 1.0)
        d[i] += g
        d[j] += g
        ent += [(i, j, -g), (j, i, -g)]
    return ent, d


def cases(rng):
    for n in (1, 2, 3, 64, 255, 256, 257, 700, 2000):
        tree = [(i, int(rng.integers(0, i))) for i in range(1, n)]
        loops = [tuple(int(q) for q in rng.integers(0, n, 2)) for _ in range(n // 10)]
        ent, d = laplacian(n, tree + loops, rng)
        yield f"loops{n}", n, ent + [(i, i, d[i]) for i in range(n)]
    for n in (300, 2048):
        ent, d = laplacian(n, [(i, i - 1) for i in range(1, n)], rng)
        yield f"path{n}", n, ent + [(i, i, d[i]) for i in range(n)]
        ent, d = laplacian(n, [(i, 0) for i in range(1, n)], rng)
        yield f"star{n}", n, ent + [(i, i, d[i]) for i in range(n)]
    n = 400  # a grid: a large core
    ent, d = laplacian(n, [(i, i - 1) for i in range(n) if i % 20] + [(i, i - 20) for i in range(20, n)], rng)
    yield "grid", n, ent + [(i, i, d[i]) for i in range(n)]
    yield "isolated", 300, [(i, i, 1.0 + i) for i in range(300)]
    n = 350  # couplings on one side of the diagonal only
    yield "one_sided", n, [(i, int(rng.integers(0, i)), -0.4) for i in range(1, n)] + [(i, i, 1.0) for i in range(n)]
    n = 310  # the diagonal in three parts, off-diagonals in two
    ent, d = laplacian(n, [(i, int(rng.integers(0, i))) for i in range(1, n)], rng)
    half = [(i, j, v / 2) for i, j, v in ent]
    yield "repeats", n, half + [(i, i, d[i] / 4) for i in range(n)] + half + [(i, i, 3 * d[i] / 8) for i in range(n)] * 2
    n = 270  # rows that need exchanges: a dominant off-diagonal pair, no diagonal on some
    ent, d = laplacian(n, [(i, i - 1) for i in range(1, n)], rng)
    swap = {10: 11, 11: 10, 100: 101, 101: 100}
    yield "exchanges", n, ent + [(i, swap.get(i, i), 50.0 + d[i]) for i in range(n)]
    n = 60
    yield "dense", n, [(i, j, 4.0 * n if i == j else rng.uniform(-1, 1)) for i in range(n) for j in range(n)]


def test_direct_solves_match_dense_lu(cuda):
    from cfdrs_b200.batch import LS_BICGSTAB, LS_PATHS, NetworkBatch
    rng = np.random.default_rng(3)
    names, mats, dense, rhs = [], [], [], []
    for name, n, ent in cases(rng):
        A = from_entries(n, ent)
        D = np.zeros((n, n))
        for i, j, v in ent:
            D[i, j] += v
        names.append(name)
        mats.append(A)
        dense.append(D)
        rhs.append(rng.uniform(-1, 1, n))
    nb = NetworkBatch(mats)
    # one Krylov step at most: every system beyond 256 rows takes the fallback
    x, rep = nb.solve_linear_systems(np.concatenate(rhs), tolerance=1e-10, max_iterations=1, method=LS_BICGSTAB)
    x2, _ = nb.solve_linear_systems(np.concatenate(rhs), tolerance=1e-10, max_iterations=1, method=LS_BICGSTAB)
    np.testing.assert_array_equal(x, x2)  # independent of scheduling
    for name, D, b, xs, p in zip(names, dense, rhs, nb.split(x), rep.path):
        n = len(b)
        assert LS_PATHS[p] in (("direct",) if n <= 256 else ("krylov_fallback", "krylov")), (name, LS_PATHS[p])
        want = np.linalg.solve(D, b)
        bound = 64 * np.sqrt(n) * np.linalg.cond(D) * np.finfo(float).eps
        assert np.linalg.norm(xs - want) <= bound * np.linalg.norm(want), name
    # new values on the kept plans
    nb.update_values(np.concatenate([2.0 * A.val for A in mats]))
    x3, _ = nb.solve_linear_systems(np.concatenate(rhs), tolerance=1e-10, max_iterations=1, method=LS_BICGSTAB)
    for name, D, xs, x0 in zip(names, dense, nb.split(x3), nb.split(x)):
        n = len(x0)
        bound = 64 * np.sqrt(n) * np.linalg.cond(D) * np.finfo(float).eps
        assert np.linalg.norm(2.0 * xs - x0) <= 2 * bound * np.linalg.norm(x0), name


def test_singular_system_fails_alone(cuda):
    from cfdrs_b200.batch import LS_BICGSTAB, LS_PATHS, NetworkBatch
    rng = np.random.default_rng(4)
    ent, d = laplacian(300, [(i, i - 1) for i in range(1, 300)], rng)
    good = from_entries(300, ent + [(i, i, d[i]) for i in range(300)])
    bad = from_entries(300, [(i, i, 1.0 if i != 7 else 0.0) for i in range(300)])
    nb = NetworkBatch([good, bad])
    x, rep = nb.solve_linear_systems(np.ones(600), tolerance=1e-10, max_iterations=1, method=LS_BICGSTAB)
    assert LS_PATHS[rep.path[0]] == "krylov_fallback" and LS_PATHS[rep.path[1]] == "failed"
    assert np.all(np.isfinite(nb.split(x)[0]))


@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
@pytest.mark.parametrize("method", ["detect", "cg"])
def test_krylov_rows_in_registers_match_shared_memory_vectors(cuda, precision, method):
    """The register form of the Krylov kernel (at most 8 rows a thread, 256
    threads) forms every sum in the order of the shared-memory form: with the same
    width in both buckets the outcome is the same bits, whichever form the wider
    bucket's row count selects."""
    import cfdrs_b200 as cf
    from cfdrs_b200 import problems as P
    from cfdrs_b200.batch import LS_CG, LS_DETECT, NetworkBatch
    rng = np.random.default_rng(9)
    prec = cf.Precision.FP64 if precision == "fp64" else cf.Precision.FP32_REFINE
    meth = LS_DETECT if method == "detect" else LS_CG
    small = [P.random_network(n, rng) for n in (257, 300, 511, 512)]
    got = []
    for extra in (None, 513):  # 64 threads: 512 rows are 8 a thread, 513 are 9 (shared memory)
        systems = small + ([P.random_network(extra, np.random.default_rng(1))] if extra else [])
        nb = NetworkBatch([A for A, _ in systems])
        nb.set_config([32, 64, 64, 256], [1, 1, 1, 1], prec)
        x, rep = nb.solve_linear_systems(np.concatenate([b for _, b in systems]), tolerance=1e-10, method=meth,
                                         precision=prec)
        rows = sum(A.nrows for A, _ in small)
        got.append((x[:rows], rep.iterations[:4], rep.termination[:4], rep.path[:4]))
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
