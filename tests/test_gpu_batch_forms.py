"""The register form of the batched Jacobi-PCG kernel at every count of rows a thread
it is made for (1, 2, 4, 8) against the shared-memory form at the same threads a
system: the same bits, iterations and terminations. The shared-memory form is
taken by a CTA of more than 512 threads, or by a bucket with more than eight rows
a thread; the kernels' names tell which ran."""
import numpy as np
import pytest

from kernel_names import kernel_names

pytestmark = pytest.mark.gpu


def solve(torch, cf, systems, keep, threads, groups, prec):
    from cfdrs_b200.batch import NetworkBatch
    cfg = cf.IterativeSolverConfig(0.0, 1e-10, 20000)
    nb = NetworkBatch([A for A, _ in systems])
    nb.set_config([threads] * 4, [groups] * 4, prec)
    b = np.concatenate([q for _, q in systems])
    names, (x, rep) = kernel_names(torch, lambda: nb.solve(b, config=cfg, precision=prec))
    return x[:nb.sys_row[keep]], rep.iterations[:keep], rep.termination[:keep], names


@pytest.mark.parametrize("precision", ["fp64", "fp32_refine"])
@pytest.mark.parametrize("rows,threads,groups,sizes,extra", [
    (1, 256, 4, (2, 33, 64, 200, 256), None),
    (2, 256, 4, (257, 300, 511, 512), None),
    (2, 512, 2, (520, 700, 1000), None),
    (4, 256, 4, (513, 516, 524), None),
    (8, 64, 1, (257, 300, 511, 512), 513),
])
def test_register_form_is_the_shared_form(cuda, rows, threads, groups, sizes, extra, precision):
    import cfdrs_b200 as cf
    from cfdrs_b200 import problems as P
    prec = cf.Precision.FP64 if precision == "fp64" else cf.Precision.FP32_REFINE
    rng = np.random.default_rng(rows)
    systems = [P.random_network(n, rng) for n in sizes]
    x1, i1, t1, n1 = solve(cuda, cf, systems, len(sizes), threads, 1, prec)
    more = systems + ([P.random_network(extra, rng)] if extra else [])
    x2, i2, t2, n2 = solve(cuda, cf, more, len(sizes), threads, groups, prec)
    T = "float, true" if prec == cf.Precision.FP32_REFINE else "double, false"
    if n1 and n2:  # as far as the profiler reports kernels
        assert f"k_batch_pcg_reg<{T}, {rows}>" in n1 and "k_batch_pcg<" not in n1
        assert f"k_batch_pcg<{T}>" in n2 and "k_batch_pcg_reg" not in n2
    np.testing.assert_array_equal(x1, x2)
    np.testing.assert_array_equal(i1, i2)
    np.testing.assert_array_equal(t1, t2)
