"""A few long rows in a matrix of short ones (one thread a row, or a few): the
default SpMV stays with the pipelines that have a row staged, and gives their bits
on both sides of the line."""
import time

import numpy as np
import pytest

from test_gpu_direct_spmv import random_csr

pytestmark = pytest.mark.gpu


def spmv_time(torch, d, x, y, fp32, path):
    d.set_path(path, fp32)
    d.spmv(x.data_ptr(), y.data_ptr(), fp32=fp32)
    d.ctx.synchronize()
    best = float("inf")
    for _ in range(5):
        t = time.perf_counter()
        for _ in range(5):
            d.spmv(x.data_ptr(), y.data_ptr(), fp32=fp32)
        d.ctx.synchronize()
        best = min(best, time.perf_counter() - t)
    return best / 5


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("short,longest", [(6, 48), (6, 49), (6, 5000), (6, 20000), (14, 96), (14, 97), (14, 3000),
                                           (30, 192), (30, 193)])
def test_long_rows(cuda, short, longest, fp32):
    from cfdrs_b200.device import DeviceCsr
    torch = cuda
    n = 20000
    lengths = np.full(n, short)
    lengths[[0, n // 2, n - 1]] = longest
    d = DeviceCsr(random_csr(n, n, lengths, seed=longest))
    dt = torch.float32 if fp32 else torch.float64
    x = torch.as_tensor(np.random.default_rng(1).uniform(-1, 1, n), device="cuda").to(dt)
    out, times = {}, {}
    for path in ("auto", "split"):
        y = torch.full((n,), float("nan"), dtype=dt, device="cuda")
        torch.cuda.synchronize()
        times[path] = spmv_time(torch, d, x, y, fp32, path)
        out[path] = y.cpu().numpy()
    d.set_path("auto", fp32)
    np.testing.assert_array_equal(out["auto"], out["split"])
    # one thread reading 20 000 entries from global memory takes many times the staged row's time
    assert times["auto"] <= 3 * times["split"] + 20e-6
