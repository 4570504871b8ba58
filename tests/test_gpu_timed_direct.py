"""CFD_PATH_TIMED on an operator whose default is the direct kernel times that kernel
too, and may keep it."""
import numpy as np
import pytest

from kernel_names import kernel_names
from test_gpu_direct_spmv import random_csr

pytestmark = pytest.mark.gpu


def kernels(torch, d, x, y, fp32):
    def call():
        d.spmv(x.data_ptr(), y.data_ptr(), fp32=fp32)
        d.ctx.synchronize()
    return kernel_names(torch, call)[0]


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("n,length", [(3000, 24), (1000, 6)])
def test_timed_may_be_the_direct_kernel(cuda, n, length, fp32):
    from cfdrs_b200.device import DeviceCsr
    torch = cuda
    A = random_csr(n, n, np.full(n, length), seed=1)
    d = DeviceCsr(A)
    dt = torch.float32 if fp32 else torch.float64
    x = torch.as_tensor(np.random.default_rng(2).uniform(-1, 1, n), device="cuda").to(dt)
    y = torch.zeros(n, dtype=dt, device="cuda")
    torch.cuda.synchronize()
    d.spmv(x.data_ptr(), y.data_ptr(), fp32=fp32)
    d.ctx.synchronize()
    want = y.clone()
    assert "k_spmv_direct" in kernels(torch, d, x, y, fp32)
    # a timing of launches of a few microseconds may go wrong once, not five times
    for _ in range(5):
        d.set_path("timed", fp32)
        d.spmv(x.data_ptr(), y.data_ptr(), fp32=fp32)
        d.ctx.synchronize()
        # the columns are random: nothing is staged or coded, so the split pipeline is the only other choice
        assert d.layout()["all_compressed"] == 0 and d.layout()["path_f32" if fp32 else "path_f64"] == 0
        ran = kernels(torch, d, x, y, fp32)
        if "k_spmv_direct" in ran:
            break
    assert "k_spmv_direct" in ran
    assert torch.equal(y, want)
    d.set_path("split", fp32)
    assert "k_spmv_direct" not in kernels(torch, d, x, y, fp32)
