"""The direct SpMV kernel (default choice of small operators) against the
bulk-copy pipelines: row results bit for bit, over row lengths around its batch
of eight and its row groups, empty rows, rectangular operators, and the sizes
where it stops being chosen."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def random_csr(nrows, ncols, lengths, seed):
    from cfdrs_b200.sparse import CsrMatrix
    rng = np.random.default_rng(seed)
    rows = [np.sort(rng.choice(ncols, size=min(k, ncols), replace=False)) for k in lengths]
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    col = np.concatenate(rows).astype(np.int32) if rows else np.zeros(0, np.int32)
    return CsrMatrix(rp, col, rng.uniform(-1, 1, len(col)), (nrows, ncols))


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("nrows,ncols,lo,hi", [
    (1, 1, 1, 1), (255, 300, 0, 3), (257, 257, 1, 9), (1000, 5000, 7, 17), (3000, 3000, 20, 40), (700, 4000, 90, 200),
    (4000, 4000, 250, 420), (60000, 60000, 4, 8), (300000, 300000, 3, 6),
])
def test_bit_identical_to_split_pipeline(cuda, nrows, ncols, lo, hi, fp32):
    from cfdrs_b200.device import DeviceCsr
    torch = cuda
    rng = np.random.default_rng(nrows)
    A = random_csr(nrows, ncols, rng.integers(lo, hi + 1, nrows), seed=1)
    d = DeviceCsr(A)
    dt = torch.float32 if fp32 else torch.float64
    x = torch.as_tensor(rng.uniform(-1, 1, ncols), device="cuda").to(dt)
    out = {}
    for path in ("auto", "split"):
        d.set_path(path, fp32)
        y = torch.full((nrows,), float("nan"), dtype=dt, device="cuda")
        torch.cuda.synchronize()
        d.spmv(x.data_ptr(), y.data_ptr(), fp32=fp32)
        d.ctx.synchronize()
        out[path] = y.cpu().numpy()
    np.testing.assert_array_equal(out["auto"], out["split"])
    want = A.to_scipy() @ x.double().cpu().numpy()
    scale = abs(A.to_scipy()) @ np.abs(x.double().cpu().numpy())
    eps = np.finfo(np.float32 if fp32 else np.float64).eps
    assert np.all(np.abs(out["auto"] - want) <= (hi + 2) * eps * scale + 1e-300)
