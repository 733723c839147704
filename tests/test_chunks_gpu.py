"""ChunkedEllpack with tall slices, read by columns first, against numpy in FP64."""
import numpy as np
import pytest
import torch

from helpers import assert_spmv_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", ["float64", "float32"])
@pytest.mark.parametrize("n", [1, 257, 5003])
def test_tall_chunks(n, real):
    """Rows of 1 to 4000 entries: slices hundreds of slots tall, mostly padding."""
    import tnl_b200 as t

    rng = np.random.default_rng(n)
    lens = np.minimum((1 / rng.random(n)).astype(int), 4000)
    lens[0] = 4000
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    row = np.repeat(np.arange(n), lens)
    cols = rng.integers(0, 4001, len(row)).astype(np.int32)
    vals = rng.uniform(-1, 1, len(row)).astype(real).astype(np.float64)
    M = t.SparseMatrix(t.ChunkedEllpack, getattr(torch, real)).assign(rp, cols, vals, 4001)
    M.getColumnIndexes()[::7] = -1  # holes within the rows are padding too
    x = rng.uniform(-1, 1, 4001).astype(real).astype(np.float64)
    out = torch.zeros(n, dtype=getattr(torch, real), device="cuda")
    M.vectorProduct(torch.tensor(x, dtype=out.dtype, device="cuda"), out)
    seg, c, v = M.getSegments(), M.getColumnIndexes().cpu().numpy(), M.getValues().cpu().numpy().astype(np.float64)
    at = seg.getGlobalIndex(row, np.concatenate([np.arange(k) for k in lens]))
    c, v = c[at], v[at]
    prod = np.where(c >= 0, v * x[c], 0.0)
    assert_spmv_close(out.cpu().numpy(), np.bincount(row, prod, minlength=n),
                      np.bincount(row, np.abs(prod), minlength=n), 1e-13 if real == "float64" else 2e-5)
