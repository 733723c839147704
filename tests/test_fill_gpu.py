"""The fill of CSR, Ellpack and SlicedEllpack storage, every slot of it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", ["float64", "float32"])
@pytest.mark.parametrize("org", [0, 1])
@pytest.mark.parametrize("fmt", ["CSR", "AdaptiveCSR", "Ellpack", "SlicedEllpack"])
@pytest.mark.parametrize("n", [1, 32, 33, 1000])
def test_fill_writes_every_slot(n, fmt, org, real):
    """Rows of 0 to 70 entries, some dropped: what is kept comes first, in
    order, and every other slot is padding."""
    import tnl_b200 as t

    rng = np.random.default_rng(n)
    lens = rng.integers(0, 24, n)
    lens[n // 2] = 69
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    row = np.repeat(np.arange(n), lens)
    cols = rng.integers(0, 500, len(row)).astype(np.int32)
    vals = rng.uniform(-1, 1, len(row))
    vals[::17] = 0.0
    vals = vals.astype(real)
    cols[::13] = -1
    M = t.SparseMatrix(t.FORMATS[fmt], getattr(torch, real), org)
    for _ in range(2):  # the second on memory that holds the first's entries
        M.assign(rp, cols, vals, 500)
        seg = M.getSegments()
        c, v = M.getColumnIndexes().cpu().numpy(), M.getValues().cpu().numpy()
        want_c, want_v = np.full(len(c), -1, np.int32), np.zeros(len(c), vals.dtype)
        keep = (vals != 0) & (cols != -1)
        r = row[keep]
        local = np.arange(len(r)) - np.searchsorted(r, r)
        at = seg.getGlobalIndex(r, local)
        want_c[at], want_v[at] = cols[keep], vals[keep]
        assert np.array_equal(c, want_c) and np.array_equal(v, want_v)


def test_failed_fill_leaves_padding(monkeypatch):
    """A fill that fails leaves a matrix without elements, whatever the memory
    held before."""
    import tnl_b200 as t

    rp = np.arange(0, 3 * 1001, 3, dtype=np.int32)
    cols, vals = np.tile(np.arange(3, dtype=np.int32), 1000), np.ones(3000)
    held = [torch.full((3072,), 7, dtype=torch.int32, device="cuda") for _ in range(8)]
    held += [torch.full((3072,), 7.0, dtype=torch.float64, device="cuda") for _ in range(8)]
    del held
    M = t.SparseMatrix(t.SlicedEllpack, torch.float64)
    monkeypatch.setattr(t.capi, "tnlb_matrix_fill_from_csr", lambda *a: t.capi.ERR_INVALID_ARGUMENT)
    with pytest.raises(ValueError):
        M.assign(rp, cols, vals, 3)
    assert M.getColumnIndexes().numel() == 3072
    assert (M.getColumnIndexes() == -1).all() and (M.getValues() == 0).all()
