"""The pipelined ILU triangular solves against the oracle, bit for bit.

Sizes where the pipeline's parts can go wrong: one row, a step of exactly
256 rows and one more, several parts, entries older than the shared-memory
ring (offset 9000 against 4096 entries) and eight entries a row.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _banded(n, offsets, seed):
    """Diagonally dominant, entries at +-offsets kept with probability 0.8."""
    from tnl_b200.generators import CSRMatrix

    rng = np.random.default_rng(seed)
    i = np.arange(n)
    r, c = [i], [i]
    for o in offsets:
        for d in (-o, o):
            m = (i + d >= 0) & (i + d < n) & (rng.random(n) < 0.8)
            r.append(i[m])
            c.append(i[m] + d)
    r, c = np.concatenate(r), np.concatenate(c)
    order = np.lexsort((c, r))
    r, c = r[order], c[order]
    v = rng.uniform(-1, 1, len(r))
    v[r == c] = 4.0 + 2.0 * len(offsets)
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(r, minlength=n), out=rp[1:])
    return CSRMatrix(rp, c.astype(np.int32), v, n)


@pytest.mark.parametrize("n,offsets", [(1, ()), (256, (1,)), (257, (16,)), (4099, (64, 257)), (30000, (150, 151)),
                                       (30000, (1, 150, 4000, 9000)), (45011, (300, 301, 302, 303)),
                                       (20021, (1, 2, 3, 4, 200, 201, 202, 203))])
def test_pipelined_ilu0_apply_bit_exact(oracle, n, offsets):
    import tnl_b200 as t
    from tnl_b200 import generators as g

    A = _banded(n, offsets, n + len(offsets))
    b = g.uniform_vector(n, 3)
    M = t.SparseMatrix(t.CSR, torch.float64).assign(A.rowptr, A.cols, A.vals)
    P = t.ILU0()
    P.update(M)
    bs = torch.tensor(b, device="cuda")
    want = oracle.prec_apply(A, 2, b)
    for _ in range(2):  # the progress words are reset by every application
        x = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
        P.solve(bs, x)
        assert np.array_equal(x.cpu().numpy(), want)
    P.solve(bs, bs)  # in place
    assert np.array_equal(bs.cpu().numpy(), want)


def test_pipelined_ilu0_apply_fp32():
    """FP32 against the same operations in numpy, rounded after each."""
    import tnl_b200 as t
    from tnl_b200 import generators as g

    A = _banded(6007, (1, 77), 5)
    b = g.uniform_vector(A.n, 3).astype(np.float32)
    M = t.SparseMatrix(t.CSR, torch.float32).assign(A.rowptr, A.cols, A.vals)
    P = t.ILU0()
    P.update(M)
    rp, cols, lu = P.factors()
    x = b.copy()
    for i in range(A.n):
        for k in range(rp[i], rp[i + 1]):
            if cols[k] < i:
                x[i] = np.float32(x[i] - np.float32(lu[k] * x[cols[k]]))
    for i in range(A.n - 1, -1, -1):
        for k in range(rp[i], rp[i + 1]):
            if cols[k] > i:
                x[i] = np.float32(x[i] - np.float32(lu[k] * x[cols[k]]))
        x[i] = np.float32(x[i] / lu[rp[i] + np.searchsorted(cols[rp[i]:rp[i + 1]], i)])
    xs = torch.empty(A.n, dtype=torch.float32, device="cuda")
    P.solve(torch.tensor(b, device="cuda"), xs)
    assert np.array_equal(xs.cpu().numpy(), x)
