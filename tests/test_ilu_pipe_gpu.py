"""The pipelined ILU triangular solves against the oracle, bit for bit.

Sizes where the pipeline's parts can go wrong: steps of exactly 256 rows and
levels of one row more, several parts, entries older than the shared-memory
ring (offset 9000 against 4096 entries), eight entries a row, and chains of
rows millions long.  (Matrices of a few rows or levels are solved level by
level.)
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _banded(n, offsets, seed, keep=0.8):
    """Diagonally dominant, entries at +-offsets kept with probability `keep`."""
    from tnl_b200.generators import CSRMatrix

    rng = np.random.default_rng(seed)
    i = np.arange(n)
    r, c = [i], [i]
    for o in offsets:
        for d in (-o, o):
            m = (i + d >= 0) & (i + d < n) & (rng.random(n) < keep)
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


def _parts(P):
    """Thread blocks of the pipelines of L and U, 0: level by level."""
    from tnl_b200 import _capi

    parts = np.zeros(2, np.int32)
    _capi.check(_capi.tnlb_precond_ilu_parts(P.handle, parts.ctypes.data))
    return tuple(parts)


@pytest.mark.parametrize("n,offsets,keep,parts", [
    (1, (), 0.8, (0, 0)), (256, (1,), 0.8, None), (257, (16,), 0.8, None), (4099, (64, 257), 0.8, (1, 1)),
    (256 * 41, (256,), 1.0, (1, 1)), (257 * 41, (257,), 1.0, (1, 1)), (30000, (150, 151), 0.8, (1, 1)),
    (30000, (1, 150, 4000, 9000), 0.8, None), (45011, (300, 301, 302, 303), 0.8, None),
    (20021, (1, 2, 3, 4, 200, 201, 202, 203), 0.8, None)])
def test_pipelined_ilu0_apply_bit_exact(oracle, n, offsets, keep, parts):
    import tnl_b200 as t
    from tnl_b200 import generators as g

    A = _banded(n, offsets, n + len(offsets), keep)
    b = g.uniform_vector(n, 3)
    M = t.SparseMatrix(t.CSR, torch.float64).assign(A.rowptr, A.cols, A.vals)
    P = t.ILU0()
    P.update(M)
    assert parts is None or _parts(P) == parts
    bs = torch.tensor(b, device="cuda")
    want = oracle.prec_apply(A, 2, b)
    for _ in range(2):  # the progress words are reset by every application
        x = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
        P.solve(bs, x)
        assert np.array_equal(x.cpu().numpy(), want)
    P.solve(bs, bs)  # in place
    assert np.array_equal(bs.cpu().numpy(), want)


def _coupled(chain, side):
    """A chain of rows, then a 5-point grid whose first row is coupled to the chain's last."""
    from tnl_b200.generators import CSRMatrix

    n = chain + side * side
    i = np.arange(n)
    r, c = [i], [i]
    k = i[1:chain + 1] if side else i[1:chain]
    r += [k, k - 1]
    c += [k - 1, k]
    if side:
        q = i[chain:]
        col = (q - chain) % side
        for o, m in ((1, col < side - 1), (side, q < n - side)):
            r += [q[m], q[m] + o]
            c += [q[m] + o, q[m]]
    r, c = np.concatenate(r), np.concatenate(c)
    order = np.lexsort((c, r))
    r, c = r[order], c[order]
    v = np.random.default_rng(9).uniform(-1, 1, len(r))
    v[r == c] = 6.0
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(r, minlength=n), out=rp[1:])
    return CSRMatrix(rp, c.astype(np.int32), v, n)


@pytest.mark.parametrize("chain,side", [(0, 300), (4000000, 0), (2500000, 1000)])
def test_pipelined_ilu0_chain_and_grid_bit_exact(oracle, chain, side):
    """A grid is several parts, a chain is one; behind a chain, the grid's parts
    wait most of a second for their first values."""
    import tnl_b200 as t
    from tnl_b200 import generators as g

    A = _coupled(chain, side)
    b = g.uniform_vector(A.n, 3)
    M = t.SparseMatrix(t.CSR, torch.float64).assign(A.rowptr, A.cols, A.vals)
    P = t.ILU0()
    P.update(M)
    assert _parts(P) == (1, 1) if side == 0 else min(_parts(P)) > 1
    x = torch.full((A.n,), float("nan"), dtype=torch.float64, device="cuda")
    P.solve(torch.tensor(b, device="cuda"), x)
    assert np.array_equal(x.cpu().numpy(), oracle.prec_apply(A, 2, b))


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


@pytest.mark.parametrize("side", [40, 300])  # level by level or one part, several parts
def test_ilu0_applied_from_two_threads(oracle, side):
    """One preconditioner on two streams at once: each application as if alone."""
    import threading

    import tnl_b200 as t
    from tnl_b200 import generators as g

    A = _coupled(0, side)
    M = t.SparseMatrix(t.CSR, torch.float64).assign(A.rowptr, A.cols, A.vals)
    P = t.ILU0()
    P.update(M)
    b = [g.uniform_vector(A.n, seed) for seed in (3, 4)]
    bs = [torch.tensor(v, device="cuda") for v in b]
    torch.cuda.synchronize()
    out = [[], []]

    def run(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(20):
                x = torch.empty_like(bs[k])
                P.solve(bs[k], x)
                out[k].append(x)

    threads = [threading.Thread(target=run, args=(k,)) for k in (0, 1)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    for k in (0, 1):
        want = oracle.prec_apply(A, 2, b[k])
        assert len(out[k]) == 20 and all(np.array_equal(x.cpu().numpy(), want) for x in out[k])
