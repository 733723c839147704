"""Products that keep a window of x or y in shared memory, against numpy in
FP64.

Matrices at the rules' edges: columns inside the window, half outside, all
over the place (the window is not taken), some runs of rows one way and some
the other, fewer and more columns than rows, and a last block and slice that
are not full.  Bounds per row: 1e-13 (FP64)
and 2e-5 (FP32) times the sum of the magnitudes that enter it, the repository's
rule for a reordered sum.
"""
import numpy as np
import pytest
import torch

from helpers import assert_spmv_close

pytestmark = pytest.mark.gpu

SHAPES = {  # rows, columns, half band (None: anywhere)
    # clipped columns: the first and the last one are shared by thousands of rows
    "narrow": (310007, 310007, 400), "wide": (310007, 310007, 20000), "anywhere": (310007, 310007, None),
    "few_columns": (310007, 200003, 5000), "many_columns": (310007, 400009, 5000),
    "mixed": (310007, 310007, "mixed"),  # first half of the rows in a band, the others anywhere
}


def _matrix(rows, columns, half, longest, seed, triangle=False):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, longest + 1, rows)
    lens[rows // 2] = longest + 20
    rp = np.zeros(rows + 1, np.int32)
    np.cumsum(lens, out=rp[1:])
    row = np.repeat(np.arange(rows), lens)
    if half is None:
        cols = rng.integers(0, columns, len(row))
    elif half == "mixed":
        cols = np.where(row < rows // 2, np.clip(row + rng.integers(-400, 401, len(row)), 0, columns - 1),
                        rng.integers(0, columns, len(row)))
    else:
        cols = np.clip(row + rng.integers(-half, half + 1, len(row)), 0, columns - 1)
    if triangle:
        cols = np.minimum(cols, row)
    vals = rng.uniform(-1, 1, len(row))
    vals[rng.random(len(row)) < 0.01] = 0.0  # dropped by the fill
    return rp, cols.astype(np.int32), vals, row


def _close(y, want, scale, real):
    assert_spmv_close(y.cpu().numpy(), want, scale, 1e-13 if real == "float64" else 2e-5)


def _vectors(real, columns, rows):
    rng = np.random.default_rng(5)
    return (rng.uniform(-1, 1, n).astype(real).astype(np.float64) for n in (columns, rows))


@pytest.mark.parametrize("real", ["float64", "float32"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("fmt", ["SlicedEllpack", "CSR"])
def test_products_of_long_rows(fmt, shape, real):
    import tnl_b200 as t

    rows, columns, half = SHAPES[shape]
    rp, cols, vals, row = _matrix(rows, columns, half, 40, 3)
    vals = vals.astype(real).astype(np.float64)
    M = t.SparseMatrix(t.FORMATS[fmt], getattr(torch, real)).assign(rp, cols, vals, columns)
    x, y0 = _vectors(real, columns, rows)
    xs, ys = (torch.tensor(v, dtype=getattr(torch, real), device="cuda") for v in (x, y0))
    out = ys.clone()
    M.vectorProduct(xs, out, -1.5, 0.5)
    prod = vals * x[cols]
    want = 0.5 * y0 - 1.5 * np.bincount(row, prod, minlength=rows)
    scale = np.abs(0.5 * y0) + 1.5 * np.bincount(row, np.abs(prod), minlength=rows)
    _close(out, want, scale, real)
    # transposed, into a part of the columns
    out = xs.clone()
    first, last = columns // 7, columns - 11
    M.transposedVectorProduct(ys, out, 2.0, 0.5, first, last)
    prod = vals * y0[row]
    inside = (np.arange(columns) >= first) & (np.arange(columns) < last)
    want = 0.5 * x + 2.0 * np.where(inside, np.bincount(cols, prod, minlength=columns), 0.0)
    scale = np.abs(0.5 * x) + 2.0 * np.bincount(cols, np.abs(prod), minlength=columns)
    _close(out, want, scale, real)


@pytest.mark.parametrize("real", ["float64", "float32"])
@pytest.mark.parametrize("half,longest", [(300, 3), (300, 20), (9000, 24), (None, 20)])
@pytest.mark.parametrize("fmt", ["SlicedEllpack", "CSR", "Ellpack"])
def test_symmetric_product(fmt, half, longest, real):
    import tnl_b200 as t

    n = 130001
    rp, cols, vals, row = _matrix(n, n, half, longest, 4, triangle=True)
    vals = vals.astype(real).astype(np.float64)
    M = t.SparseMatrix(t.FORMATS[fmt], getattr(torch, real), symmetric=True).assign(rp, cols, vals, n)
    x, y0 = _vectors(real, n, n)
    xs, out = (torch.tensor(v, dtype=getattr(torch, real), device="cuda") for v in (x, y0))
    M.vectorProduct(xs, out, 1.5, -1.0)
    low = cols < row
    want, scale = -y0, np.abs(y0)
    for r, c, v in ((row, cols, vals), (cols[low], row[low], vals[low])):
        want = want + 1.5 * np.bincount(r, v * x[c], minlength=n)
        scale = scale + 1.5 * np.bincount(r, np.abs(v * x[c]), minlength=n)
    _close(out, want, scale, real)


@pytest.mark.parametrize("shape", ["narrow", "mixed", "anywhere"])
def test_window_product_in_a_graph(shape):
    """Captured, where the two kernels of a product follow one another, and replayed."""
    import tnl_b200 as t

    rows, columns, half = SHAPES[shape]
    rp, cols, vals, _ = _matrix(rows, columns, half, 40, 3)
    M = t.SparseMatrix(t.SlicedEllpack, torch.float64).assign(rp, cols, vals, columns)
    x, y0 = (torch.tensor(v, device="cuda") for v in _vectors("float64", columns, rows))
    want, out = y0.clone(), y0.clone()
    M.vectorProduct(x, want, -1.5, 0.5)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        M.vectorProduct(x, out, -1.5, 0.5, synchronize=False)
    out.copy_(y0)
    graph.replay()
    assert torch.equal(out, want)
