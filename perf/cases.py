"""The work that a program has this framework do, as measurable cases.

A case is one call, or one short solve, through the public Python API on
matrices of the kinds the framework is used on:

* ``grid``: cell-centred diffusion operators (5-point in 2D, 7-point in 3D)
  with a log-normal coefficient, optionally with a time-step term on the
  diagonal and first-order upwind convection;
* ``powerlaw``: Zipf 1.73 row lengths of 1 to 4096 (mean about 16) with
  uniform columns, as of graphs and networks;
* ``fem``: 9 to 45 entries a row (mean 27) inside a band, as of
  unstructured meshes.

Three kinds of call: products (``vectorProduct`` of every format, general
and symmetric, and ``transposedVectorProduct``), the set-up of a matrix from
CSR arrays (``assign``), and Krylov solves (CG, BiCGStab, GMRES, the
mixed-precision PCG) of a stated number of iterations, as a time step with a
fixed iteration budget makes them; the mixed-precision solve runs to its
tolerance, which is its contract.
"""
from __future__ import annotations

import math

import torch

import tnl_b200 as tnl

REALS = {"f64": torch.float64, "f32": torch.float32}
FORMATS = ("CSR", "AdaptiveCSR", "Ellpack", "SlicedEllpack", "ChunkedEllpack", "BiEllpack")
ZIPF, ZIPF_CAP, FEM_MIN, FEM_MAX = 1.73, 4096, 9, 45


def listed():
    return [
        # A coarse-grid operator in single precision: one launch, nothing but latency.
        {"name": "product_csr_f32_grid_31x33", "call": "product", "matrix": "grid", "shape": "31x33", "sigma": 1.0,
         "format": "CSR", "real": "f32", "residual": False},
        # The 5-point operator of a megapixel grid, the size of the linear-solver benchmark.
        {"name": "product_csr_f64_grid_1024x1024", "call": "product", "matrix": "grid", "shape": "1024x1024",
         "sigma": 1.0, "format": "CSR", "real": "f64", "residual": False},
        # A graph's matrix-vector product at the size of the headline benchmark.
        {"name": "product_csr_f64_powerlaw_4194304", "call": "product", "matrix": "powerlaw", "n": 4194304,
         "format": "CSR", "real": "f64", "residual": False},
        # An unstructured mesh in the GPU format of choice, single precision, as a residual b - A x.
        {"name": "residual_sliced_f32_fem_1000003", "call": "product", "matrix": "fem", "n": 1000003,
         "format": "SlicedEllpack", "real": "f32", "residual": True},
        # Very uneven rows in the format made for them.
        {"name": "product_chunked_f64_powerlaw_700001", "call": "product", "matrix": "powerlaw", "n": 700001,
         "format": "ChunkedEllpack", "real": "f64", "residual": False},
        # A^T x of an unstructured mesh (adjoints, least squares).
        {"name": "transposed_csr_f64_fem_500009", "call": "transposed", "matrix": "fem", "n": 500009,
         "format": "CSR", "real": "f64", "residual": False},
        # Set-up of a matrix from device CSR arrays: capacities, metadata, fill.
        {"name": "assign_sliced_f64_fem_1000003", "call": "assign", "matrix": "fem", "n": 1000003,
         "format": "SlicedEllpack", "real": "f64"},
        # A time step on a small grid: many short iterations.
        {"name": "cg_jacobi_f64_grid_100x100", "call": "cg", "matrix": "grid", "shape": "100x100", "sigma": 1.0,
         "mass": 0.01, "format": "CSR", "real": "f64", "precond": "Diagonal", "iterations": 100},
        # The linear-solver benchmark's CG at its own size.
        {"name": "cg_jacobi_f64_grid_1024x1024", "call": "cg", "matrix": "grid", "shape": "1024x1024", "sigma": 1.0,
         "mass": 0.01, "format": "CSR", "real": "f64", "precond": "Diagonal", "iterations": 200},
        # Convection-diffusion in 3D, odd sides.
        {"name": "bicgstab_jacobi_f64_grid_95x96x97", "call": "bicgstab", "matrix": "grid", "shape": "95x96x97",
         "sigma": 1.0, "mass": 0.05, "velocity": 1.0, "format": "CSR", "real": "f64", "precond": "Diagonal",
         "iterations": 40},
        # GMRES(30) with ILU(0), the reference's strongest pair, across one restart.
        {"name": "gmres_ilu0_f64_grid_1000x1024", "call": "gmres", "matrix": "grid", "shape": "1000x1024",
         "sigma": 1.0, "mass": 0.001, "velocity": 0.5, "format": "CSR", "real": "f64", "precond": "ILU0",
         "variant": "MGSR", "restart": 30, "iterations": 40},
        # The mixed-precision PCG with FSAI at the size of the preconditioner evaluation.
        {"name": "reliable_fsai_grid_2048x2048", "call": "reliable", "matrix": "grid", "shape": "2048x2048",
         "sigma": 1.0, "mass": 0.01, "format": "CSR", "real": "f64", "inner": "fsai", "tol": 1e-10,
         "counted": 268},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _shape(rng, lo, hi, dim):
    """Grid sides whose product is about log-uniform in [lo, hi], each side drawn by itself."""
    n = _log(rng, lo, hi)
    side = n ** (1.0 / dim)
    sides = [max(5, int(side * rng.uniform(0.7, 1.0 / 0.7))) for _ in range(dim - 1)]
    last = max(5, n // math.prod(sides))
    return "x".join(str(s) for s in sides + [last])


def _matrix(rng, n_max):
    kind = rng.choice(("grid", "grid", "powerlaw", "fem"))
    if kind == "grid":
        dim = rng.choice((2, 3))
        return {"matrix": "grid", "shape": _shape(rng, 1000, n_max, dim), "sigma": rng.choice((0.0, 1.0, 2.0))}
    return {"matrix": kind, "n": _log(rng, 1000, n_max if kind == "powerlaw" else n_max // 4)}


def draw(rng):
    call = rng.choice(("product", "product", "product", "product", "transposed", "symmetric", "assign", "cg", "cg",
                       "bicgstab", "gmres", "gmres", "reliable"))
    real = rng.choice(("f64", "f64", "f32"))
    if call in ("product", "transposed", "symmetric", "assign"):
        case = {"call": call, **_matrix(rng, 4194304 if call == "product" else 2000000), "real": real}
        formats = FORMATS
        if case["matrix"] == "powerlaw":  # padding to the longest row of a graph is not used
            formats = ("CSR", "AdaptiveCSR", "ChunkedEllpack", "BiEllpack")
        if call != "product":
            formats = [f for f in formats if f != "Ellpack"]
        case["format"] = rng.choice(formats)
        if call != "assign":
            case["residual"] = rng.choice((False, False, True))
        return case
    dim = rng.choice((2, 3))
    case = {"call": call, "matrix": "grid", "sigma": rng.choice((0.5, 1.0)), "format": "CSR", "real": "f64"}
    if call == "cg":
        case.update(shape=_shape(rng, 1000, 1000000, dim), mass=0.01, real=real, precond="Diagonal",
                    iterations=rng.randint(20, 200))
        case["format"] = rng.choice(("CSR", "CSR", "SlicedEllpack", "Ellpack"))
    elif call == "bicgstab":
        case.update(shape=_shape(rng, 1000, 1000000, dim), mass=0.05, velocity=rng.choice((0.5, 1.0, 2.0)),
                    precond=rng.choice(("Diagonal", "Diagonal", "ILU0")), iterations=rng.randint(10, 40))
    elif call == "gmres":
        case.update(shape=_shape(rng, 1000, 1000000, dim), mass=0.001, velocity=rng.choice((0.5, 1.0, 2.0)),
                    precond=rng.choice(("ILU0", "ILU0", "Diagonal")),
                    variant=rng.choice(("MGSR", "MGSR", "MGS", "CGSR", "CWY")), restart=rng.choice((10, 30)),
                    iterations=rng.randint(10, 40))
        if case["variant"] == "CWY" and case["iterations"] % (case["restart"] + 1) == 0:
            case["iterations"] += 1  # a budget that ends on a cycle's first reflection leaves nothing to update
    else:
        case.update(shape=_shape(rng, 10000, 4000000, dim), mass=0.01, inner=rng.choice(("fsai", "fsai", "jacobi")),
                    tol=rng.choice((1e-8, 1e-10)))
    return case


# ---------------------------------------------------------------- matrices

class _CSR:
    """Device CSR arrays (int32 rowptr and cols, FP64 values), n rows and columns."""

    def __init__(self, rowptr, cols, vals):
        self.rowptr, self.cols, self.vals = rowptr, cols, vals
        self.n = rowptr.numel() - 1


def _generator(seed, stream):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 16 + stream)
    return g


def _rand(seed, stream, size, lo=-1.0, hi=1.0):
    u = torch.rand(size, dtype=torch.float64, device="cuda", generator=_generator(seed, stream))
    return u * (hi - lo) + lo


def _field(shape, sigma, seed):
    """exp of a Gaussian random field of correlation length 0.1, scaled to standard deviation sigma."""
    if sigma == 0.0:
        return torch.ones(shape, dtype=torch.float64, device="cuda")
    w = torch.randn(shape, dtype=torch.float64, device="cuda", generator=_generator(seed, 1))
    W = torch.fft.rfftn(w)
    k2 = torch.zeros((), dtype=torch.float64, device="cuda")
    for a, s in enumerate(shape):
        f = torch.fft.rfftfreq(s, device="cuda") if a == len(shape) - 1 else torch.fft.fftfreq(s, device="cuda")
        f = f.to(torch.float64) * s * 2.0 * math.pi
        k2 = k2 + (f * f).reshape([-1 if b == a else 1 for b in range(len(shape))])
    g = torch.fft.irfftn(W * torch.exp(-k2 * 0.00125), s=shape)
    g = g - g.mean()
    return torch.exp(g * (sigma / g.std()))


def _grid(case, seed):
    """The operator by diagonals: sorted (column - row) offsets and the n x D weights (0 outside the grid)."""
    shape = tuple(int(s) for s in case["shape"].split("x"))
    k = _field(shape, case["sigma"], seed)
    k = k / k.mean()
    dim, v = len(shape), float(case.get("velocity", 0.0))
    diag = torch.full(shape, float(case.get("mass", 0.0)), dtype=torch.float64, device="cuda")
    parts, stride = [], 1
    strides = []
    for s in reversed(shape):
        strides.insert(0, stride)
        stride *= s
    for a in range(dim):
        for side in (-1, 1):
            n_a = shape[a]
            me = k.narrow(a, 1, n_a - 1) if side < 0 else k.narrow(a, 0, n_a - 1)
            nb = k.narrow(a, 0, n_a - 1) if side < 0 else k.narrow(a, 1, n_a - 1)
            w = 2.0 * k  # a wall lies half a cell away
            w.narrow(a, 1 if side < 0 else 0, n_a - 1).copy_(2.0 * me * nb / (me + nb))
            w = w + (v if side < 0 else 0.0)  # upwind: the flow comes from the lower side
            diag += w
            w.select(a, 0 if side < 0 else n_a - 1).zero_()  # Dirichlet: no entry
            parts.append((side * strides[a], -w.reshape(-1)))
    parts.append((0, diag.reshape(-1)))
    parts.sort(key=lambda p: p[0])
    return [p[0] for p in parts], torch.stack([p[1] for p in parts], dim=1)


def _grid_csr(offsets, weights):
    n = weights.shape[0]
    mask = weights != 0.0
    rowptr = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    rowptr[1:] = torch.cumsum(mask.sum(1), 0).to(torch.int32)
    cols = torch.arange(n, dtype=torch.int32, device="cuda")[:, None] + torch.tensor(offsets, dtype=torch.int32,
                                                                                      device="cuda")
    return _CSR(rowptr, cols[mask], weights[mask])


def _grid_apply(offsets, weights, x):
    """A x with every row summed in ascending column order."""
    y = torch.zeros_like(x)
    for j, o in enumerate(offsets):
        y += weights[:, j] * torch.roll(x, -o)  # entries that would wrap have weight 0
    return y


def _uneven(case, seed):
    """powerlaw and fem: row lengths drawn once for the size (the same for every seed, so that the storage is);
    a row's columns are drawn one from each of its equal strata, so they ascend, all different."""
    n = case["n"]
    if case["matrix"] == "powerlaw":
        p = torch.arange(1, min(ZIPF_CAP, n) + 1, dtype=torch.float64, device="cuda") ** -ZIPF
        cdf = torch.cumsum(p, 0)
        u = _rand(n, 2, n, 0.0, 1.0) * cdf[-1]
        lens = (torch.searchsorted(cdf, u) + 1).clamp_(max=p.numel())
        first, width = torch.zeros_like(lens), torch.full_like(lens, n)
    else:
        lens = torch.randint(FEM_MIN, FEM_MAX + 1, (n,), device="cuda", generator=_generator(n, 2))
        half = min(n // 2, max(64, int(n ** (2.0 / 3.0))))
        i = torch.arange(n, device="cuda")
        first = (i - half).clamp_(min=0)
        width = (i + half).clamp_(max=n) - first
    rowptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(lens, 0, out=rowptr[1:])
    nnz = int(rowptr[-1])
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), lens, output_size=nnz)
    j = torch.arange(nnz, device="cuda") - rowptr[row]
    lo, hi = j * width[row] // lens[row], (j + 1) * width[row] // lens[row]
    cols = first[row] + lo + (_rand(seed, 3, nnz, 0.0, 1.0) * (hi - lo)).to(torch.int64).clamp_(max=hi - lo - 1)
    return _CSR(rowptr.to(torch.int32), cols.to(torch.int32), _rand(seed, 4, nnz))


def _csr(case, seed):
    A = _grid_csr(*_grid(case, seed)) if case["matrix"] == "grid" else _uneven(case, seed)
    if case["call"] == "symmetric":  # one triangle is stored
        row = torch.repeat_interleave(torch.arange(A.n, device="cuda"), (A.rowptr[1:] - A.rowptr[:-1]).to(torch.int64))
        low = A.cols <= row
        rowptr = torch.zeros(A.n + 1, dtype=torch.int32, device="cuda")
        rowptr[1:] = torch.cumsum(torch.bincount(row[low], minlength=A.n), 0).to(torch.int32)
        A = _CSR(rowptr, A.cols[low], A.vals[low])
    return A


def _rounded(case, A):
    """The values as the matrix stores them, in FP64."""
    return A.vals.to(REALS[case["real"]]).to(torch.float64)


def _vectors(case, n, seed):
    real = REALS[case["real"]]
    return _rand(seed, 5, n).to(real), _rand(seed, 6, n).to(real)


def _system(case, seed):
    """A solve's matrix and right-hand side b = A x of a drawn x."""
    offsets, weights = _grid(case, seed)
    weights = weights.to(REALS[case["real"]])
    x = _rand(seed, 5, weights.shape[0])
    b = _grid_apply(offsets, weights.to(torch.float64), x).to(weights.dtype)
    return offsets, weights, x, b


# ------------------------------------------------------------------- calls

def _new_matrix(case, A):
    M = tnl.SparseMatrix(getattr(tnl, case["format"]), REALS[case["real"]], symmetric=case["call"] == "symmetric")
    return M.assign(A.rowptr, A.cols, A.vals, A.n)


def prepare(case, seed):
    call = case["call"]
    if call in ("product", "transposed", "symmetric"):
        A = _csr(case, seed)
        M = _new_matrix(case, A)
        x, b = _vectors(case, A.n, seed)
        launch = tnl.LaunchConfiguration("Adaptive") if case["format"] == "AdaptiveCSR" else None
        return {"case": case, "M": M, "x": x, "b": b, "y": torch.zeros_like(b), "launch": launch}
    if call == "assign":
        A = _csr(case, seed)
        return {"case": case, "rowptr": A.rowptr, "cols": A.cols, "vals": A.vals.to(REALS[case["real"]]), "n": A.n}
    offsets, weights, _, b = _system(case, seed)
    M = _new_matrix(case, _grid_csr(offsets, weights))
    if call == "reliable":
        return {"case": case, "M": M, "b": b}
    solver = {"cg": tnl.CG, "bicgstab": tnl.BICGStab, "gmres": tnl.GMRES}[call]()
    solver.setMatrix(M)
    P = getattr(tnl, case["precond"])()
    P.update(M)
    solver.setPreconditioner(P)
    solver.setConvergenceResidue(0.0)
    solver.setMaxIterations(case["iterations"])
    if call == "gmres":
        solver.setup({"gmres-variant": case["variant"], "gmres-restarting-min": case["restart"],
                      "gmres-restarting-max": case["restart"]})
    return {"case": case, "solver": solver, "b": b}


def run(state):
    case = state["case"]
    call = case["call"]
    if call in ("product", "transposed", "symmetric"):
        M, x, y = state["M"], state["x"], state["y"]
        alpha, beta = 1.0, 0.0
        if case["residual"]:
            y.copy_(state["b"])
            alpha, beta = -1.0, 1.0
        if call == "transposed":
            M.transposedVectorProduct(x, y, alpha, beta, synchronize=False)
        else:
            M.vectorProduct(x, y, alpha, beta, launchConfig=state["launch"], synchronize=False)
        return y
    if call == "assign":
        M = tnl.SparseMatrix(getattr(tnl, case["format"]), REALS[case["real"]])
        M.assign(state["rowptr"], state["cols"], state["vals"], state["n"])
        return M.getColumnIndexes(), M.getValues()
    x = torch.zeros_like(state["b"])
    if call == "reliable":
        result = tnl.solve_mixed_reliable(state["M"], state["b"], x, tol=case["tol"], inner=case["inner"])
        return x, int(result["converged"])
    state["solver"].solve(state["b"], x)
    return x


# ------------------------------------------------------- bytes, tolerances

# Iterations of the mixed-precision PCG on these operators (time-step term
# 0.01) to 1e-10, where a case does not give its own count.
RELIABLE_ITERATIONS = {"fsai": 130, "jacobi": 160}


def _nnz(case):
    if case["matrix"] == "grid":
        shape = [int(s) for s in case["shape"].split("x")]
        n = math.prod(shape)
        return n, n + sum(2 * (n - n // s) for s in shape)
    n = case["n"]
    if case["matrix"] == "fem":
        return n, n * (FEM_MIN + FEM_MAX) // 2
    ks = range(1, min(ZIPF_CAP, n) + 1)
    return n, int(n * sum(k ** (1.0 - ZIPF) for k in ks) / sum(k ** -ZIPF for k in ks))


def _steps(case):
    """Products with A of a solve's iterations; the stopping rule lets one more than the stated number run."""
    count = case["iterations"] + 1
    if case.get("variant") != "CWY":
        return count
    cycles, rest = divmod(count, case["restart"] + 1)  # a cycle of m products counts m + 1 reflections
    return cycles * case["restart"] + max(rest - 1, 0)


def work(case):
    n, nnz = _nnz(case)
    R = 8 if case["real"] == "f64" else 4
    call = case["call"]
    if call == "symmetric":
        nnz = (nnz + n) // 2 if case["matrix"] == "grid" else nnz // 2
    matrix = nnz * (R + 4) + 4 * (n + 1)
    if call in ("product", "transposed", "symmetric"):
        flops = 4 * nnz if call == "symmetric" else 2 * nnz
        return {"bytes": matrix + (3 if case["residual"] else 2) * n * R, "flops": flops}
    if call == "assign":
        return {"bytes": 2 * matrix, "flops": 0}
    if call == "reliable":
        # FP32 iterations: A's values, two factors, r, p in FP32 and x in FP64
        low = (nnz + n) // 2
        its = case.get("counted") or RELIABLE_ITERATIONS[case["inner"]] * (5 if case["tol"] < 1e-9 else 4) // 5
        factors = 2 * low * 2 if case["inner"] == "fsai" else 4 * n
        return {"bytes": its * (4 * nnz + factors + 32 * n),
                "flops": its * (2 * nnz + (4 * low if case["inner"] == "fsai" else n) + 12 * n)}
    its = _steps(case)
    precond = matrix if case["precond"] == "ILU0" else n * R
    if call == "cg":
        return {"bytes": its * (matrix + precond + 6 * n * R), "flops": its * (2 * nnz + 13 * n)}
    if call == "bicgstab":
        return {"bytes": its * (2 * (matrix + precond) + 8 * n * R), "flops": its * (4 * nnz + 22 * n)}
    # GMRES: every basis vector read once in each pass of the orthogonalisation
    m, passes = case["restart"], 2 if case["variant"] in ("MGSR", "CGSR") else 1
    basis = passes * sum(i % m + 1 for i in range(its))
    return {"bytes": its * (matrix + precond + 2 * n * R) + basis * n * R,
            "flops": its * (4 * nnz if case["precond"] == "ILU0" else 2 * nnz) + 4 * basis * n}


def tolerance(case):
    call, f64 = case["call"], case["real"] == "f64"
    if call == "assign":
        return "exact"
    if call in ("product", "transposed", "symmetric"):
        return {"rel": 2e-15 if f64 else 1e-6}
    if call == "cg":
        return {"rel": 1e-14 if f64 else 3e-6}
    if call == "bicgstab":  # its recurrences amplify a change in the order of a sum, up to 9e-11 seen in 2D
        return {"rel": 4e-10}
    if call == "gmres":
        return {"rel": 1e-14}
    # what the stopping residue leaves of the error on these operators
    return {"rel": 4e-8 if case["tol"] < 1e-9 else 4e-6}


# ------------------------------------------------------------------- exact

def _matvec(rowptr, cols, vals, n, x, chunk=1 << 25):
    """A x in FP64 and the entries' rows; a row's entries are dealt over 16 partial sums."""
    parts = torch.zeros(16 * n, dtype=torch.float64, device="cuda")
    lens = (rowptr[1:] - rowptr[:-1]).to(torch.int64)
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), lens, output_size=cols.numel())
    for s in range(0, cols.numel(), chunk):
        e = min(s + chunk, cols.numel())
        slot = row[s:e] * 16 + torch.arange(s, e, device="cuda") % 16
        parts.index_add_(0, slot, vals[s:e] * x[cols[s:e].to(torch.int64)])
    return parts.reshape(n, 16).sum(1), row


class _ILU0:
    """ILU(0) of a grid operator by diagonals: only the pivots differ from A's own entries."""

    def __init__(self, case, offsets, weights):
        shape = [int(s) for s in case["shape"].split("x")]
        level = torch.zeros(shape, dtype=torch.int64, device="cuda")
        for a, s in enumerate(shape):
            level += torch.arange(s, device="cuda").reshape([-1 if b == a else 1 for b in range(len(shape))])
        level = level.reshape(-1)
        order = torch.argsort(level, stable=True)
        self.levels = list(torch.split(order, torch.bincount(level).tolist()))
        self.n, D = weights.shape
        low = [j for j in range(D) if offsets[j] < 0]
        self.diag = [j for j in range(D) if offsets[j] == 0][0]
        self.parts = []
        pivot = weights[:, self.diag].clone()
        index = torch.arange(self.n, device="cuda")
        # factors of row i: L_ij = a_ij / pivot_j, U_ij = a_ij
        mirror = {j: offsets.index(-offsets[j]) for j in range(D)}
        for side in (low, [j for j in range(D) if offsets[j] > 0]):
            nb = torch.stack([(index + offsets[j]).clamp_(0, self.n - 1) for j in side], 1)
            self.parts.append((side, nb))
        nb = self.parts[0][1]
        back = torch.stack([weights[nb[:, q], mirror[j]] for q, j in enumerate(low)], 1)
        a = weights[:, low]
        for rows in self.levels[1:]:
            pivot[rows] -= (a[rows] * back[rows] / pivot[nb[rows]]).sum(1)
        self.pivot = pivot
        self.lower = a / pivot[nb]
        self.upper = weights[:, self.parts[1][0]]
        self.steps = [(r, self.lower[r], self.parts[0][1][r], self.upper[r], self.parts[1][1][r], pivot[r])
                      for r in self.levels]

    def solve(self, b):
        x = b.clone()
        for rows, lo, nb, _, _, _ in self.steps[1:]:
            x[rows] -= (lo * x[nb]).sum(1)
        for rows, _, _, up, nb, piv in reversed(self.steps):
            x[rows] = (x[rows] - (up * x[nb]).sum(1)) / piv
        return x


def _cg(A, M, b, steps):
    x = torch.zeros_like(b)
    r = b.clone()
    z = M(r)
    p, rz = z.clone(), torch.dot(r, z)
    for _ in range(steps):
        Ap = A(p)
        alpha = rz / torch.dot(p, Ap)
        x += alpha * p
        r -= alpha * Ap
        z = M(r)
        old, rz = rz, torch.dot(r, z)
        p = z + (rz / old) * p
    return x


def _bicgstab(A, M, b, steps):
    x = torch.zeros_like(b)
    r = M(b)
    rh, p = r.clone(), r.clone()
    rho = torch.dot(r, rh)
    for _ in range(steps):
        Ap = M(A(p))
        alpha = rho / torch.dot(Ap, rh)
        s = r - alpha * Ap
        As = M(A(s))
        omega = torch.dot(As, s) / torch.dot(As, As)
        x += alpha * p + omega * s
        r = s - omega * As
        old, rho = rho, torch.dot(r, rh)
        p = r + (rho / old) * (alpha / omega) * (p - omega * Ap)
    return x


def _gmres(A, M, b, steps, m):
    x = torch.zeros_like(b)
    while steps > 0:
        r = M(b - A(x))
        beta = torch.linalg.vector_norm(r)
        k = min(m, steps)
        V = torch.zeros(k + 1, b.numel(), dtype=torch.float64, device="cuda")
        H = torch.zeros(k + 1, k, dtype=torch.float64, device="cuda")
        V[0] = r / beta
        for i in range(k):
            w = M(A(V[i]))
            for _ in range(2):
                h = V[:i + 1] @ w
                w = w - h @ V[:i + 1]
                H[:i + 1, i] += h
            H[i + 1, i] = torch.linalg.vector_norm(w)
            V[i + 1] = w / H[i + 1, i]
        e = torch.zeros(k + 1, 1, dtype=torch.float64, device="cuda")
        e[0] = beta
        x = x + torch.linalg.lstsq(H, e).solution[:, 0] @ V[:k]
        steps -= k
    return x


def exact(case, seed):
    call = case["call"]
    if call == "assign":
        return None  # moved, not computed
    if call in ("product", "transposed", "symmetric"):
        A = _csr(case, seed)
        vals = _rounded(case, A)
        x, b = (v.to(torch.float64) for v in _vectors(case, A.n, seed))
        if call == "transposed":
            row = torch.repeat_interleave(torch.arange(A.n, device="cuda"),
                                          (A.rowptr[1:] - A.rowptr[:-1]).to(torch.int64))
            y = torch.zeros_like(x).index_add_(0, A.cols.to(torch.int64), vals * x[row])
        else:
            y, row = _matvec(A.rowptr, A.cols, vals, A.n, x)
            if call == "symmetric":
                off = A.cols < row
                y.index_add_(0, A.cols[off].to(torch.int64), vals[off] * x[row[off]])
        return b - y if case["residual"] else y
    offsets, weights, x, b = _system(case, seed)
    if call == "reliable":
        return x, None  # solved to a tolerance: the solution itself
    weights, b = weights.to(torch.float64), b.to(torch.float64)
    if case["precond"] == "ILU0":
        M = _ILU0(case, offsets, weights).solve
    else:
        d = weights[:, offsets.index(0)]
        M = lambda v: v / d  # noqa: E731
    A = lambda v: _grid_apply(offsets, weights, v)  # noqa: E731
    steps = _steps(case)
    if call == "cg":
        return _cg(A, M, b, steps)
    if call == "bicgstab":
        return _bicgstab(A, M, b, steps)
    return _gmres(A, M, b, steps, case["restart"])
