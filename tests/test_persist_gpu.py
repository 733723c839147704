"""CG and BiCGStab in one resident kernel, against the same iterations in
FP64 numpy.

Sizes at the edges of the split over blocks, rows of 5, 8 and 16 slots at
most in each.  Up to 20,000 rows (12,000 of more than 8 FP64 slots) one
cluster of 16 blocks: one row, fewer rows than blocks have, a last block that
is not full.  Above that the grid: the smallest, runs that are no multiple of
32, every format and organisation, and more rows than the owners' vectors have
room for in shared memory.  Well-conditioned matrices and a few iterations, so
that rounding does not grow: one iteration adds a few ulp of the largest
entries, 1e-13 and 2e-5 are over 50 times that.
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ITERATIONS = 5


def _matrix(n, offsets, symmetric, seed):
    """The diagonally dominant matrix by diagonals and its CSR arrays."""
    rng = np.random.default_rng(seed)
    diags = {}
    for o in offsets:
        if o >= n:
            continue
        diags[o] = rng.uniform(-1, 1, n - o) * (rng.random(n - o) < 0.8)
        diags[-o] = diags[o] if symmetric else rng.uniform(-1, 1, n - o) * (rng.random(n - o) < 0.8)
    i = np.arange(n)
    r, c, v = [i], [i], [np.full(n, 4.0 + 2.0 * len(offsets)) + rng.random(n)]
    for o, d in diags.items():
        k = np.flatnonzero(d)
        r.append(k - min(o, 0))
        c.append(k + max(o, 0))
        v.append(d[k])
    r, c, v = np.concatenate(r), np.concatenate(c), np.concatenate(v)
    order = np.lexsort((c, r))
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(r, minlength=n), out=rp[1:])
    return rp, c[order].astype(np.int32), v[order], r[order]


def _cg(A, M, b, steps):
    x, r = np.zeros_like(b), b.copy()
    z = M(r)
    p, rz = z.copy(), r @ z
    for _ in range(steps):
        Ap = A(p)
        alpha = rz / (p @ Ap)
        x, r = x + alpha * p, r - alpha * Ap
        z = M(r)
        rz, old = r @ z, rz
        p = z + rz / old * p
    return x


def _bicgstab(A, M, b, steps):
    x, r = np.zeros_like(b), M(b)
    ra, p, rho = r.copy(), r.copy(), r @ r
    for _ in range(steps):
        Ap = M(A(p))
        alpha = rho / (Ap @ ra)
        s = r - alpha * Ap
        As = M(A(s))
        omega = (As @ s) / (As @ As)
        x, r = x + alpha * p + omega * s, s - omega * As
        rho, old = r @ ra, rho
        p = r + rho / old * alpha / omega * (p - omega * Ap)
    return x


CASES = [(1, (), "CSR", None), (128, (1,), "CSR", None), (129, (1, 5), "Ellpack", 0), (4001, (3, 70), "Ellpack", 1),
         (4001, (1, 2, 3, 70), "SlicedEllpack", 0), (19009, (1, 2, 3, 4, 5, 600), "SlicedEllpack", 1),
         (12001, (1, 2, 3, 4, 5, 6, 90), "CSR", None), (20001, (1, 40), "SlicedEllpack", 1),
         (20011, (1, 2, 3, 4, 5, 6, 300), "CSR", None), (40009, (2, 70), "Ellpack", 0),
         (40009, (1, 2, 70), "Ellpack", 1), (40009, (1, 2, 3, 4, 5, 70), "SlicedEllpack", 0),
         (40009, (1, 2, 3, 4, 5, 70), "SlicedEllpack", 1), (90001, (1, 2, 3, 4, 5, 600), "Ellpack", 1),
         (151553, (1, 2, 300), "CSR", None), (1500007, (1, 1200), "CSR", None)]


@pytest.mark.parametrize("real", ["float64", "float32"])
@pytest.mark.parametrize("solver,precond", [("CG", True), ("CG", False), ("BICGStab", True), ("BICGStab", False)])
@pytest.mark.parametrize("n,offsets,fmt,org", CASES)
def test_resident_solver_matches_numpy(n, offsets, fmt, org, solver, precond, real):
    import tnl_b200 as t

    if n == 1 and solver == "BICGStab":
        pytest.skip("0 / 0: its first half step solves one row")
    rp, cols, vals, rows = _matrix(n, offsets, solver == "CG", n + len(offsets))
    dtype = getattr(torch, real)
    vals = vals.astype(real).astype(np.float64)
    b = np.random.default_rng(1).uniform(-1, 1, n).astype(real).astype(np.float64)
    diag = vals[rows == cols]
    A = lambda v: np.bincount(rows, vals * v[cols], minlength=n)  # noqa: E731
    M = (lambda v: v / diag) if precond else (lambda v: v)  # noqa: E731
    steps = ITERATIONS if n > 1 else 1  # one row is solved by the first
    want = (_cg if solver == "CG" else _bicgstab)(A, M, b, steps)
    mat = t.SparseMatrix(t.FORMATS[fmt], dtype, org).assign(rp, cols, vals)
    S = getattr(t, solver)()
    S.setMatrix(mat)
    if precond:
        P = t.Diagonal()
        P.update(mat)
        S.setPreconditioner(P)
    S.setConvergenceResidue(0.0)
    S.setMaxIterations(steps - 1)  # the stopping rule lets one more run
    if n == 1:
        S.setConvergenceResidue(1e-5)
    bs = torch.tensor(b, dtype=dtype, device="cuda")
    for _ in range(2):
        x = torch.zeros(n, dtype=dtype, device="cuda")
        S.solve(bs, x)
        err = np.linalg.norm(x.cpu().numpy().astype(np.float64) - want)
        assert err <= (1e-13 if real == "float64" else 2e-5) * np.linalg.norm(want)


@pytest.mark.parametrize("n", [4001, 40009])  # one cluster, the grid
def test_resident_bicgstab_restarts(n):
    """100 iterations where 30 reach the rounding level: (r, r_ast) falls below
    the restart's threshold again and again, and x stays the solution."""
    import tnl_b200 as t

    rp, cols, vals, rows = _matrix(n, (1, 70), False, 7)
    want = np.random.default_rng(2).uniform(-1, 1, n)
    b = np.bincount(rows, vals * want[cols], minlength=n)
    mat = t.SparseMatrix(t.CSR, torch.float64).assign(rp, cols, vals)
    S = t.BICGStab()
    S.setMatrix(mat)
    S.setConvergenceResidue(0.0)
    S.setMaxIterations(100)
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    S.solve(torch.tensor(b, device="cuda"), x)
    assert S.getIterations() == 102
    assert np.linalg.norm(x.cpu().numpy() - want) <= 1e-13 * np.linalg.norm(want)


def test_resident_cg_over_several_launches():
    """More iterations than one launch runs (2048): the state carries over, so
    that the recursive residual still tells the true one."""
    import tnl_b200 as t
    from tnl_b200 import generators as g

    L = g.laplacian_2d(1000)
    mat = t.SparseMatrix(t.CSR, torch.float64).assign(L.rowptr, L.cols, L.vals)
    S = t.CG()
    S.setMatrix(mat)
    S.setConvergenceResidue(0.0)
    S.setMaxIterations(2100)
    b = torch.tensor(g.uniform_vector(L.n, 1), device="cuda")
    x = torch.zeros_like(b)
    S.solve(b, x)
    assert S.getIterations() == 2102
    assert abs(t.true_residual(mat, b, x) / S.getResidue() - 1) < 1e-3


@pytest.mark.parametrize("real", ["float64", "float32"])
@pytest.mark.parametrize("variant", ["MGS", "MGSR"])
@pytest.mark.parametrize("n", [33, 20000, 20001, 151553])
def test_resident_gram_schmidt_matches_numpy(n, variant, real):
    """Seven GMRES iterations across a restart of 4: one cluster, the grid."""
    import tnl_b200 as t

    rp, cols, vals, rows = _matrix(n, (1, 5), False, n)
    dtype = getattr(torch, real)
    vals = vals.astype(real).astype(np.float64)
    b = np.random.default_rng(1).uniform(-1, 1, n).astype(real).astype(np.float64)
    x = np.zeros(n)
    for steps in (4, 3):
        r = b - np.bincount(rows, vals * x[cols], minlength=n)
        V, H = [r / np.linalg.norm(r)], np.zeros((steps + 1, steps))
        for i in range(steps):
            w = np.bincount(rows, vals * V[i][cols], minlength=n)
            for _ in range(2):
                for k in range(i + 1):
                    h = w @ V[k]
                    H[k, i] += h
                    w = w - h * V[k]
            H[i + 1, i] = np.linalg.norm(w)
            V.append(w / H[i + 1, i])
        e = np.zeros(steps + 1)
        e[0] = np.linalg.norm(r)
        x = x + np.linalg.lstsq(H, e, rcond=None)[0] @ np.array(V[:steps])
    mat = t.SparseMatrix(t.CSR, dtype).assign(rp, cols, vals)
    S = t.GMRES()
    S.setMatrix(mat)
    S.setConvergenceResidue(0.0)
    S.setMaxIterations(6)
    S.setup({"gmres-variant": variant, "gmres-restarting-min": 4, "gmres-restarting-max": 4})
    y = torch.zeros(n, dtype=dtype, device="cuda")
    S.solve(torch.tensor(b, dtype=dtype, device="cuda"), y)
    err = np.linalg.norm(y.cpu().numpy().astype(np.float64) - x)
    assert err <= (1e-13 if real == "float64" else 2e-5) * np.linalg.norm(x)


def test_resident_solvers_on_two_streams():
    """Two threads, each on a stream of its own, with systems of different forms:
    the results of one thread alone."""
    import threading

    import tnl_b200 as t

    systems = []
    for k, (n, offsets, solver) in enumerate([(9001, (1, 70), "CG"), (60013, (1, 2, 300), "BICGStab"),
                                              (60013, (1, 300), "CG"), (9001, (1, 2, 70), "GMRES")]):
        rp, cols, vals, _ = _matrix(n, offsets, solver == "CG", k)
        mat = t.SparseMatrix(t.CSR, torch.float64).assign(rp, cols, vals)
        systems.append((solver, mat, torch.tensor(np.random.default_rng(k).uniform(-1, 1, n), device="cuda")))
    torch.cuda.synchronize()

    def solve(which, out):
        with torch.cuda.stream(torch.cuda.Stream()):
            for solver, mat, b in which:
                S = getattr(t, solver)()
                S.setMatrix(mat)
                S.setConvergenceResidue(0.0)
                S.setMaxIterations(ITERATIONS)
                x = torch.zeros_like(b)
                S.solve(b, x)
                out.append(x)

    want = []
    solve(systems, want)
    for _ in range(3):
        got = [[], []]
        threads = [threading.Thread(target=solve, args=(order, out))
                   for order, out in ((systems, got[0]), (systems[::-1], got[1]))]
        for th in threads:
            th.start()
        for th in threads:
            th.join()
        assert len(got[0]) == len(got[1]) == len(want)
        for a, b, w in zip(got[0], got[1][::-1], want):
            assert torch.equal(a, w) and torch.equal(b, w)
