"""CG and BiCGStab on systems that fit on chip (one kernel for all iterations)
against the oracle's solvers, where that kernel's shape changes: one row, one
block and two, the largest cluster and the first system beyond it, several
rows per thread, rows as long as they may be, padded layouts, launches of a
few iterations each, and every way a solve ends.

x at a residue of 1e-10 within what that residue allows. The iteration counts move with the order of
the sums (BiCGStab's by a fifth on these systems): they have to lie where the
oracle's lie when the last digit of b changes (eight runs), or as far again on
either side, and two more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _spd(n, offsets, seed=0):
    """Symmetric, diagonally dominant, with face coefficients exp(N(0, 1)): some tens of iterations."""
    g = np.random.default_rng(seed)
    rows, cols, vals = [np.arange(n)], [np.arange(n)], [None]
    diag = np.full(n, 0.5)
    for o in offsets:
        if o >= n:
            continue
        i = np.arange(n - o)
        k = np.exp(g.normal(size=n - o))
        for r, c in ((i, i + o), (i + o, i)):
            rows.append(r)
            cols.append(c)
            vals.append(-k)
            np.add.at(diag, r, k)
    vals[0] = diag
    rows, cols, vals = np.concatenate(rows), np.concatenate(cols), np.concatenate(vals)
    order = np.lexsort((cols, rows))
    off = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    return off, cols[order].astype(np.int32), vals[order], n


CASES = {
    "one_row": lambda: _spd(1, []),
    "n_31": lambda: _spd(31, [1, 5]),
    "n_512": lambda: _spd(512, [1, 32]),
    "n_513": lambda: _spd(513, [1, 32]),
    "n_4099": lambda: _spd(4099, [1, 64]),
    "n_16384": lambda: _spd(16384, [1, 128]),
    "n_16385": lambda: _spd(16385, [1, 128]),
    "rows_of_65": lambda: _spd(3000, list(range(1, 33))),
}


def _solver(b2s_lib, kind):
    return {"cg": b2s_lib.CG, "bicgstab": b2s_lib.BICGStab}[kind]()


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
@pytest.mark.parametrize("precond", [None, "diagonal"])
def test_resident_vs_oracle(b2s_lib, cuda, oracle, name, kind, precond):
    csr = CASES[name]()
    n = csr[3]
    b = np.random.default_rng(4).uniform(-1, 1, n)
    want = oracle.solve(kind, csr, b, rtol=1e-10, precond=precond is not None)
    g = np.random.default_rng(5)
    counts = [want["iterations"]] + [
        oracle.solve(kind, csr, b * (1 + 2.0 ** -52 * g.uniform(-1, 1, n)), rtol=1e-10,
                     precond=precond is not None)["iterations"] for _ in range(7)]
    spread = max(counts) - min(counts) + 2
    # A = a Laplacian + 0.5 I, so an error is at most twice its residual r, and
    # the residue bounds |r| by 1e-10 |b| or, preconditioned with M = diag(A),
    # |M^-1 r| by 1e-10 |M^-1 b|; the oracle's solution is as far off
    d = csr[2][csr[1] == np.repeat(np.arange(n), np.diff(csr[0]))]
    bound = 4e-10 * (np.linalg.norm(b) if precond is None else np.max(d) * np.linalg.norm(b / d))
    for segments, interval in (("CSR", 0), ("SlicedEllpack", 0), ("Ellpack", 7)):
        M = b2s_lib.SparseMatrix.from_csr(*csr[:3], n, segments=segments)
        s = _solver(b2s_lib, kind)
        s.setMatrix(M)
        s.setPreconditioner(precond)
        s.setConvergenceResidue(1e-10)
        s.setCheckInterval(interval)
        for _ in range(2):  # the second solve goes on from the first one's count of meetings
            x = cuda.zeros(n, dtype=cuda.float64, device="cuda")
            ok = s.solve(cuda.tensor(b, device="cuda"), x)
            tag = (segments, interval, s.getIterations(), counts)
            assert ok == want["converged"], tag
            assert min(counts) - spread <= s.getIterations() <= max(counts) + spread, tag
            xh = x.cpu().numpy()
            if np.isnan(want["x"]).any():  # BiCGStab's 0 / 0 after an exact first step
                assert np.array_equal(np.isnan(xh), np.isnan(want["x"])), tag
            else:
                assert np.max(np.abs(xh - want["x"])) <= bound, tag


@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
@pytest.mark.parametrize("n", [900, 20000])
def test_resident_ends(b2s_lib, cuda, kind, n):
    """The iteration limit, a zero right-hand side, an exact guess, NaN."""
    csr = _spd(n, [1, 30])
    M = b2s_lib.SparseMatrix.from_csr(*csr[:3], n)
    b = cuda.rand(n, dtype=cuda.float64, device="cuda")
    s = _solver(b2s_lib, kind)
    s.setMatrix(M)
    s.setConvergenceResidue(1e-10)
    s.setMaxIterations(5)
    x = cuda.zeros_like(b)
    assert not s.solve(b, x) and 5 <= s.getIterations() <= 7
    s.setMaxIterations(100000)
    assert s.solve(b, x)
    its = s.getIterations()
    assert s.solve(b, x) and s.getIterations() <= 2 < its  # from the solution
    x.zero_()
    assert s.solve(cuda.zeros_like(b), x) and bool((x == 0).all())
    b[7] = float("nan")
    x.zero_()
    assert not s.solve(b, x)
    b[7] = 0.5
    x.zero_()
    assert s.solve(b, x) and s.getIterations() >= 3  # the state of the failed solve is gone


@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
@pytest.mark.parametrize("n", [900, 20000])
def test_resident_single_and_mixed_precision(b2s_lib, cuda, oracle, kind, n):
    csr = _spd(n, [1, 30])
    b = np.random.default_rng(6).uniform(-1, 1, n)
    want = oracle.solve(kind, csr, b, rtol=1e-10)
    M = b2s_lib.SparseMatrix.from_csr(*csr[:3], n, keep_fp32_copy=True)
    s = _solver(b2s_lib, kind)
    s.setMatrix(M)
    s.setConvergenceResidue(1e-10)
    s.setPrecision(True)
    x = cuda.zeros(n, dtype=cuda.float64, device="cuda")
    assert s.solve(cuda.tensor(b, device="cuda"), x)
    assert np.max(np.abs(x.cpu().numpy() - want["x"])) <= 1e-7 * np.max(np.abs(want["x"]))
    F = b2s_lib.SparseMatrix.from_csr(*csr[:3], n, real="float")
    s = _solver(b2s_lib, kind)
    s.setMatrix(F)
    s.setConvergenceResidue(1e-4)
    x = cuda.zeros(n, dtype=cuda.float32, device="cuda")
    assert s.solve(cuda.tensor(b, dtype=cuda.float32, device="cuda"), x)
    r = np.linalg.norm(oracle.spmv("csr", "col", csr, x.cpu().numpy().astype(np.float64)) - b)
    assert r <= 1e-3 * np.linalg.norm(b)  # the recurrence's residue, and FP32's rounding on top


# beyond one cluster a block takes n / 148 rows, here 541 to 2,095 (the last block fewer):
# two, four and eight to a thread; FP64 BiCGStab at most four
@pytest.mark.parametrize("n", [80_001, 160_003, 310_005])
@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
@pytest.mark.parametrize("mixed", [False, True])
def test_resident_rows_per_thread(b2s_lib, cuda, oracle, n, kind, mixed):
    csr = _spd(n, [1, 700])
    b = np.random.default_rng(8).uniform(-1, 1, n)
    for precond in (None, "diagonal"):
        want = oracle.solve(kind, csr, b, rtol=1e-10, precond=precond is not None)
        d = csr[2][csr[1] == np.repeat(np.arange(n), np.diff(csr[0]))]  # the bound: test_resident_vs_oracle
        bound = 4e-10 * (np.linalg.norm(b) if precond is None else np.max(d) * np.linalg.norm(b / d))
        for segments in ("CSR", "SlicedEllpack", "Ellpack"):
            M = b2s_lib.SparseMatrix.from_csr(*csr[:3], n, segments=segments, keep_fp32_copy=mixed)
            s = _solver(b2s_lib, kind)
            s.setMatrix(M)
            s.setPreconditioner(precond)
            s.setConvergenceResidue(1e-10)
            s.setPrecision(mixed)
            x = cuda.zeros(n, dtype=cuda.float64, device="cuda")
            assert s.solve(cuda.tensor(b, device="cuda"), x), (precond, segments)
            err = np.max(np.abs(x.cpu().numpy() - want["x"]))
            assert err <= bound, (precond, segments, err, bound)
