"""Handles that are used again after their matrix was permuted in place: what
was captured with the arrays' old addresses must not run again. Each result
equals, bit for bit, that of a handle made after the permutation."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 110_000  # above the row count from which products go through row patterns


def _band(offsets, seed):
    g = np.random.default_rng(seed)
    i = np.arange(N)
    c = i[:, None] + np.asarray(offsets)[None, :]
    keep = (c >= 0) & (c < N)
    val = g.uniform(-1, 1, c.shape)
    val[:, list(offsets).index(0)] = 2.0 * len(offsets)
    off = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int32)
    return off, c[keep].astype(np.int32), val[keep]


def _same_bits(cuda, a, b):
    return cuda.equal(a.view(cuda.int64), b.view(cuda.int64))


PERMUTATIONS = {
    # patterns before and after, of other rows
    "roll": lambda: np.roll(np.arange(N), 3),
    # more patterns than are kept: the columns are read again
    "random": lambda: np.random.default_rng(1).permutation(N),
}


def _permute(M, where, name):
    p = PERMUTATIONS[name]().astype(np.int32)
    (M.permuteColumns if where == "columns" else M.permuteRows)(p)


@pytest.mark.parametrize("where,segments", [("columns", "CSR"), ("columns", "SlicedEllpack"), ("columns", "BiEllpack"),
                                            ("rows", "CSR")])
@pytest.mark.parametrize("name", list(PERMUTATIONS))
@pytest.mark.parametrize("solver", ["GMRES", "TFQMR", "SOR"])
def test_solver_used_again(b2s_lib, cuda, where, segments, name, solver):
    csr = _band([-400, -1, 0, 1, 400], 3)
    M = b2s_lib.SparseMatrix.from_csr(*csr, N, segments=segments)
    b = cuda.rand(N, dtype=cuda.float64, device="cuda")

    def solve(s):
        x = cuda.zeros_like(b)
        s.solve(b, x)
        return x

    def make():
        s = getattr(b2s_lib, solver)()
        s.setMatrix(M)
        s.setConvergenceResidue(1e-10)
        s.setMaxIterations(12)  # permuted, the system need not converge
        return s

    s = make()
    before = solve(s)
    _permute(M, where, name)
    again = solve(s)
    assert not _same_bits(cuda, again, before)
    assert _same_bits(cuda, again, solve(make()))


@pytest.mark.parametrize("name", list(PERMUTATIONS))
@pytest.mark.parametrize("pinned", [True, False])
def test_host_products_used_again(b2s_lib, cuda, name, pinned):
    """Host vectors go through a pipeline whose schedule follows the columns
    (page-locked ones through a captured graph)."""
    M = b2s_lib.SparseMatrix.from_csr(*_band([-400, -1, 0, 1, 400], 4), N)
    x = cuda.rand(N, dtype=cuda.float64)
    y = cuda.zeros(N, dtype=cuda.float64)
    if pinned:
        x, y = x.pin_memory(), y.pin_memory()
    M.vectorProduct(x, y)
    _permute(M, "columns", name)
    want = cuda.zeros(N, dtype=cuda.float64, device="cuda")
    M.vectorProduct(x.cuda(), want)
    for _ in range(2):
        y.fill_(float("nan"))
        M.vectorProduct(x, y)
        assert _same_bits(cuda, y, want.cpu())


@pytest.mark.parametrize("where", ["columns", "rows"])
@pytest.mark.parametrize("longest", [6, 400])  # substitutions by blocks and a warp per row
def test_factors_used_again(b2s_lib, cuda, where, longest):
    """ILU(0) factors are those of the matrix at the time they were made."""
    n, g = 3000, np.random.default_rng(8)
    cols = [np.unique(np.concatenate([[i], g.integers(0, n, g.integers(0, longest + 1))])) for i in range(n)]
    off = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    col = np.concatenate(cols).astype(np.int32)
    val = g.uniform(-1, 1, len(col))
    val[col == np.repeat(np.arange(n), np.diff(off))] = 2.0 * longest + 4.0
    M = b2s_lib.SparseMatrix.from_csr(off, col, val, n)
    P = b2s_lib.Preconditioner(M, "ilu0")
    b = cuda.rand(n, dtype=cuda.float64, device="cuda")
    before, after = cuda.zeros_like(b), cuda.zeros_like(b)
    P.solve(b, before)
    (M.permuteColumns if where == "columns" else M.permuteRows)(g.permutation(n).astype(np.int32))
    P.solve(b, after)
    assert _same_bits(cuda, before, after)
