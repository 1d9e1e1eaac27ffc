"""The triangular substitutions by blocks of rows against the oracle's ILU(0)
(the operations of TNL's host loops in their order): equal bits.

Patterns where a block plan can go wrong: one row, sizes around a batch of 32
rows and around one block, chains (one row per level), rows of no, few and
many entries, dependencies on far blocks, and rows too long for a lane or too
uneven for a batch (the warp-per-row kernel)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _band(n, offsets, seed=0):
    """Diagonally dominant matrix with the given diagonals."""
    g = np.random.default_rng(seed)
    cols = [np.array(sorted({i} | {i + o for o in offsets if 0 <= i + o < n}), np.int32) for i in range(n)]
    off = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    col = np.concatenate(cols)
    val = g.uniform(-1, 1, len(col))
    val[col == np.repeat(np.arange(n), np.diff(off))] = 4.0 + len(offsets)
    return off, col, val, n


def _random(n, longest, seed):
    g = np.random.default_rng(seed)
    cols = [np.unique(np.concatenate([[i], g.integers(0, n, g.integers(0, longest + 1))])).astype(np.int32)
            for i in range(n)]
    off = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    col = np.concatenate(cols)
    val = g.uniform(-1, 1, len(col))
    val[col == np.repeat(np.arange(n), np.diff(off))] = 2.0 * longest + 4.0
    return off, col, val, n


def _uneven(n):
    """Rows past the first 128 depend on row 0, every 32nd of them on rows 0 to 99 too."""
    cols = [np.arange(100 if i % 32 == 0 else 1) for i in range(n)]
    cols = [np.array([i]) if i < 128 else np.append(c, i) for i, c in enumerate(cols)]
    off = np.concatenate([[0], np.cumsum([len(c) for c in cols])]).astype(np.int32)
    col = np.concatenate(cols).astype(np.int32)
    val = np.random.default_rng(5).uniform(-1, 1, len(col))
    val[off[1:] - 1] = 200.0
    return off, col, val, n


CASES = {
    "one_row": lambda: _band(1, []),
    "diagonal": lambda: _band(70, []),
    "chain_31": lambda: _band(31, [-1, 1]),
    "chain_5000": lambda: _band(5000, [-1, 1]),  # a level per row
    "chain_20000": lambda: _band(20000, [-1, 1]),  # and across three blocks
    "narrow_17000": lambda: _band(17000, [-3, -1, 1, 3]),  # a few rows per level and block
    "far_8193": lambda: _band(8193, [-4096, -1, 1, 4096, 8000]),
    "grid_4097": lambda: _band(4097, [-64, -1, 1, 64]),
    "random_short": lambda: _random(20000, 6, 1),
    "random_ragged": lambda: _random(9000, 40, 2),
    # a row of 100 among 31 of one entry in every batch
    "uneven": lambda: _uneven(4096),
    "long_rows": lambda: _random(3000, 400, 3),  # the warp-per-row kernel
}


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("real", ["f64", "f32"])
def test_block_substitutions_bitwise(b2s_lib, cuda, oracle, name, real):
    csr = CASES[name]()
    n = csr[3]
    b = np.random.default_rng(7).uniform(-1, 1, n)
    want = oracle.ilu0_apply(csr, b, real)
    dt = cuda.float64 if real == "f64" else cuda.float32
    A = b2s_lib.SparseMatrix.from_csr(*csr[:3], n, real="double" if real == "f64" else "float")
    P = b2s_lib.Preconditioner(A, "ilu0")
    bd = cuda.tensor(b, dtype=dt, device="cuda")
    x = cuda.zeros_like(bd)
    for _ in range(3):  # the passes put each other's scratch back
        P.solve(bd, x)
        assert np.array_equal(x.cpu().numpy().astype(np.float64), want)
    P.solve(x.copy_(bd), x)  # in place
    assert np.array_equal(x.cpu().numpy().astype(np.float64), want)


def test_block_substitutions_not_a_number(b2s_lib, cuda):
    """NaN and infinity go through; the value that marks a pending row ends as a NaN."""
    n = 3000
    A = b2s_lib.SparseMatrix.from_csr(*_band(n, [-1, 1])[:3], n)
    P = b2s_lib.Preconditioner(A, "ilu0")
    for bad in (float("nan"), float("inf")):
        b = cuda.ones(n, dtype=cuda.float64, device="cuda")
        b[1500] = bad
        x = cuda.zeros_like(b)
        P.solve(b, x)
        assert not bool(cuda.isfinite(x[1500]))
    b = cuda.ones(n, dtype=cuda.float64, device="cuda")
    b.view(cuda.int64)[0] = 0xFFF3B25D5EA10F0F - (1 << 64)
    x = cuda.zeros_like(b)
    P.solve(b, x)
    assert bool(cuda.isnan(x).all())


def test_memory_of_a_chain(b2s_lib, cuda, oracle):
    """One row per level: the plans of both triangles stay near the factors' size."""
    n = 400_000
    g = np.random.default_rng(2)
    i = np.repeat(np.arange(n), 3).reshape(n, 3) + np.array([-1, 0, 1])
    keep = (i >= 0) & (i < n)
    off = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int32)
    val = g.uniform(-1, 1, i.shape)
    val[:, 1] = 4.0
    csr = (off, i[keep].astype(np.int32), val[keep], n)
    A = b2s_lib.SparseMatrix.from_csr(*csr[:3], n)
    cuda.cuda.synchronize()
    before = cuda.cuda.mem_get_info()[0]
    P = b2s_lib.Preconditioner(A, "ilu0")
    held = before - cuda.cuda.mem_get_info()[0]
    # per row: 3 values of the factors, position of the diagonal, flag, order, two scratch values (52 bytes),
    # and in each plan a batch (16), row, length, diagonal (16) and one slot (12): 140 bytes
    assert held <= 160 * n + (48 << 20), held / n  # allocations take whole 2 MB pages
    b = g.uniform(-1, 1, n)
    x = cuda.zeros(n, dtype=cuda.float64, device="cuda")
    P.solve(cuda.tensor(b, device="cuda"), x)
    assert np.array_equal(x.cpu().numpy(), oracle.ilu0_apply(csr, b, "f64"))
