"""Products through row patterns (one byte per row in place of the columns)
against the oracle, at the limits of what is kept as patterns: 255 and 256
patterns, rows of 64 and 65 elements, 2,048 offsets and more, empty rows,
explicit zeros, rectangular matrices, counts around the warp, row-group and
slice sizes; every layout that reads patterns, row ranges, both value types;
and after the columns were permuted in place.

Each row within the forward error bound of its dot product,
2 (L + 3) u (|alpha| (|A| |x|)_i + |beta y0_i|)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAYOUTS = [("CSR", 0), ("Ellpack", 0), ("SlicedEllpack", 8), ("SlicedEllpack", 32), ("SlicedEllpack", 64),
           ("ChunkedEllpack", 0), ("BiEllpack", 0)]


def _rows(cols_of, cols, seed=0, zeros=False):
    g = np.random.default_rng(seed)
    off = np.concatenate([[0], np.cumsum([len(c) for c in cols_of])]).astype(np.int32)
    col = np.concatenate([np.asarray(c, np.int32) for c in cols_of] + [np.zeros(0, np.int32)])
    val = g.normal(size=len(col))
    if zeros and len(val):
        val[g.integers(0, len(val), max(1, len(val) // 9))] = 0.0
    return off, col.astype(np.int32), val, cols


def _stencil(n, offsets, cols=None, **kw):
    cols = n if cols is None else cols
    return _rows([[i + o for o in offsets if 0 <= i + o < cols] for i in range(n)], cols, **kw)


def _distinct(n, patterns, seed=1):
    """`patterns` distinct rows {0, 1 + k}, the rest of the rows repeating them."""
    return _rows([[i, i + 1 + i % patterns] for i in range(n)], n + patterns + 2, seed)


CASES = {
    "one_row": lambda: _stencil(1, [0]),
    "tri_31": lambda: _stencil(31, [-1, 0, 1]),
    "five_4097": lambda: _stencil(4097, [-64, -1, 0, 1, 64]),
    "seven_33x": lambda: _stencil(33 * 67, [-67, -33, -1, 0, 1, 33, 67], seed=3, zeros=True),
    "wide": lambda: _stencil(700, [0, 3, 900], cols=1700),
    "tall": lambda: _stencil(1700, [-900, -3, 0], cols=700),
    "empty_rows": lambda: _rows([[] if i % 3 == 0 else [i // 3, 500 + i // 3] for i in range(1025)], 1100),
    "patterns_255": lambda: _distinct(2000, 255),
    "patterns_256": lambda: _distinct(2000, 256),
    "row_64": lambda: _rows([list(range(i, i + (64 if i % 40 == 0 else 2))) for i in range(640)], 800),
    "row_65": lambda: _rows([list(range(i, i + (65 if i % 40 == 0 else 2))) for i in range(640)], 800),
    "offsets_over": lambda: _rows([list(range(i, i + 1 + i % 66)) for i in range(1980)], 2100),
}


def _check(b2s_lib, cuda, oracle, M, csr, real, tag):
    off, col, val, cols = csr
    rows = len(off) - 1
    dt, u = (np.float64, 2.0 ** -53) if real == "double" else (np.float32, 2.0 ** -24)
    tdt = cuda.float64 if real == "double" else cuda.float32
    val = val.astype(dt).astype(np.float64)
    g = np.random.default_rng(5)
    x, y0 = g.uniform(-1, 1, cols).astype(dt), g.uniform(-1, 1, rows).astype(dt)
    row_of = np.repeat(np.arange(rows), np.diff(off))
    absax = np.bincount(row_of, weights=np.abs(val * x.astype(np.float64)[col]), minlength=rows)
    for alpha, beta, rb, re in [(1.0, 0.0, 0, 0), (-1.5, 0.5, 0, 0), (0.75, 1.0, rows // 3, rows // 3 + rows // 2 + 1),
                                (1.0, 0.0, rows // 64 * 32, 0)]:
        end = rows if re == 0 else min(re, rows)
        want = oracle.spmv("csr", "col", (off, col, val, cols), x.astype(np.float64), y0.astype(np.float64), alpha, beta,
                           rb, end)
        y = cuda.tensor(y0, dtype=tdt, device="cuda")
        M.vectorProduct(cuda.tensor(x, dtype=tdt, device="cuda"), y, alpha, beta, rb, end)
        y = y.cpu().numpy()
        inside = np.zeros(rows, bool)
        inside[rb:end] = True
        bound = 2.0 * (np.diff(off) + 3.0) * u * (abs(alpha) * absax + abs(beta * y0.astype(np.float64)))
        assert np.array_equal(y[~inside], y0[~inside]), (tag, rb, re)
        assert np.all(np.abs(y - want)[inside] <= bound[inside] + 1e-300), (tag, alpha, beta, rb, re)


@pytest.mark.parametrize("name", list(CASES))
@pytest.mark.parametrize("real", ["double", "float"])
def test_pattern_products(b2s_lib, cuda, oracle, name, real):
    csr = CASES[name]()
    for segments, ss in LAYOUTS:
        M = b2s_lib.SparseMatrix.from_csr(*csr[:3], csr[3], segments=segments, real=real, slice_size=ss)
        _check(b2s_lib, cuda, oracle, M, csr, real, (name, segments, ss))


@pytest.mark.parametrize("segments", ["CSR", "SlicedEllpack", "BiEllpack"])
def test_columns_permuted_in_place(b2s_lib, cuda, oracle, segments):
    n = 900
    off, col, val, cols = _stencil(n, [-30, -1, 0, 1, 30])
    for iperm in (np.arange(n)[::-1].copy(), np.random.default_rng(2).permutation(n), np.roll(np.arange(n), 5)):
        iperm = iperm.astype(np.int32)
        M = b2s_lib.SparseMatrix.from_csr(off, col, val, cols, segments=segments)
        M.permuteColumns(iperm)
        _check(b2s_lib, cuda, oracle, M, (off, iperm[col].astype(np.int32), val, cols), "double", segments)
