"""Products through row patterns (one byte per row in place of the columns)
against the oracle, at the limits of what is kept as patterns: 255 and 256
patterns, rows of 64 and 65 elements, 2,040 and 2,400 offsets, empty rows, explicit zeros,
rectangular matrices, the smallest matrix that has patterns and odd row counts; every layout that reads patterns, row ranges, both value types;
and after the columns were permuted in place.

Each row within the forward error bound of its dot product,
2 (L + 3) u (|alpha| (|A| |x|)_i + |beta y0_i|)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAYOUTS = [("CSR", 0), ("Ellpack", 0), ("SlicedEllpack", 8), ("SlicedEllpack", 32), ("SlicedEllpack", 64),
           ("ChunkedEllpack", 0), ("BiEllpack", 0)]


N = 100000  # matrices below keep their columns


def _rows(length, offsets_of, cols, seed=0, zeros=False, rows=N):
    """Row i: the first length[i % len(length)] of offsets_of(i, k) + i inside [0, cols)."""
    g = np.random.default_rng(seed)
    i = np.arange(rows)
    width = int(np.max(length)) if np.size(length) else 0
    L = np.resize(np.asarray(length), rows)
    c = i[:, None] + offsets_of(i[:, None], np.arange(width)[None, :]) if width else np.zeros((rows, 0), np.int64)
    keep = (np.arange(width)[None, :] < L[:, None]) & (c >= 0) & (c < cols)
    off = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int32)
    col = c[keep].astype(np.int32)
    val = g.normal(size=len(col))
    if zeros and len(val):
        val[g.integers(0, len(val), len(val) // 9)] = 0.0
    return off, col, val, cols


def _stencil(n, offsets, cols=None, **kw):
    o = np.asarray(offsets, np.int64)
    return _rows([len(o)], lambda i, k: o[k] + 0 * i, n if cols is None else cols, rows=n, **kw)


def _distinct(patterns):
    """`patterns` distinct rows {0, 1 + i % patterns}."""
    return _rows([2], lambda i, k: np.where(k == 0, 0, 1 + i % patterns), N + patterns + 2)


CASES = {
    "one_row": lambda: _stencil(1, [0]),
    "tri_31": lambda: _stencil(31, [-1, 0, 1]),
    "five_below": lambda: _stencil(N - 1, [-300, -1, 0, 1, 300]),
    "five": lambda: _stencil(N, [-300, -1, 0, 1, 300]),
    "five_odd": lambda: _stencil(N + 33, [-300, -1, 0, 1, 300], seed=2),
    # whole slices of ChunkedEllpack: one chunk per row, which its pattern kernel needs
    "five_chunks": lambda: _stencil(391 * 256, [-300, -1, 0, 1, 300], seed=4),
    "seven_zeros": lambda: _stencil(N + 31, [-2500, -50, -1, 0, 1, 50, 2500], seed=3, zeros=True),
    "wide": lambda: _stencil(N, [0, 3, 90000], cols=N + 70000),
    "tall": lambda: _stencil(N + 1, [-90000, -3, 0], cols=N // 2),
    "empty_rows": lambda: _rows([0, 2, 2], lambda i, k: 500 * k, N + 600),
    "patterns_255": lambda: _distinct(255),
    "patterns_256": lambda: _distinct(256),
    "row_64": lambda: _rows([64] + [2] * 39, lambda i, k: k + 0 * i, N + 100),
    "row_65": lambda: _rows([65] + [2] * 39, lambda i, k: k + 0 * i, N + 100),
    "offsets_2040": lambda: _rows([60], lambda i, k: k + 2 * (i % 34), N + 200),
    "offsets_2400": lambda: _rows([60], lambda i, k: k + 2 * (i % 40), N + 200),
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
    n = N
    off, col, val, cols = _stencil(n, [-30, -1, 0, 1, 30])
    for iperm in (np.arange(n)[::-1].copy(), np.random.default_rng(2).permutation(n), np.roll(np.arange(n), 5)):
        iperm = iperm.astype(np.int32)
        M = b2s_lib.SparseMatrix.from_csr(off, col, val, cols, segments=segments)
        M.permuteColumns(iperm)
        _check(b2s_lib, cuda, oracle, M, (off, iperm[col].astype(np.int32), val, cols), "double", segments)


def test_layouts_that_keep_patterns(b2s_lib, cuda):
    """By the memory that a matrix holds before and after its columns are shuffled beyond any
    pattern: ChunkedEllpack in FP32 reads its columns faster, the others keep patterns."""
    from b2s._abi import MatrixInfo
    n = 391 * 256
    off, col, val, cols = _stencil(n, [-300, -1, 0, 1, 300])
    shuffle = np.random.default_rng(1).permutation(n).astype(np.int32)
    for segments, _ in LAYOUTS:
        for real in ("double", "float"):
            M = b2s_lib.SparseMatrix.from_csr(off, col, val, cols, segments=segments, real=real)
            before = M.info.device_bytes
            M.permuteColumns(shuffle)
            info = MatrixInfo()
            assert b2s_lib.lib.b2s_matrix_get_info(M.handle, C.byref(info)) == b2s_lib.OK
            after = info.device_bytes
            kept = not (segments == "ChunkedEllpack" and real == "float")
            assert (before - after >= n) == kept, (segments, real, before - after)
