"""Assembly on both sides of the row length up to which rows are sorted in
shared memory (32 triplets) against the oracle: the longest row at and past the
limit, repeated columns, caller's capacities, the last row of a group of 32;
rows so long that the count of triplets stops early."""
import numpy as np
import pytest

import fixtures as F
from test_assembly_gpu import LAYOUTS, REAL, _check

pytestmark = pytest.mark.gpu


def _triplets(longest, rows, cols, seed):
    g = np.random.default_rng(seed)
    length = g.integers(0, 6, rows)
    length[[0, 31, rows - 1]] = [longest, 1, longest]
    ri = np.repeat(np.arange(rows), length).astype(np.int32)
    ci = g.integers(0, cols, len(ri)).astype(np.int32)  # 40 columns: repeats in the long rows
    order = g.permutation(len(ri))
    return ri[order], ci[order], g.normal(size=len(ri))


@pytest.mark.parametrize("longest", [1, 31, 32, 33, 70])
@pytest.mark.parametrize("fmt", ["csr", "slicedellpack", "biellpack"])
@pytest.mark.parametrize("dup", ["set", "add"])
def test_rows_at_the_limit(b2s_lib, cuda, oracle, longest, fmt, dup):
    for rows, real in ((33, "f64"), (200, "f32")):
        ri, ci, v = _triplets(longest, rows, 40, longest + rows)
        want = oracle.from_coo(fmt, "col", rows, 40, ri, ci, v, dup == "add", real)
        M = b2s_lib.SparseMatrix.from_coo(rows, 40, ri, ci, v, segments=LAYOUTS[fmt], real=REAL[real], duplicates=dup,
                                          slice_size=F.SLICE.get(fmt, 0))
        _check(M, want, fmt)


@pytest.mark.parametrize("longest", [32, 33])
def test_capacities_of_the_caller(b2s_lib, cuda, oracle, longest):
    rows = 100
    ri, ci, v = _triplets(longest, rows, 40, 9)
    caps = np.bincount(ri, minlength=rows).astype(np.int32) + 1
    want = oracle.from_coo("slicedellpack", "col", rows, 40, ri, ci, v, True, "f64", caps=caps)
    M = b2s_lib.SparseMatrix.from_coo(rows, 40, ri, ci, v, segments="SlicedEllpack", duplicates="add",
                                      row_capacities=caps)
    _check(M, want, "slicedellpack")
    caps[0] = 1  # fewer than the row's distinct columns
    with pytest.raises(b2s_lib.B2SError) as e:
        b2s_lib.SparseMatrix.from_coo(rows, 40, ri, ci, v, segments="SlicedEllpack", duplicates="add",
                                      row_capacities=caps)
    assert "row number 0" in str(e.value)


@pytest.mark.parametrize("real", ["f64", "f32"])
@pytest.mark.parametrize("at", [0, 20000, 39999])
@pytest.mark.parametrize("dup", ["set", "add"])
def test_one_long_row_among_short_ones(b2s_lib, cuda, oracle, real, at, dup):
    """The count stops somewhere inside the list: whatever it saw, the result is the sort's."""
    rows, cols, g = 40000, 5000, np.random.default_rng(at)
    length = g.integers(0, 4, rows)
    length[at] = 30000
    ri = np.repeat(np.arange(rows), length).astype(np.int32)
    ci = g.integers(0, cols, len(ri)).astype(np.int32)
    order = g.permutation(len(ri))
    ri, ci, v = ri[order], ci[order], g.normal(size=len(ri))
    want = oracle.from_coo("csr", "col", rows, cols, ri, ci, v, dup == "add", real)
    M = b2s_lib.SparseMatrix.from_coo(rows, cols, ri, ci, v, segments="CSR", real=REAL[real], duplicates=dup)
    _check(M, want, "csr")
    ri[len(ri) // 2] = rows  # an index that the count may never have come to
    with pytest.raises(b2s_lib.B2SError) as e:
        b2s_lib.SparseMatrix.from_coo(rows, cols, ri, ci, v, segments="CSR", real=REAL[real], duplicates=dup)
    assert "outside" in str(e.value)


def test_more_triplets_than_short_rows_hold(b2s_lib, cuda, oracle):
    """More than 32 triplets per row on average: no count at all."""
    g = np.random.default_rng(3)
    ri, ci, v = (g.integers(0, 30, 3000).astype(np.int32), g.integers(0, 70, 3000).astype(np.int32), g.normal(size=3000))
    want = oracle.from_coo("slicedellpack", "col", 30, 70, ri, ci, v, True, "f64")
    M = b2s_lib.SparseMatrix.from_coo(30, 70, ri, ci, v, segments="SlicedEllpack", duplicates="add")
    _check(M, want, "slicedellpack")
