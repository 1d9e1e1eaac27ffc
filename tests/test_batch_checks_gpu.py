"""Batches are refused at creation when a row's offsets are out of order or a
column lies outside its system: the kernel turns columns into places of the
system's vectors, in another block's shared memory among others."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [5, 0, 40, 1, 0, 33]  # rows of each system, empty ones among them


def _batch():
    """Tridiagonal systems as the diagonal blocks of one matrix."""
    rp = np.concatenate([[0], np.cumsum(SIZES)]).astype(np.int64)
    cols, count = [], []
    for s, n in enumerate(SIZES):
        for i in range(n):
            c = [j for j in (i - 1, i, i + 1) if 0 <= j < n]
            cols += [int(rp[s]) + j for j in c]
            count.append(len(c))
    off = np.concatenate([[0], np.cumsum(count)]).astype(np.int32)
    col = np.array(cols, np.int32)
    val = np.where(col == np.repeat(np.arange(len(count)), count), 4.0, -1.0)
    return off, col, val, rp, np.array([1, 2, 8, 3, 1, 2], np.int32)


def _column(row, value):
    def change(off, col):
        col[off[row]] = value
    return change


def _offset(row, value):
    def change(off, col):
        off[row] = value
    return change


# the systems' first rows are 0, 5, 5, 45, 46 and 46
BAD = {
    "the system before": _column(5, 4),
    "the system after": _column(44, 45),
    "one row alone": _column(45, 46),
    "past the last system": _column(78, 79),
    "negative": _column(0, -1),
    "far": _column(20, 2 ** 31 - 1),
    "offsets fall": _offset(10, 3),
    "offset past the end": _offset(10, 10 ** 6),
    "negative offset": _offset(3, -4),
}


@pytest.mark.parametrize("name", list(BAD))
@pytest.mark.parametrize("device", [True, False])
def test_refused(b2s_lib, cuda, name, device):
    off, col, val, rp, nr = _batch()
    BAD[name](off, col)
    csr = [cuda.tensor(a, device="cuda") for a in (off, col, val)] if device else [off, col, val]
    with pytest.raises(b2s_lib.B2SError) as e:
        b2s_lib.BatchedCG(*csr, rp, nr)
    assert "outside its system" in str(e.value)


def test_empty_systems_are_accepted(b2s_lib, cuda):
    off, col, val, rp, nr = _batch()
    bt = b2s_lib.BatchedCG(off, col, val, rp, nr, tol=1e-12, cluster_size=2)
    x = np.random.default_rng(1).uniform(-1, 1, bt.vector_length)
    b = np.zeros_like(x)
    for s, n in enumerate(SIZES):
        v = slice(int(bt.vec_off[s]), int(bt.vec_off[s + 1]))
        xs = x[v].reshape(n, -1) if n else x[v].reshape(0, 1)
        y = 4.0 * xs
        y[1:] -= xs[:-1]
        y[:-1] -= xs[1:]
        b[v] = y.reshape(-1)
    got = cuda.zeros(bt.vector_length, dtype=cuda.float64, device="cuda")
    assert bt.solve(cuda.tensor(b, device="cuda"), got)
    assert np.max(np.abs(got.cpu().numpy() - x)) <= 1e-10  # condition number below 3, residue 1e-12
