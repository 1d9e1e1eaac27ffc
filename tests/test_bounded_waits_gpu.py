"""Bounded waits between the blocks of a kernel: what a call does when they run
out (the limits are set so low that they do), and when another kernel keeps the
device busy meanwhile."""
import threading

import numpy as np
import pytest

from test_resident_gpu import _spd

pytestmark = pytest.mark.gpu


def _solver(b2s_lib, kind, M, precond=None, mixed=False):
    s = getattr(b2s_lib, kind)()
    s.setMatrix(M)
    s.setPreconditioner(precond)
    s.setConvergenceResidue(1e-10)
    s.setPrecision(mixed)
    return s


def _limit(b2s_lib, s, looks):
    s._ensure()
    assert b2s_lib.lib.b2s_solver_set_wait_limit(s._solver, looks) == b2s_lib.OK


@pytest.mark.parametrize("kind", ["CG", "BICGStab"])
@pytest.mark.parametrize("precond", [None, "diagonal"])
@pytest.mark.parametrize("mixed", [False, True])
def test_solve_goes_on_without_the_resident_kernel(b2s_lib, cuda, oracle, kind, precond, mixed):
    """One poll, and as many as let some meetings of all blocks pass and others not."""
    n = 20000  # 79 blocks, beyond one cluster
    csr = _spd(n, [1, 30])
    b = np.random.default_rng(6).uniform(-1, 1, n)
    want = oracle.solve(kind.lower(), csr, b, rtol=1e-10, precond=precond is not None)
    M = b2s_lib.SparseMatrix.from_csr(*csr[:3], n, keep_fp32_copy=mixed)
    bd = cuda.tensor(b, device="cuda")
    # A is a Laplacian + 0.5 I: an error is at most twice its residual, the oracle's solution is as far off
    d = csr[2][csr[1] == np.repeat(np.arange(n), np.diff(csr[0]))]
    bound = 4e-10 * (np.linalg.norm(b) if precond is None else np.max(d) * np.linalg.norm(b / d))
    s = _solver(b2s_lib, kind, M, precond, mixed)
    for looks in (0, 1, 4, 8, 12, 20, 0):
        _limit(b2s_lib, s, looks)
        x = cuda.zeros_like(bd)
        assert s.solve(bd, x), looks
        assert np.max(np.abs(x.cpu().numpy() - want["x"])) <= bound, looks


@pytest.mark.parametrize("kind", ["CG", "BICGStab"])
def test_solves_beside_a_long_kernel(b2s_lib, cuda, kind):
    """A batch holds shared memory on every SM for some hundred milliseconds;
    solves on another stream have the same result as alone or, where a wait
    ran out, one as good."""
    from b2s import workloads as W
    n = 40000
    csr = _spd(n, [1, 200])
    M = b2s_lib.SparseMatrix.from_csr(*csr[:3], n)
    x0 = np.random.default_rng(1).uniform(-1, 1, n)
    b = np.bincount(np.repeat(np.arange(n), np.diff(csr[0])), weights=csr[2] * x0[csr[1]], minlength=n)
    bd = cuda.tensor(b, device="cuda")
    s = _solver(b2s_lib, kind, M)
    off, col, val, rp, nr = W.batched_poisson2d(320, seed=5, lo=64, hi=160)
    bt = b2s_lib.BatchedCG(off, col, val, rp, nr, tol=1e-9, cluster_size=8)
    B = cuda.rand(bt.vector_length, dtype=cuda.float64, device="cuda")
    alone, mixed = cuda.zeros_like(B), cuda.zeros_like(B)
    side = cuda.cuda.Stream()
    assert bt.solve(B, alone, stream=side)
    cuda.cuda.synchronize()
    ok, running = [], threading.Event()

    def batch():
        running.set()
        for _ in range(3):
            mixed.zero_()
            cuda.cuda.synchronize()
            ok.append(bt.solve(B, mixed, stream=side))

    t = threading.Thread(target=batch)
    t.start()
    running.wait()
    solves = 0
    while t.is_alive() or solves == 0:
        x = cuda.zeros_like(bd)
        assert s.solve(bd, x)
        assert float((x.cpu() - cuda.tensor(x0)).abs().max()) <= 2e-10 * np.linalg.norm(b)
        solves += 1
    t.join()
    assert ok == [True] * 3
    assert cuda.equal(alone, mixed)


def _chain(n):
    i = np.repeat(np.arange(n, dtype=np.int64), 3).reshape(n, 3) + np.array([-1, 0, 1])
    keep = (i >= 0) & (i < n)
    off = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.int32)
    val = np.random.default_rng(3).uniform(-1, 1, i.shape)
    val[:, 1] = 4.0
    return off, i[keep].astype(np.int32), val[keep], n


def test_substitutions_give_up_and_recover(b2s_lib, cuda, oracle):
    csr = _chain(20000)  # three blocks
    n = csr[3]
    M = b2s_lib.SparseMatrix.from_csr(*csr[:3], n)
    b = np.random.default_rng(4).uniform(-1, 1, n)
    want = oracle.ilu0_apply(csr, b, "f64")
    P = b2s_lib.Preconditioner(M, "ilu0")
    bd = cuda.tensor(b, device="cuda")
    x = cuda.zeros_like(bd)
    for _ in range(2):
        assert b2s_lib.lib.b2s_precond_set_wait_limit(P._h, 1) == b2s_lib.OK
        with pytest.raises(b2s_lib.B2SError) as e:
            P.solve(bd, x)
        assert "gave up" in str(e.value)
        assert b2s_lib.lib.b2s_precond_set_wait_limit(P._h, 0) == b2s_lib.OK
        P.solve(bd, x)
        assert np.array_equal(x.cpu().numpy(), want)
    s = _solver(b2s_lib, "BICGStab", M, "ilu0")
    _limit(b2s_lib, s, 1)
    with pytest.raises(b2s_lib.B2SError) as e:
        s.solve(bd, x)
    assert "gave up" in str(e.value)
    _limit(b2s_lib, s, 0)
    x.zero_()
    assert s.solve(bd, x)


def test_substitutions_of_a_long_chain(b2s_lib, cuda):
    """Millions of dependent steps take longer than a fixed limit: the limits follow the chain."""
    n = 3_700_000
    off, col, val, _ = _chain(n)
    val[:] = np.where(col == np.repeat(np.arange(n), np.diff(off)), 4.0, -1.0)
    P = b2s_lib.Preconditioner(b2s_lib.SparseMatrix.from_csr(off, col, val, n), "ilu0")
    b = np.full(n, 2.0)
    b[[0, -1]] = 3.0  # A times 1, and for a tridiagonal matrix ILU(0) is exact
    x = cuda.zeros(n, dtype=cuda.float64, device="cuda")
    P.solve(cuda.tensor(b, device="cuda"), x)
    assert float((x - 1).abs().max()) <= 1e-14  # dominant by 2: each step halves an error, a few ulp are left


@pytest.mark.parametrize("n", [5, 3001, 20001])  # one block, one cluster, all blocks
@pytest.mark.parametrize("mixed", [False, True])
def test_bicgstab_restarts_within_the_time_limit(b2s_lib, cuda, n, mixed):
    """4 I + a cyclic shift, b = e_0: after the first step r is orthogonal to r_ast exactly, so
    BiCGStab restarts. Restarts count no iteration: only the clock ends a solve of nothing else."""
    off = np.arange(0, 2 * n + 1, 2, dtype=np.int32)
    col = np.sort(np.stack([np.arange(n), (np.arange(n) - 1) % n], axis=1), axis=1).astype(np.int32)
    val = np.where(col == np.arange(n)[:, None], 4.0, 1.0)
    M = b2s_lib.SparseMatrix.from_csr(off, col.reshape(-1), val.reshape(-1), n, keep_fp32_copy=mixed)
    s = _solver(b2s_lib, "BICGStab", M, mixed=mixed)
    s._ensure()
    b = cuda.zeros(n, dtype=cuda.float64, device="cuda")
    b[0] = 1.0
    x = cuda.zeros_like(b)
    assert b2s_lib.lib.b2s_solver_set_time_limit(s._solver, 1e-9) == b2s_lib.OK
    with pytest.raises(b2s_lib.B2SError) as e:
        s.solve(b, x)
    assert "exceeded" in str(e.value)
    assert b2s_lib.lib.b2s_solver_set_time_limit(s._solver, 0.0) == b2s_lib.OK
    x.zero_()
    assert s.solve(b, x)
    assert float((b - 4.0 * x - cuda.roll(x, 1)).norm()) <= 2e-10
