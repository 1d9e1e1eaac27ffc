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
