"""The work a program does with this framework, as measurable cases.

Three families, over the matrices that the benchmark and the tests use
(``b2s.workloads``: 2D 5-point Poisson, 3D 7-point Laplacian, variable
coefficient diffusion, upwind convection-diffusion, irregular rows), built
here on the GPU so that a case is prepared quickly:

* ``spmv``  -- ``SparseMatrix.vectorProduct`` on device vectors: every
  layout, FP64 and FP32, with and without multiplicators, from a 1k-row
  system that is all latency to matrices well beyond the L2 cache;
* ``solve`` -- ``CG`` / ``BICGStab`` / ``GMRES`` ``solve( b, x )`` to a
  residue of 1e-10: plain FP64 and mixed precision, without preconditioner,
  with the diagonal one and with ILU(0);
* ``batch`` -- ``BatchedCG``: many small systems of uneven sizes in a launch;
* ``assemble`` -- a matrix from triplets in no particular order followed by
  its first product, as one step of a program whose matrix changes.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "tnl-dev_b200"))
import b2s  # noqa: E402


# ---------------------------------------------------------------------------
# cases
def listed():
    return [
        # one product of a small 2D system, as an application's own solver loop
        # calls it thousands of times: launch and latency
        dict(name="spmv_csr_f64_poisson256", kind="spmv", matrix="poisson2d", nx=256, ny=256, nz=1, segments="CSR",
             real="double", keeper="plain"),
        # the headline product: CSR, FP64, 2.1M rows, larger than L2
        dict(name="spmv_csr_f64_laplace128", kind="spmv", matrix="laplace3d", nx=128, ny=128, nz=128, segments="CSR",
             real="double", keeper="plain"),
        # a padded layout in single precision on an odd-sized grid, y updated in place
        dict(name="spmv_biell_f32_laplace", kind="spmv", matrix="laplace3d", nx=129, ny=127, nz=121,
             segments="BiEllpack", real="float", keeper="scaled"),
        # irregular rows (log-normal lengths, uniform columns): CSR and the layout
        # that TNL offers for such rows
        dict(name="spmv_csr_f64_irregular2m", kind="spmv", matrix="irregular", nx=2_000_000, ny=1, nz=1,
             segments="CSR", real="double", keeper="plain"),
        dict(name="spmv_chunked_f32_irregular", kind="spmv", matrix="irregular", nx=700_001, ny=1, nz=1,
             segments="ChunkedEllpack", real="float", keeper="plain"),
        # small solve, the plain method on its smallest configured system
        dict(name="cg_f64_poisson256", kind="solve", solver="cg", matrix="poisson2d", nx=256, ny=256, nz=1,
             segments="CSR", mixed=False, precond="none"),
        # the mixed-precision solve of the largest SPD system
        dict(name="cg_mixed_diffusion160", kind="solve", solver="cg", matrix="diffusion3d", nx=160, ny=160, nz=160,
             segments="CSR", mixed=True, precond="none"),
        # nonsymmetric, short recurrence, FP64, on sliced storage
        dict(name="bicgstab_f64_convdiff128", kind="solve", solver="bicgstab", matrix="convdiff3d", nx=128, ny=128,
             nz=128, segments="SlicedEllpack", mixed=False, precond="none"),
        # nonsymmetric, long recurrence, mixed precision, a middle-sized ragged grid
        dict(name="gmres_mixed_convdiff", kind="solve", solver="gmres", matrix="convdiff3d", nx=101, ny=90, nz=83,
             segments="CSR", mixed=True, precond="none"),
        # preconditioned: incomplete factors, whose substitutions are chains of dependencies
        dict(name="bicgstab_ilu0_convdiff64", kind="solve", solver="bicgstab", matrix="convdiff3d", nx=64, ny=64,
             nz=64, segments="CSR", mixed=False, precond="ilu0"),
        # many small systems, 1 to 8 right-hand sides each
        dict(name="batch_512_systems", kind="batch", systems=512, lo=32, hi=256),
        # assembly from unordered triplets and the first product
        dict(name="assemble_poisson1500", kind="assemble", matrix="poisson2d", nx=1500, ny=1333, nz=1,
             segments="CSR", real="double"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(rng, matrix, rows):
    """Ragged grid dimensions with about `rows` points."""
    if matrix == "irregular":
        return rows, 1, 1
    d = 2 if matrix == "poisson2d" else 3
    side = rows ** (1.0 / d)
    dims = [max(3, int(round(side * rng.uniform(0.8, 1.25)))) for _ in range(d)]
    return tuple(dims + [1] * (3 - d))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv", "solve", "solve", "solve", "batch", "assemble"])
    if kind == "spmv":
        m = rng.choice(["poisson2d", "laplace3d", "irregular"])
        layouts = ["CSR", "CSR", "SlicedEllpack", "ChunkedEllpack", "BiEllpack"]
        if m != "irregular":
            layouts += ["Ellpack", "Multidiagonal"]
        nx, ny, nz = _grid(rng, m, _log(rng, 1000, 4_000_000 if m != "irregular" else 2_000_000))
        return dict(kind=kind, matrix=m, nx=nx, ny=ny, nz=nz, segments=rng.choice(layouts),
                    real=rng.choice(["double", "float"]), keeper=rng.choice(["plain", "plain", "scaled"]))
    if kind == "solve":
        solver = rng.choice(["cg", "bicgstab", "gmres"])
        m = rng.choice(["poisson2d", "diffusion3d"]) if solver == "cg" else "convdiff3d"
        mixed = rng.random() < 0.4
        precond = "none" if mixed else rng.choice(["none", "diagonal", "ilu0"])
        top = 300_000 if m == "poisson2d" else 3_000_000
        if precond == "ilu0":  # an application walks chains as long as the grid's sides
            top = 20_000 if m == "poisson2d" else 200_000
        nx, ny, nz = _grid(rng, m, _log(rng, 1000, top))
        return dict(kind=kind, solver=solver, matrix=m, nx=nx, ny=ny, nz=nz,
                    segments=rng.choice(["CSR", "CSR", "SlicedEllpack"]), mixed=mixed, precond=precond)
    if kind == "batch":
        lo = rng.randint(16, 64)
        return dict(kind=kind, systems=_log(rng, 16, 600), lo=lo, hi=rng.randint(lo + 8, 256))
    nx, ny, nz = _grid(rng, "poisson2d", _log(rng, 1000, 3_000_000))
    return dict(kind=kind, matrix="poisson2d", nx=nx, ny=ny, nz=nz, segments=rng.choice(["CSR", "SlicedEllpack"]),
                real=rng.choice(["double", "double", "float"]))


# ---------------------------------------------------------------------------
# matrices, built on the GPU: (offsets int32, columns int32, values float64, rows of the nonzeros int64)
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _grid_of(case):
    return case["nz"], case["ny"], case["nx"]  # C order: x fastest


def _stencil(case, g):
    """Rows of the grid operator, columns ascending in each row."""
    nz, ny, nx = _grid_of(case)
    n = nx * ny * nz
    m = case["matrix"]
    i = torch.arange(n, device="cuda", dtype=torch.int64)
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    axes = [(x, nx, 1), (y, ny, nx)] + ([(z, nz, nx * ny)] if m != "poisson2d" else [])
    lower, upper = [], []
    diag = torch.zeros(n, device="cuda", dtype=torch.float64)
    if m == "convdiff3d":  # unit velocity of cell Peclet number 10, upwinded
        v = torch.randn(3, generator=g, device="cuda", dtype=torch.float64)
        v = (10.0 * v / v.norm()).tolist()
    for d, (c, size, step) in enumerate(axes):
        if m == "diffusion3d":  # a coefficient exp(N(0, 1)) on every cell face
            shape = [nz, ny, nx]
            shape[2 - d] += 1
            k = torch.exp(torch.randn(shape, generator=g, device="cuda", dtype=torch.float64))
            lo = k.narrow(2 - d, 0, size).reshape(-1)
            hi = k.narrow(2 - d, 1, size).reshape(-1)
            diag = diag + lo + hi
        elif m == "convdiff3d":
            lo = torch.full((n,), 1.0 + max(v[d], 0.0), device="cuda", dtype=torch.float64)
            hi = torch.full((n,), 1.0 + max(-v[d], 0.0), device="cuda", dtype=torch.float64)
            diag = diag + lo + hi
        else:
            lo = hi = torch.ones(n, device="cuda", dtype=torch.float64)
            diag = diag + 2.0
        lower.append((c > 0, i - step, -lo))
        upper.append((c < size - 1, i + step, -hi))
    full = [(torch.ones_like(i, dtype=torch.bool), i, diag)]
    terms = lower[::-1] + full + upper
    keep = torch.stack([t[0] for t in terms], dim=1)
    cols = torch.stack([t[1] for t in terms], dim=1)[keep].to(torch.int32)
    vals = torch.stack([t[2] for t in terms], dim=1)[keep]
    count = keep.sum(dim=1)
    return count, cols, vals


def _irregular(case, g):
    """Log-normal row lengths (median 12), uniform columns without repeats, N(0, 1) values."""
    n = case["nx"]
    count = torch.exp(torch.randn(n, generator=g, device="cuda", dtype=torch.float64) + math.log(12.0)).round()
    count = count.clamp(1, min(2048, n // 2)).to(torch.int64)
    row = torch.repeat_interleave(torch.arange(n, device="cuda", dtype=torch.int64), count)
    col = torch.randint(0, n, (row.numel(),), generator=g, device="cuda", dtype=torch.int64)
    key = torch.unique(row * n + col)  # sorted; the few repeats are dropped
    row, col = key // n, key % n
    vals = torch.randn(key.numel(), generator=g, device="cuda", dtype=torch.float64)
    return torch.bincount(row, minlength=n), col.to(torch.int32), vals


def _csr(case, g):
    count, cols, vals = _irregular(case, g) if case["matrix"] == "irregular" else _stencil(case, g)
    off = torch.zeros(count.numel() + 1, device="cuda", dtype=torch.int64)
    torch.cumsum(count, 0, out=off[1:])
    row = torch.repeat_interleave(torch.arange(count.numel(), device="cuda", dtype=torch.int64), count)
    return off.to(torch.int32), cols, vals, row


def _times(csr, x):
    """A x in plain torch, 64 bits, row by row in the row's order."""
    off, cols, vals, _ = csr
    return torch.segment_reduce(vals * x[cols.long()], "sum", offsets=off.long())


def _uniform(n, g, dtype=torch.float64):
    return (2.0 * torch.rand(n, generator=g, device="cuda", dtype=torch.float64) - 1.0).to(dtype)


KEEPERS = {"plain": (1.0, 0.0), "scaled": (-0.75, 0.5)}


def _spmv_inputs(case, seed):
    g = _gen(seed)
    csr = _csr(case, g)
    n = csr[0].numel() - 1
    dt = torch.float64 if case["real"] == "double" else torch.float32
    return csr, _uniform(n, g, dt), _uniform(n, g, dt)


def _solve_inputs(case, seed):
    """A x = b with a known x: entries uniform around 1."""
    g = _gen(seed)
    csr = _csr(case, g)
    x = 1.0 + 0.5 * _uniform(csr[0].numel() - 1, g)
    return csr, x, _times(csr, x)


def _batch_inputs(case, seed):
    """The block-diagonal batch: system s a shifted 5-point Laplacian on an
    nx_s x ny_s grid, right-hand sides interleaved per system. The sizes are
    the case's, the shifts and right-hand sides the seed's."""
    k = case["systems"]
    r = np.random.Generator(np.random.Philox(1000 * k + case["lo"] + 7 * case["hi"]))
    nx, ny = r.integers(case["lo"], case["hi"] + 1, k), r.integers(case["lo"], case["hi"] + 1, k)
    nrhs = r.integers(1, 9, k).astype(np.int32)
    shift = np.random.Generator(np.random.Philox(int(seed) + 5)).uniform(0.0, 0.1, k)
    rows = (nx * ny).astype(np.int64)
    row_ptr = np.concatenate([[0], np.cumsum(rows)]).astype(np.int64)
    cu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    sys_of = torch.repeat_interleave(torch.arange(k, device="cuda"), cu(rows))
    i = torch.arange(int(row_ptr[-1]), device="cuda", dtype=torch.int64)
    loc = i - cu(row_ptr)[sys_of]
    sx, sy = cu(nx)[sys_of], cu(ny)[sys_of]
    x, y = loc % sx, loc // sx
    keep = torch.stack([y > 0, x > 0, x >= 0, x < sx - 1, y < sy - 1], dim=1)
    cols = torch.stack([i - sx, i - 1, i, i + 1, i + sx], dim=1)[keep].to(torch.int32)
    vals = torch.full((i.numel(), 5), -1.0, device="cuda", dtype=torch.float64)
    vals[:, 2] = 4.0 + cu(shift)[sys_of]
    count = keep.sum(dim=1)
    off = torch.zeros(i.numel() + 1, device="cuda", dtype=torch.int64)
    torch.cumsum(count, 0, out=off[1:])
    b = _uniform(int((rows * nrhs).sum()), _gen(seed))
    return off.to(torch.int32), cols, vals[keep], row_ptr, nrhs, nx, ny, shift, b


def _assemble_inputs(case, seed):
    g = _gen(seed)
    off, cols, vals, row = _csr(case, g)
    # every element's value is its own, and the triplets come in no order
    vals = vals * (1.0 + 0.25 * _uniform(vals.numel(), g))
    dt = torch.float64 if case["real"] == "double" else torch.float32
    order = torch.randperm(vals.numel(), generator=g, device="cuda")
    x = _uniform(off.numel() - 1, g, dt)
    return (off, cols, vals.to(dt), row), order, x


# ---------------------------------------------------------------------------
SOLVERS = {"cg": b2s.CG, "bicgstab": b2s.BICGStab, "gmres": b2s.GMRES}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        (off, cols, vals, _), x, y = _spmv_inputs(case, seed)
        A = b2s.SparseMatrix.from_csr(off, cols, vals, segments=case["segments"], real=case["real"])
        alpha, beta = KEEPERS[case["keeper"]]
        return dict(kind=kind, A=A, x=x, y=y, alpha=alpha, beta=beta)
    if kind == "solve":
        (off, cols, vals, _), _, b = _solve_inputs(case, seed)
        A = b2s.SparseMatrix.from_csr(off, cols, vals, segments=case["segments"], real="double",
                                      keep_fp32_copy=bool(case["mixed"]))
        s = SOLVERS[case["solver"]]()
        s.setMatrix(A)
        s.setConvergenceResidue(1e-10)
        s.setPreconditioner(case["precond"])
        s.setPrecision(bool(case["mixed"]))
        if case["solver"] == "gmres":
            s.setup({"gmres-variant": "CGSR", "gmres-restarting-min": 30, "gmres-restarting-max": 30})
        return dict(kind=kind, solver=s, b=b, x=torch.zeros_like(b))
    if kind == "batch":
        off, cols, vals, row_ptr, nrhs, _, _, _, b = _batch_inputs(case, seed)
        return dict(kind=kind, solver=b2s.BatchedCG(off, cols, vals, row_ptr, nrhs, tol=1e-8), b=b,
                    x=torch.zeros_like(b))
    (off, cols, vals, row), order, x = _assemble_inputs(case, seed)
    return dict(kind=kind, rows=off.numel() - 1, r=row[order].to(torch.int32), c=cols[order].contiguous(),
                v=vals[order].contiguous(), x=x, y=torch.zeros_like(x), segments=case["segments"], real=case["real"])


def run(s):
    kind = s["kind"]
    if kind == "spmv":
        s["A"].vectorProduct(s["x"], s["y"], s["alpha"], s["beta"])
        return s["y"]
    if kind in ("solve", "batch"):
        s["x"].zero_()  # the initial guess
        if not s["solver"].solve(s["b"], s["x"]):
            raise RuntimeError("the solve did not converge")
        return s["x"]
    A = b2s.SparseMatrix.from_coo(s["rows"], s["rows"], s["r"], s["c"], s["v"], segments=s["segments"],
                                  real=s["real"], duplicates="add")
    A.vectorProduct(s["x"], s["y"])
    return s["y"]


# ---------------------------------------------------------------------------
def _sizes(case):
    """Rows and stored elements of a case's matrix (irregular: their expected number)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    if case["matrix"] == "irregular":
        return n, int(n * 12.0 * math.exp(0.5))
    d = [nx, ny] + ([nz] if case["matrix"] != "poisson2d" else [])
    return n, n + sum(2 * (n - n // s) for s in d)


def work(case):
    """Bytes: every array once. A solve's operations: those of its iterations,
    whose number is a round estimate from the grid's side."""
    if case["kind"] == "batch":
        n = case["systems"] * ((case["lo"] + case["hi"]) / 2.0) ** 2
        its = 1.3 * (case["lo"] + case["hi"]) / 2.0
        return dict(bytes=n * (5 * 12 + 4 + 4.5 * 16), flops=n * 4.5 * 20 * its)
    n, nnz = _sizes(case)
    if case["kind"] == "assemble":
        sv = 8 if case["real"] == "double" else 4
        return dict(bytes=nnz * (8 + sv) + nnz * (4 + sv) + 4 * n + 2 * sv * n, flops=2 * nnz)
    if case["kind"] == "spmv":
        sv = 8 if case["real"] == "double" else 4
        idx = 0 if case["segments"] == "Multidiagonal" else 4
        y = 2 if case["keeper"] == "scaled" else 1
        return dict(bytes=nnz * (sv + idx) + (4 * n if idx else 0) + (1 + y) * sv * n, flops=2 * nnz)
    side = max(case["nx"], case["ny"], case["nz"])
    its = {"cg": (2.0 if case["matrix"] == "poisson2d" else 20.0) * side,
           "bicgstab": 1.5 * side * (0.3 if case["precond"] == "ilu0" else 1.0), "gmres": 3.5 * side}[case["solver"]]
    per = {"cg": 2 * nnz + 10 * n, "bicgstab": 4 * nnz + 20 * n, "gmres": 2 * nnz + 130 * n}[case["solver"]]
    return dict(bytes=12 * nnz + 4 * n + 16 * n, flops=its * per)


def tolerance(case):
    # products: up to 3e-16 and 1.1e-7 off exact() were measured, with long rows summed
    # in trees; another order of a 2048-element row's sum moves its last digits
    if case["kind"] in ("spmv", "assemble"):
        return {"rel": 1e-15} if case["real"] == "double" else {"rel": 5e-7}
    # solves stop at a residue of 1e-10 (1e-8 for the batch), an iteration more or less
    # apart: up to 1.4e-8 (CG), 1e-9 (the others) and 2e-8 (the batch) off exact()
    if case["kind"] == "batch":
        return {"rel": 1e-7}
    return {"rel": 5e-8} if case["solver"] == "cg" else {"rel": 5e-9}


def exact(case, seed):
    kind = case["kind"]
    if kind == "spmv":
        csr, x, y = _spmv_inputs(case, seed)
        off, cols, vals, row = csr
        vals = vals.to(x.dtype).double()
        alpha, beta = (float(torch.tensor(v, dtype=x.dtype)) for v in KEEPERS[case["keeper"]])
        return alpha * _times((off, cols, vals, row), x.double()) + beta * y.double()
    if kind == "solve":
        return _solve_inputs(case, seed)[1]
    if kind == "assemble":
        (off, cols, vals, row), _, x = _assemble_inputs(case, seed)
        return _times((off, cols, vals.double(), row), x.double())
    # the batch: each grid's Laplacian is diagonal in the sine basis
    _, _, _, row_ptr, nrhs, nx, ny, shift, b = _batch_inputs(case, seed)
    out, at = [], 0
    for s in range(case["systems"]):
        a, c, k = int(nx[s]), int(ny[s]), int(nrhs[s])
        rhs = b[at:at + a * c * k].reshape(c, a, k)
        at += a * c * k
        lam, S = [], []
        for m in (a, c):
            j = torch.arange(1, m + 1, device="cuda", dtype=torch.float64)
            S.append(math.sqrt(2.0 / (m + 1)) * torch.sin(math.pi / (m + 1) * j[:, None] * j[None, :]))
            lam.append(2.0 - 2.0 * torch.cos(math.pi * j / (m + 1)))
        h = torch.einsum("ij,pq,jqk->ipk", S[1], S[0], rhs)
        h = h / (lam[1][:, None] + lam[0][None, :] + float(shift[s]))[:, :, None]
        out.append(torch.einsum("ij,pq,jqk->ipk", S[1], S[0], h).reshape(-1))
    return torch.cat(out)
