"""Workloads of this library, each one pass through its public entry points.

`listed()` are the named ones, `draw(rng)` gives another of the same ranges.
`prepare(case, seed)` makes what a program has in hand before the call (the
uploaded matrix or the engine with its systems, and the vectors), `run(state)`
makes one pass, `work(case)` counts the bytes and operations a pass cannot do
without, and `exact(case, seed)` is the pass's result in 64 bits from plain
torch.

kinds:
  spmv    y = A x, device vectors, synchronous (kokkos_spmv.spmv)
  batch   Y = A X with k right-hand sides (kokkos_spmv.batch_spmv)
  cg      one plain FP64 conjugate-gradient solve (kokkos_spmv.cg_solve_local)
  engine  one mixed-precision Jacobi-PCG solve of a system the engine keeps,
          with a new right-hand side (BatchSolver.resolve / step / solution)
  serve   a batch of uneven systems admitted, solved and taken out
          (BatchSolver.solve)

matrices:
  lap2d, lap3d  5- / 7-point Laplacians, L^2 / L^3 rows (assembled on the device)
  varcoef       7-point variable-coefficient Poisson, exp(N(0,1)) on the faces
  gauge         the 5-point periodic lattice-gauge operator, L^2 rows
  banded        `count` banded SPD systems of 32..4096 rows in one handle, two
                random entries per row outside the band
  powerlaw      n rows of lognormal length (mean 16), columns uniform
"""
import math

import numpy as np
import torch

from num_b200 import generators as gen
from num_b200 import kokkos_spmv as kspmv
from num_b200.solver import BatchSolver

_VEC = {"fp64": torch.float64, "fp32": torch.float32, "bf16": torch.float32}


def listed():
    return [
        # A call inside a small time step or a test: latency and launches count.
        {"name": "spmv_lap2d_64", "kind": "spmv", "matrix": "lap2d", "L": 64, "precision": "fp64"},
        # The headline product: 7-point stencil on 160^3.
        {"name": "spmv_lap3d_160", "kind": "spmv", "matrix": "lap3d", "L": 160,
         "precision": "fp64"},
        # General coefficients, an odd grid, FP32 values and vectors.
        {"name": "spmv_varcoef_127_fp32", "kind": "spmv", "matrix": "varcoef", "L": 127,
         "precision": "fp32"},
        # Thousands of small uneven matrices multiplied in one launch.
        {"name": "spmv_banded_4096", "kind": "spmv", "matrix": "banded", "count": 4096,
         "precision": "fp64"},
        # Scattered columns and uneven rows: a graph or a network.
        {"name": "spmv_powerlaw_1m", "kind": "spmv", "matrix": "powerlaw", "n": 1_000_000,
         "precision": "fp64"},
        # Many right-hand sides at once, wide (a block method) ...
        {"name": "batch_lap3d_100_k128", "kind": "batch", "matrix": "lap3d", "L": 100, "k": 128},
        # ... and narrow (a few sources on a lattice).
        {"name": "batch_gauge_500_k8", "kind": "batch", "matrix": "gauge", "L": 500, "k": 8},
        # Plain CG solves to 1e-8: small, medium, and a 3-D grid of a million rows.
        {"name": "cg_lap2d_256", "kind": "cg", "matrix": "lap2d", "L": 256},
        {"name": "cg_lap2d_500", "kind": "cg", "matrix": "lap2d", "L": 500},
        {"name": "cg_lap3d_100", "kind": "cg", "matrix": "lap3d", "L": 100},
        # Mixed precision with FP64 refinement on one large system, solved
        # again for each new right-hand side (a time stepper).
        {"name": "engine_varcoef_128_fp32", "kind": "engine", "matrix": "varcoef", "L": 128,
         "precision": "fp32"},
        # A batch of uneven requests through the engine.
        {"name": "serve_48_fp32", "kind": "serve", "count": 48, "side": 512, "rows": 65536,
         "precision": "fp32"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmv", "spmv", "spmv", "batch", "cg", "cg", "engine", "serve"])
    if kind == "spmv":
        c = {"kind": kind, "matrix": rng.choice(["lap2d", "lap3d", "varcoef", "gauge", "banded",
                                                 "powerlaw"]),
             "precision": rng.choice(["fp64", "fp32", "bf16"])}
        size = {"lap2d": ("L", 32, 2000), "lap3d": ("L", 10, 160), "varcoef": ("L", 10, 128),
                "gauge": ("L", 32, 700), "banded": ("count", 64, 4096),
                "powerlaw": ("n", 10_000, 1_000_000)}[c["matrix"]]
        c[size[0]] = _log(rng, size[1], size[2])
        return c
    if kind == "batch":
        c = {"kind": kind, "matrix": rng.choice(["lap2d", "lap3d", "gauge", "varcoef"]),
             "k": _log(rng, 2, 128)}
        c["L"] = _log(rng, 32, 500) if c["matrix"] in ("lap2d", "gauge") else _log(rng, 10, 100)
        return c
    if kind == "cg":
        c = {"kind": kind, "matrix": rng.choice(["lap2d", "lap3d", "varcoef"])}
        c["L"] = _log(rng, 32, 500) if c["matrix"] == "lap2d" else _log(rng, 10, 100)
        return c
    if kind == "engine":
        return {"kind": kind, "matrix": "varcoef", "L": _log(rng, 16, 128),
                "precision": rng.choice(["fp64", "fp32"])}
    return {"kind": kind, "count": rng.randint(8, 48), "side": _log(rng, 64, 512),
            "rows": _log(rng, 1024, 65536), "precision": rng.choice(["fp64", "fp32"])}


# ---- matrices ------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _csr(rows, cols, vals, n):
    """CSR of sorted (row, column) triplets on the GPU."""
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(rows, minlength=n), 0, out=rp[1:])
    return rp.to(torch.int32), cols.to(torch.int32), vals


def _stencil(L, dim, vals, valid):
    """Rows given as candidates in ascending column order."""
    n = L ** dim
    i = torch.arange(n, device="cuda")
    off = [-(L ** 2), -L, -1, 0, 1, L, L ** 2] if dim == 3 else [-L, -1, 0, 1, L]
    cols = torch.stack([i + o for o in off], 1)
    rows = i[:, None].expand_as(cols)
    return _csr(rows[valid], cols[valid], vals[valid], n)


def _laplacian(L, dim):
    i = torch.arange(L ** dim, device="cuda")
    c = [(i // L ** d) % L for d in range(dim)]
    on = torch.ones_like(i, dtype=torch.bool)
    valid = torch.stack([c[d] > 0 for d in reversed(range(dim))] + [on]
                        + [c[d] < L - 1 for d in range(dim)], 1)
    v = torch.full(valid.shape, -1.0, dtype=torch.float64, device="cuda")
    v[:, dim] = 2.0 * dim
    return _stencil(L, dim, v, valid)


def _varcoef(L, g):
    def face(*shape):
        return torch.exp(torch.randn(*shape, dtype=torch.float64, device="cuda", generator=g))

    cx, cy, cz = face(L, L, L + 1), face(L, L + 1, L), face(L + 1, L, L)  # [z, y, x]
    xm, xp = cx[:, :, :-1].reshape(-1), cx[:, :, 1:].reshape(-1)
    ym, yp = cy[:, :-1, :].reshape(-1), cy[:, 1:, :].reshape(-1)
    zm, zp = cz[:-1].reshape(-1), cz[1:].reshape(-1)
    v = torch.stack([-zm, -ym, -xm, xm + xp + ym + yp + zm + zp, -xp, -yp, -zp], 1)
    i = torch.arange(L ** 3, device="cuda")
    x, y, z = i % L, (i // L) % L, i // (L * L)
    valid = torch.stack([z > 0, y > 0, x > 0, x >= 0, x < L - 1, y < L - 1, z < L - 1], 1)
    return _stencil(L, 3, v, valid)


def _powerlaw(n, g, mean=16.0, sigma=1.2, most=2048):
    mu = math.log(mean) - sigma * sigma / 2
    z = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    lens = torch.clamp(torch.round(torch.exp(mu + sigma * z)), 1, most).long()
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    cols = torch.randint(0, n, rows.shape, device="cuda", generator=g)
    key = torch.unique(rows * n + cols)
    v = torch.randn(key.shape, dtype=torch.float64, device="cuda", generator=g)
    return _csr(key // n, key % n, v, n)


def _banded(sizes, hbs, g):
    """Banded SPD systems (half-bandwidth hbs[m], two random mirrored entries
    per row, off-diagonals U[-1, 0], strictly dominant diagonal) as one
    block-diagonal CSR."""
    n = torch.as_tensor(sizes, device="cuda")
    hb = torch.as_tensor(hbs, device="cuda")
    N = int(sum(sizes))
    start = torch.cumsum(n, 0) - n
    owner = torch.repeat_interleave(torch.arange(len(sizes), device="cuda"), n)
    i = torch.arange(N, device="cuda")
    local, size, half = i - start[owner], n[owner], hb[owner]
    keys = []
    for d in range(1, int(max(hbs)) + 1):
        ok = (d <= half) & (local + d < size)
        keys.append(i[ok] * N + i[ok] + d)
    for _ in range(2):
        u = torch.rand(N, dtype=torch.float64, device="cuda", generator=g)
        j = (u * size).long().clamp_(max=N) + start[owner]
        ok = (j - i).abs() > half
        keys.append(torch.minimum(i, j)[ok] * N + torch.maximum(i, j)[ok])
    key = torch.unique(torch.cat(keys))
    a, b = key // N, key % N
    v = -torch.rand(key.shape, dtype=torch.float64, device="cuda", generator=g)
    rows, cols, vals = torch.cat([a, b]), torch.cat([b, a]), torch.cat([v, v])
    order = torch.argsort(rows * N + cols)
    rows, cols, vals = rows[order], cols[order], vals[order]
    lens = torch.bincount(rows, minlength=N)
    diag = 1.05 * torch.segment_reduce(vals.abs(), "sum", lengths=lens) + 1e-3
    rows, cols = torch.cat([rows, i]), torch.cat([cols, i])
    vals = torch.cat([vals, diag])
    order = torch.argsort(rows * N + cols)
    return _csr(rows[order], cols[order], vals[order], N)


def _split(csr, sizes):
    """The systems of a block-diagonal CSR as host (row_ptr, col_idx, values, n)."""
    rp, ci, v = (t.cpu().numpy() for t in csr)
    out, r0 = [], 0
    for n in sizes:
        z0, z1 = int(rp[r0]), int(rp[r0 + n])
        out.append((rp[r0:r0 + n + 1] - rp[r0], ci[z0:z1] - np.int32(r0), v[z0:z1], int(n)))
        r0 += n
    return out


def _sizes(case):
    """Rows and half-bandwidths of a `banded` case's systems (the case's own;
    the seed draws their entries)."""
    rng = np.random.default_rng(case["count"])
    n = np.rint(np.exp(rng.uniform(math.log(32), math.log(4096), case["count"]))).astype(np.int64)
    return n.tolist(), rng.integers(1, 9, case["count"]).tolist()


def _matrix(case, seed):
    """The case's matrix as (row_ptr, col_idx, values FP64) on the GPU."""
    m = case["matrix"]
    if m == "lap2d":
        return _laplacian(case["L"], 2)
    if m == "lap3d":
        return _laplacian(case["L"], 3)
    if m == "varcoef":
        return _varcoef(case["L"], _gen(seed))
    if m == "gauge":
        A = gen.lattice_gauge(case["L"], rng=np.random.default_rng(int(seed)))
        return tuple(torch.from_numpy(a).cuda() for a in (A.row_ptr, A.col_idx, A.values))
    if m == "banded":
        return _banded(*_sizes(case), _gen(seed))
    return _powerlaw(case["n"], _gen(seed))


def _upload(case, seed):
    m, prec = case["matrix"], case.get("precision", "fp64")
    if m in ("lap2d", "lap3d"):
        return kspmv.laplacian(2 if m == "lap2d" else 3, case["L"], precision=prec)
    csr = _matrix(case, seed)
    if m == "banded":
        sizes = _sizes(case)[0]
        return kspmv.upload_csr_batched([(rp, ci, v, n, n) for rp, ci, v, n in _split(csr, sizes)],
                                        precision=prec)
    rp, ci, v = (t.cpu().numpy() for t in csr)
    n = rp.shape[0] - 1
    return kspmv.upload_csr(rp, ci, v, n, n, precision=prec)


def _requests(case, seed):
    """A served batch: half 5-point Laplacians with sides log-uniform in
    [32, side], half banded systems with rows log-uniform in [256, rows] (the
    sizes are the case's own; the seed draws entries and right-hand sides)."""
    rng = np.random.default_rng([case["count"], case["side"], case["rows"]])
    count, systems = case["count"], []
    lap = [int(round(math.exp(rng.uniform(math.log(32), math.log(case["side"])))))
           for _ in range(count // 2)]
    band = [int(round(math.exp(rng.uniform(math.log(256), math.log(case["rows"])))))
            for _ in range(count - count // 2)]
    hbs = rng.integers(1, 9, len(band)).tolist()
    band = _split(_banded(band, hbs, _gen(seed)), band)
    for k in range(count):
        if k % 2 and k // 2 < len(lap):
            L = lap[k // 2]
            rp, ci, v = (t.cpu().numpy() for t in _laplacian(L, 2))
            systems.append((rp, ci, v, L * L))
        else:
            systems.append(band.pop())
    rng = np.random.default_rng(int(seed))
    return [(A, rng.standard_normal(A[3])) for A in systems]


# ---- one pass ------------------------------------------------------------------------

def prepare(case, seed):
    kspmv.init(0)
    kind, g = case["kind"], _gen(seed + 7919)
    if kind == "serve":
        systems = _requests(case, seed)
        rows = sum(A[3] + 8 for A, _ in systems)
        nnz = sum(A[1].shape[0] + 32 for A, _ in systems)
        S = BatchSolver(max_rows=rows, max_nnz=nnz, max_systems=len(systems),
                        precision=case["precision"])
        return {"kind": kind, "S": S, "systems": systems}
    if kind == "engine":
        rp, ci, v = (t.cpu().numpy() for t in _matrix(case, seed))
        n = rp.shape[0] - 1
        b = np.random.default_rng(int(seed)).standard_normal(n)
        S = BatchSolver(max_rows=n + 8, max_nnz=ci.shape[0] + 32, max_systems=1,
                        precision=case["precision"])
        slot = S.admit((rp, ci, v, n), b, tol=1e-10, max_iter=20000)
        return {"kind": kind, "S": S, "slot": slot, "b": b}
    M = _upload(case, seed)
    if kind == "cg":
        b = torch.randn(M.nrows, dtype=torch.float64, device="cuda", generator=g)
        return {"kind": kind, "M": M, "b": b}
    if kind == "batch":
        X = torch.rand(M.ncols, case["k"], dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        return {"kind": kind, "M": M, "X": X, "Y": torch.empty_like(X)}
    dt = _VEC[case["precision"]]
    x = torch.rand(M.ncols, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    return {"kind": kind, "M": M, "x": x.to(dt), "y": torch.empty(M.nrows, dtype=dt, device="cuda")}


def run(s):
    kind = s["kind"]
    if kind == "spmv":
        kspmv.spmv(s["M"], s["x"], s["y"])
        return s["y"]
    if kind == "batch":
        kspmv.batch_spmv(s["M"], s["X"], s["Y"])
        return s["Y"]
    if kind == "cg":
        x = torch.zeros_like(s["b"])
        info = kspmv.cg_solve_local(s["M"], s["b"], x, tol=1e-8, max_iter=20000)
        return {"x": x, **info}
    if kind == "engine":
        S, slot = s["S"], s["slot"]
        S.resolve(slot, s["b"])
        while slot in S.active:
            S.step(64)
        info = S.status(slot)
        return {"x": S.solution(slot), "iters": info["iters"], "converged": info["converged"]}
    got = s["S"].solve(s["systems"], tol=1e-8, max_iter=20000, chunk=64)
    return {"x": [x for x, _ in got], "iters": np.array([i["iters"] for _, i in got]),
            "converged": np.array([i["converged"] for _, i in got])}


# ---- what a pass cannot do without ---------------------------------------------------

def _shape(case):
    """(rows, nonzeros) of the case, expected where they are random."""
    m = case["matrix"]
    if m == "powerlaw":
        return case["n"], 16.0 * case["n"]
    if m == "banded":
        mean = (4096 - 32) / math.log(4096 / 32)
        return case["count"] * mean, case["count"] * mean * (1 + 2 * 4.5 + 4)
    L = case["L"]
    if m == "gauge":
        return L * L, 5.0 * L * L
    return (L * L, 5.0 * L * L - 4 * L) if m == "lap2d" else (L ** 3, 7.0 * L ** 3 - 6 * L * L)


def _iterations(case):
    """About how many CG iterations the case's solve takes."""
    L = case["L"]
    return {"lap2d": 2.9 * L, "lap3d": 2.8 * L, "varcoef": 5.4 * L}[case["matrix"]]


def work(case):
    """Inputs read once and results written once: the matrix (values, 32-bit
    columns and row offsets), the vectors; for the solvers the operations of
    every iteration, whose data can stay on chip or in cache."""
    kind = case["kind"]
    if kind == "serve":
        ml = math.log
        n2 = case["side"] ** 2
        lap = (n2 - 32 ** 2) / (2 * ml(case["side"] / 32)) if case["side"] > 32 else n2
        band = (case["rows"] - 256) / ml(case["rows"] / 256) if case["rows"] > 256 else 256
        half = case["count"] / 2
        return {"bytes": half * lap * (12 * 5 + 20) + half * band * (12 * 14 + 20),
                "flops": half * lap * 22 * 2 * math.sqrt(lap) + half * band * 40 * 30}
    n, nnz = _shape(case)
    v = {"fp64": 8, "fp32": 4, "bf16": 2}[case.get("precision", "fp64")]
    if kind == "spmv":
        return {"bytes": (v + 4) * nnz + 4 * (n + 1) + 2 * n * (8 if v == 8 else 4),
                "flops": 2 * nnz}
    if kind == "batch":
        k = case["k"]
        return {"bytes": 12 * nnz + 4 * (n + 1) + 16 * n * k, "flops": 2 * nnz * k}
    return {"bytes": 12 * nnz + 4 * (n + 1) + 16 * n,
            "flops": _iterations(case) * (2 * nnz + 12 * n)}


# ---- the same in 64 bits, from plain torch -------------------------------------------

def _sparse(csr):
    rp, ci, v = csr
    n = rp.shape[0] - 1
    return torch.sparse_csr_tensor(rp.long(), ci.long(), v, size=(n, n), dtype=torch.float64)


def _pcg(csr, b, tol=1e-13, most=20000):
    """Jacobi PCG in 64 bits, to a residual where only rounding is left."""
    rp, ci, v = csr
    n = rp.shape[0] - 1
    A = _sparse(csr)
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), (rp[1:] - rp[:-1]).long())
    on = ci.long() == rows
    dinv = torch.ones(n, dtype=torch.float64, device="cuda")
    dinv[rows[on]] = 1.0 / v[on]
    x = torch.zeros_like(b)
    r, z = b.clone(), dinv * b
    p, rz, stop = z.clone(), torch.dot(b, z), tol * torch.linalg.norm(b)
    for k in range(most):
        Ap = A @ p
        alpha = rz / torch.dot(p, Ap)
        x += alpha * p
        r -= alpha * Ap
        if k % 16 == 15 and bool(torch.linalg.norm(r) < stop):
            break
        z = dinv * r
        rz_new = torch.dot(r, z)
        p = z + (rz_new / rz) * p
        rz = rz_new
    return x


def _poisson(L, dim, b):
    """The solution of the constant-coefficient Laplacian by sine transforms."""
    k = torch.arange(1, L + 1, dtype=torch.float64, device="cuda")
    S = torch.sin(math.pi * k[:, None] * k[None, :] / (L + 1)) * math.sqrt(2.0 / (L + 1))
    lam = 2.0 - 2.0 * torch.cos(math.pi * k / (L + 1))
    x = b.reshape([L] * dim)

    def each(x):
        for d in range(dim):
            x = torch.movedim(torch.tensordot(S, x, dims=([1], [d])), 0, d)
        return x

    den = sum(lam.reshape([L if e == d else 1 for e in range(dim)]) for d in range(dim))
    return each(each(x) / den).reshape(-1)


def exact(case, seed):
    kind, g = case["kind"], _gen(seed + 7919)
    if kind == "serve":
        systems = _requests(case, seed)
        rp, ci, v, b, r0, z0 = [torch.zeros(1, dtype=torch.int64)], [], [], [], 0, 0
        for (p, c, w, n), rhs in systems:
            rp.append(torch.from_numpy(p[1:].astype(np.int64)) + z0)
            ci.append(torch.from_numpy(c.astype(np.int64)) + r0)
            v.append(torch.from_numpy(np.ascontiguousarray(w)))
            b.append(torch.from_numpy(rhs))
            r0, z0 = r0 + n, z0 + int(p[n])
        whole = tuple(torch.cat(t).cuda() for t in (rp, ci, v))
        x = _pcg(whole, torch.cat(b).cuda())
        return {"x": list(torch.split(x, [A[3] for A, _ in systems])), "iters": None,
                "converged": None}
    csr = _matrix(case, seed)
    n = csr[0].shape[0] - 1
    if kind == "engine":
        b = torch.from_numpy(np.random.default_rng(int(seed)).standard_normal(n)).cuda()
        return {"x": _pcg(csr, b), "iters": None, "converged": None}
    if kind == "cg":
        b = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
        x = (_pcg(csr, b) if case["matrix"] == "varcoef" else
             _poisson(case["L"], 2 if case["matrix"] == "lap2d" else 3, b))
        return {"x": x, "iters": None, "residual": None, "converged": None}
    if kind == "batch":
        X = torch.rand(n, case["k"], dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        return _sparse(csr) @ X
    # values and x as the matrix and the call hold them
    store = {"fp64": torch.float64, "fp32": torch.float32, "bf16": torch.bfloat16}[case["precision"]]
    v = csr[2] if store == torch.float64 else csr[2].float().to(store)
    x = torch.rand(n, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
    return _sparse((csr[0], csr[1], v.double())) @ x.to(_VEC[case["precision"]]).double()
