"""A step's graphs against the persistent step, which has none: large systems
admitted while others iterate, so that the lists change under kept graphs, and
solvers made for one system, whose lists hold little more than its tiles.  The
same bits and iteration counts."""
import numpy as np
import pytest

from num_b200 import generators as gen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _off_diagonal(A):
    """A with one more symmetric pair, far from its diagonals: not in diagonal
    form."""
    S = A.to_scipy().tolil()
    S[1001, 90_002] = S[90_002, 1001] = -0.125
    S = S.tocsr()
    S.sort_indices()
    return gen.Csr(S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data, A.nrows, A.ncols)


def _run(nmlib, first, later, persistent):
    """Two steps of `first`, then one more system of `later` after each further
    step; everything solved to the end."""
    from num_b200.solver import BatchSolver
    rng = np.random.default_rng(11)
    first = [(A, rng.standard_normal(A.nrows)) for A in first]
    later = [(A, rng.standard_normal(A.nrows)) for A in later]
    nmlib.nm_solver_set_persistent(persistent)
    try:
        S = BatchSolver(max_rows=sum(A.nrows + 8 for A, _ in first + later),
                        max_nnz=sum(A.nnz + 32 for A, _ in first + later), max_systems=64)
        slots = S.admit_many(first, max_iter=150)
        S.step(8)
        S.step(8)
        for A, b in later:
            slots.append(S.admit(A, b, max_iter=150))
            S.step(8)
        while S.active:
            S.step(32)
        return [(x, i["iters"], i["residual"]) for x, i in S.take_many(slots)]
    finally:
        nmlib.nm_solver_set_persistent(0)


# Tiles of 4,096 rows.  Beside 33 tiles of a system that is not in diagonal
# form, the tiles in diagonal form grow past a power of two while those of all
# systems stay under one: 35 -> 69 of 128, and 103 -> 137 of 256; then further.
@pytest.mark.parametrize("before", [1, 3])
def test_diagonal_systems_admitted_between_steps(kspmv, nmlib, before):
    varcoef = gen.varcoef_poisson_3d(52, seed=3)[0]
    lap = gen.laplacian_2d(370)
    first = [_off_diagonal(gen.laplacian_2d(363)), varcoef] + [lap] * (before - 1)
    a, b = (_run(nmlib, first, [lap, varcoef, lap], persistent) for persistent in (0, 1))
    for (x, it, res), (y, jt, sres) in zip(a, b):
        assert it == jt and res == sres and np.array_equal(x, y)


def _tridiag(n):
    i = np.arange(n, dtype=np.int64)
    cols = np.stack([i - 1, i, i + 1], 1)
    valid = (cols >= 0) & (cols < n)
    vals = np.stack([np.full(n, -1.0), 2.5 + 0.1 * np.sin(i), np.full(n, -1.0)], 1)
    rp = np.concatenate([[0], np.cumsum(valid.sum(1))]).astype(np.int32)
    return gen.Csr(rp, cols[valid].astype(np.int32), vals[valid].copy(), n, n)


# 33, 65 and 74 tiles (8 and 4 CTAs to a tile) and 257 and 270 (2 CTAs of 8 row
# blocks each): the first past a power of two, and one further on
@pytest.mark.parametrize("n", [131_073, 262_145, 300_008, 1_048_577, 1_104_000])
def test_solver_made_for_one_system(kspmv, nmlib, n):
    from num_b200.solver import BatchSolver
    A = _tridiag(n)
    b = np.random.default_rng(n).standard_normal(n)
    out = []
    for persistent in (0, 1):
        nmlib.nm_solver_set_persistent(persistent)
        try:
            S = BatchSolver(max_rows=n + 8, max_nnz=A.nnz + 32, max_systems=1)
            s = S.admit(A, b, max_iter=200)
            while s in S.active:
                S.step(32)
            out.append(S.take(s))
        finally:
            nmlib.nm_solver_set_persistent(0)
    (x, i), (y, j) = out
    assert i["iters"] == j["iters"] and i["residual"] == j["residual"] and np.array_equal(x, y)
