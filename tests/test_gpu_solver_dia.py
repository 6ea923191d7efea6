"""Large engine systems in diagonal form (bs_spmv_dia) against the persistent
step, which multiplies from their CSR arrays with the same sums: the same bits
and iteration counts."""
import numpy as np
import pytest

from num_b200 import generators as gen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _off_diagonal(A):
    """A with one more symmetric pair, far from its diagonals, in rows that a
    look at a few rows does not meet: not in diagonal form."""
    S = A.to_scipy().tolil()
    S[1001, 90_002] = S[90_002, 1001] = -0.125
    S = S.tocsr()
    S.sort_indices()
    return gen.Csr(S.indptr.astype(np.int32), S.indices.astype(np.int32), S.data, A.nrows, A.ncols)


def _tridiag(n):
    i = np.arange(n, dtype=np.int64)
    cols = np.stack([i - 1, i, i + 1], 1)
    valid = (cols >= 0) & (cols < n)
    vals = np.stack([np.full(n, -1.0), 2.5 + 0.1 * np.sin(i), np.full(n, -1.0)], 1)
    rp = np.concatenate([[0], np.cumsum(valid.sum(1))]).astype(np.int32)
    return gen.Csr(rp, cols[valid].astype(np.int32), vals[valid].copy(), n, n)


def _solve(nmlib, systems, precision, persistent):
    from num_b200.solver import BatchSolver
    nmlib.nm_solver_set_persistent(persistent)
    try:
        S = BatchSolver(max_rows=sum(A.nrows + 8 for A in systems),
                        max_nnz=sum(A.nnz + 32 for A in systems), max_systems=len(systems),
                        precision=precision)
        rng = np.random.default_rng(9)
        out = S.solve([(A, rng.standard_normal(A.nrows)) for A in systems], tol=1e-8,
                      max_iter=150, chunk=32)
        return [(x, i["iters"], i["residual"]) for x, i in out]
    finally:
        nmlib.nm_solver_set_persistent(0)


# one row past the first size in diagonal form and one just below; 3, 5 and 7
# diagonals, constant and varying; ragged last tiles and blocks; alone, beside
# a system that is not in diagonal form, and beside small ones
@pytest.mark.parametrize("precision", ["fp32", "fp64", "bf16"])
@pytest.mark.parametrize("case", ["edge", "lap2d_363", "lap3d_52", "varcoef_52", "tridiag",
                                  "off_diagonal", "mixed"])
def test_diagonal_systems_equal_the_persistent_step(kspmv, nmlib, case, precision):
    systems = {"edge": lambda: [_tridiag(131_072), _tridiag(131_073)],
               "lap2d_363": lambda: [gen.laplacian_2d(363)],
               "lap3d_52": lambda: [gen.laplacian_3d(52)],
               "varcoef_52": lambda: [gen.varcoef_poisson_3d(52, seed=3)[0]],
               "tridiag": lambda: [_tridiag(200_003)],
               "off_diagonal": lambda: [_off_diagonal(gen.laplacian_2d(363))],
               "mixed": lambda: [gen.varcoef_poisson_3d(52, seed=3)[0], gen.laplacian_2d(40),
                                 _off_diagonal(gen.laplacian_2d(363)), gen.laplacian_2d(370)],
               }[case]()
    a, b = (_solve(nmlib, systems, precision, persistent) for persistent in (0, 1))
    for (x, it, res), (y, jt, sres) in zip(a, b):
        assert it == jt and res == sres and np.array_equal(x, y)


def test_diagonal_system_solved_again_in_its_slot(kspmv, nmlib):
    from num_b200.solver import BatchSolver
    A = gen.varcoef_poisson_3d(52, seed=3)[0]
    rng = np.random.default_rng(10)
    b1, b2 = rng.standard_normal(A.nrows), rng.standard_normal(A.nrows)

    def solve(S, slot):
        while slot in S.active:
            S.step(32)
        return S.solution(slot), S.status(slot)["iters"]

    S = BatchSolver(max_rows=2 * A.nrows + 16, max_nnz=2 * A.nnz + 64, max_systems=2)
    s = S.admit(A, b1, tol=1e-8)
    x1 = solve(S, s)
    S.resolve(s, b2)
    x2 = solve(S, s)
    S.take(s)
    s = S.admit(A, b1, tol=1e-8)  # the ranges it left
    again = solve(S, s)
    assert again[1] == x1[1] and np.array_equal(again[0], x1[0])
    T = BatchSolver(max_rows=A.nrows + 8, max_nnz=A.nnz + 32, max_systems=1)
    t = T.admit(A, b2, tol=1e-8)
    fresh = solve(T, t)
    assert fresh[1] == x2[1] and np.array_equal(fresh[0], x2[0])
