"""The CG solve on the diagonal form against the CUDA-graph path and the
oracle: the same bits up to 262,144 rows, where every path sums in one order;
above, the same iteration count (+-1) and solutions within 1e-9."""
import ctypes as C

import numpy as np
import pytest

from num_b200 import generators as gen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _tridiag(n):
    i = np.arange(n, dtype=np.int64)
    cols = np.stack([i - 1, i, i + 1], 1)
    valid = (cols >= 0) & (cols < n)
    vals = np.broadcast_to(np.array([-1.0, 2.001, -1.0]), (n, 3))
    rp = np.concatenate([[0], np.cumsum(valid.sum(1))]).astype(np.int32)
    return gen.Csr(rp, cols[valid].astype(np.int32), vals[valid].copy(), n, n)


def _eight(n, rng):
    """Symmetric, dominant, offsets 0, 3 and its mirror, ...: 7 diagonals, and
    an eighth that only the last rows have."""
    i = np.arange(n, dtype=np.int64)
    offs = [-700, -300, -3, 0, 3, 300, 700]
    cols = i[:, None] + np.array(offs)
    valid = (cols >= 0) & (cols < n)
    vals = np.where(np.array(offs) == 0, 7.5, -1.0) * np.ones((n, 1))
    rp = np.concatenate([[0], np.cumsum(valid.sum(1))]).astype(np.int64)
    ci, v = cols[valid], vals[valid].copy()
    # an entry of value 0 far left of the last row: the eighth diagonal
    ci = np.insert(ci, rp[n - 1], 5)
    v = np.insert(v, rp[n - 1], 0.0)
    rp[n] += 1
    return gen.Csr(rp.astype(np.int32), ci.astype(np.int32), v, n, n)


def _solve(kspmv, nmlib, M, b, mode, **kw):
    nmlib.nm_cg_set_persistent(mode)
    try:
        x = torch.zeros(b.shape[0], dtype=torch.float64, device="cuda")
        info = kspmv.cg_solve_local(M, b, x, **kw)
        path = C.c_int32(-1)
        nmlib.nm_cg_last_path(M._h, C.byref(path))
        return info, x.cpu().numpy(), path.value
    finally:
        nmlib.nm_cg_set_persistent(1)


# one and two tiles per CTA, a ragged last tile, 2 and 4 rows per thread, the
# last size with tile sums and the first without, 4, 8, 11 and 14 rows per
# thread; even and odd distances between a CTA's rows and those it reads
@pytest.mark.parametrize("case", ["lap2d_182", "lap2d_200", "lap2d_256", "lap2d_301",
                                  "lap2d_512", "lap2d_513", "lap3d_33", "lap3d_58", "lap3d_80",
                                  "lap2d_600", "lap2d_1029", "lap3d_65", "lap3d_89", "lap3d_90",
                                  "lap3d_101", "tridiag_40001", "tridiag_262145",
                                  "tridiag_400001", "eight_50001", "eight_300001",
                                  "varcoef_33", "varcoef_64"])
def test_diagonal_solve(kspmv, nmlib, case):
    name, size = case.split("_")
    rng = np.random.default_rng(11)
    A = {"lap2d": gen.laplacian_2d, "lap3d": gen.laplacian_3d, "tridiag": _tridiag,
         "eight": lambda n: _eight(n, rng),
         "varcoef": lambda L: gen.varcoef_poisson_3d(L, seed=3)[0]}[name](int(size))
    M = kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, A.nrows, A.ncols)
    b = torch.from_numpy(rng.standard_normal(A.nrows)).cuda()
    kw = {"tol": 1e-8, "max_iter": 400 if A.nrows > 262144 else 3000}
    info, x, path = _solve(kspmv, nmlib, M, b, 1, **kw)
    assert path == 5
    ginfo, gx, gpath = _solve(kspmv, nmlib, M, b, 0, **kw)
    assert gpath == 0
    if A.nrows <= 262144:
        assert info == ginfo and np.array_equal(x, gx)
    else:
        assert abs(info["iters"] - ginfo["iters"]) <= 1
        assert info["converged"] == ginfo["converged"]
        assert np.linalg.norm(x - gx) <= 1e-9 * np.linalg.norm(gx)
    again = _solve(kspmv, nmlib, M, b, 1, **kw)
    assert again[0] == info and np.array_equal(again[1], x)


@pytest.mark.parametrize("max_iter", [1, 2, 3])
def test_diagonal_solve_stops_where_the_graph_path_does(kspmv, nmlib, max_iter):
    A = gen.laplacian_2d(190)
    M = kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, A.nrows, A.ncols)
    rng = np.random.default_rng(12)
    b = torch.from_numpy(rng.standard_normal(A.nrows)).cuda()
    for tol in (1e-30, 0.9, 0.3):
        one = _solve(kspmv, nmlib, M, b, 1, tol=tol, max_iter=max_iter)
        two = _solve(kspmv, nmlib, M, b, 0, tol=tol, max_iter=max_iter)
        assert one[0] == two[0] and np.array_equal(one[1], two[1])


def test_diagonal_solve_of_a_singular_matrix(kspmv, nmlib):
    # p.Ap = 0: NaN to max_iter without the guard, an error with it
    n = 40_000
    A = gen.diagonal(np.zeros(n))
    M = kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, n, n)
    info, x, path = _solve(kspmv, nmlib, M, torch.ones(n, dtype=torch.float64, device="cuda"), 1,
                           max_iter=7)
    assert path == 5 and info["iters"] == 7 and not info["converged"]
    assert np.isnan(info["residual"]) and not np.isfinite(x).any()
    D = kspmv.distribute_csr(A.row_ptr, A.col_idx, A.values, n, n)
    with pytest.raises(RuntimeError, match="near zero"):
        kspmv.cg_solve(D, torch.ones(n, dtype=torch.float64, device="cuda"),
                       torch.zeros(n, dtype=torch.float64, device="cuda"))
