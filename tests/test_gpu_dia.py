"""Matrices whose nonzeros lie on few diagonals: the SpMV on their diagonal
form against the oracle's serial row loop and the row-block kernel, bit for
bit (every row is summed by one thread in CSR order on both)."""
import numpy as np
import pytest

from num_b200 import generators as gen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _diagonals(nrows, ncols, offs, rng, keep=1.0, constant=False):
    """Entries on the diagonals col - row in `offs`, each kept with
    probability `keep` per run of 64 rows."""
    r = np.arange(nrows, dtype=np.int64)
    cols = r[:, None] + np.asarray(sorted(offs), np.int64)[None, :]
    valid = (cols >= 0) & (cols < ncols)
    runs = rng.random((nrows // 64 + 1, len(offs))) < keep
    valid &= runs[r // 64]
    rp = np.concatenate([[0], np.cumsum(valid.sum(1))]).astype(np.int32)
    vals = np.broadcast_to(rng.standard_normal(len(offs)), cols.shape) if constant \
        else rng.standard_normal(cols.shape)
    return gen.Csr(rp, cols[valid].astype(np.int32), vals[valid].copy(), nrows, ncols)


def _case(name):
    rng = np.random.default_rng(77)
    if name.startswith("lap2d"):
        return gen.laplacian_2d(int(name[6:]))
    if name.startswith("lap3d"):
        return gen.laplacian_3d(int(name[6:]))
    if name == "varcoef_19":
        return gen.varcoef_poisson_3d(19, seed=3)[0]
    if name == "gauge_40":
        return gen.lattice_gauge(40)
    if name == "wide":  # rectangular, 16 diagonals, some absent in runs of rows
        return _diagonals(3001, 4100, [-900, -64, -33, -2, -1, 0, 1, 2, 3, 31, 64, 65, 500, 999,
                                       1000, 1099], rng, keep=0.95)
    if name == "tall":  # rows past the last column are empty
        return _diagonals(1000, 700, [-3, 0, 5], rng)
    if name == "eight":  # the most an 8-bit mask holds
        return _diagonals(1500, 1500, [-40, -7, -1, 0, 1, 2, 7, 40], rng)
    if name == "const_9":
        return _diagonals(2500, 2500, [-50, -49, -1, 0, 1, 49, 50, 51, 400], rng, constant=True)
    if name == "many":  # 17 diagonals: one more than the form holds
        return _diagonals(2000, 2000, list(range(-8, 9)), rng)
    if name == "unsorted":  # columns descend within a row
        A = gen.laplacian_2d(20)
        order = np.concatenate([np.arange(A.row_ptr[i], A.row_ptr[i + 1])[::-1]
                                for i in range(A.nrows)])
        return gen.Csr(A.row_ptr, A.col_idx[order], A.values[order], A.nrows, A.ncols)
    n = int(name[5:])  # "diag_<n>"
    return gen.diagonal(rng.standard_normal(n))


CASES = ["lap2d_1", "lap2d_32", "lap2d_33", "lap2d_400", "lap3d_17", "lap3d_54", "varcoef_19",
         "gauge_40", "wide", "tall", "eight", "const_9", "many", "unsorted", "diag_1", "diag_31",
         "diag_129", "diag_256", "diag_151553"]


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("name", CASES)
def test_diagonal_form_bit_exact(kspmv, oracle, name, offset):
    A = _case(name)
    rng = np.random.default_rng(5)
    x = rng.uniform(-1, 1, A.ncols)
    for precision, xt in (("fp64", x), ("fp32", x.astype(np.float32)),
                          ("bf16", x.astype(np.float32))):
        if precision == "bf16":
            from num_b200.kokkos_spmv import _values_for
            v = (_values_for(A.values, "bf16")[0].astype(np.uint32) << 16).view(np.float32)
        else:
            v = A.values.astype(xt.dtype)
        ref = oracle.spmv(A.row_ptr, A.col_idx, v, xt)
        M = kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, A.nrows, A.ncols,
                             precision=precision)
        buf = torch.full((A.ncols + 1,), float("nan"), device="cuda",
                         dtype=torch.from_numpy(xt).dtype)
        buf[offset:offset + A.ncols] = torch.from_numpy(xt)
        for kernel in ("auto", "blocks"):
            kspmv.tune(M, kernel=kernel)
            y = torch.full((A.nrows,), float("nan"), device="cuda", dtype=buf.dtype)
            kspmv.spmv(M, buf[offset:offset + A.ncols], y)
            assert np.array_equal(y.cpu().numpy(), ref), (precision, kernel)


def test_diagonal_form_keeps_absent_entries_out(kspmv, oracle):
    # infinities and NaN of x reach only the rows that have an entry there,
    # and a diagonal of zeros still multiplies (0 * inf = NaN)
    A = gen.laplacian_2d(40)
    x = np.random.default_rng(6).standard_normal(A.ncols)
    x[[0, 39, 700, 1599]] = [np.inf, np.nan, -np.inf, np.nan]
    for v in (A.values, np.where(A.values == 4.0, 4.0, 0.0)):
        M = kspmv.upload_csr(A.row_ptr, A.col_idx, v, A.nrows, A.ncols)
        y = torch.empty(A.nrows, dtype=torch.float64, device="cuda")
        kspmv.spmv(M, torch.from_numpy(x).cuda(), y)
        ref = oracle.spmv(A.row_ptr, A.col_idx, v, x)
        assert np.array_equal(y.cpu().numpy(), ref, equal_nan=True)


def test_diagonal_form_of_an_assembled_laplacian(kspmv, oracle):
    A = gen.laplacian_3d(33)
    x = np.random.default_rng(7).standard_normal(A.ncols)
    M = kspmv.laplacian(3, 33)
    y = torch.empty(A.nrows, dtype=torch.float64, device="cuda")
    kspmv.spmv(M, torch.from_numpy(x).cuda(), y)
    assert np.array_equal(y.cpu().numpy(), oracle.spmv(A.row_ptr, A.col_idx, A.values, x))


# chunks of one and several lanes, ragged last chunks, 16-byte loads or not,
# the widest masks, one run and many
@pytest.mark.parametrize("k", [1, 2, 3, 7, 16, 17, 33, 34, 130])
@pytest.mark.parametrize("name", ["lap2d_1", "lap2d_33", "lap3d_17", "varcoef_19", "gauge_40",
                                  "wide", "tall", "eight", "const_9", "diag_129"])
def test_diagonal_form_multi_rhs_bit_exact(kspmv, oracle, name, k):
    A = _case(name)
    X = np.random.default_rng(k).standard_normal((A.ncols, k))
    M = kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, A.nrows, A.ncols)
    ref = oracle.batch_spmv(A.row_ptr, A.col_idx, A.values, X)
    for offset in (0, 1):  # X on a 16-byte boundary, and 8 bytes off it
        buf = torch.full((A.ncols * k + 1,), float("nan"), dtype=torch.float64, device="cuda")
        Xd = buf[offset:offset + A.ncols * k].view(A.ncols, k)
        Xd.copy_(torch.from_numpy(X))
        Y = torch.full((A.nrows, k), float("nan"), dtype=torch.float64, device="cuda")
        kspmv.batch_spmv(M, Xd, Y)
        assert np.array_equal(Y.cpu().numpy(), ref), offset
