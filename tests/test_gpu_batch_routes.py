"""Multi-RHS products on both sides of the lines between the kernels of the
diagonal form and the CSR kernels, and between the instances for 9, 12 and 16
diagonals and the one that walks the masks: the oracle's bits."""
import numpy as np
import pytest

from num_b200 import generators as gen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

OFFS = [-900, -500, -64, -33, -2, -1, 0, 1, 2, 31, 64, 65, 500, 999, 1000, 1100]


def _diagonals(n, count, keep, constant):
    rng = np.random.default_rng(count)
    lo = (16 - count) // 2
    i = np.arange(n, dtype=np.int64)
    cols = i[:, None] + np.array(OFFS[lo:lo + count])
    valid = (cols >= 0) & (cols < n) & (rng.random((n // 32 + 1, count)) < keep)[i // 32]
    rp = np.concatenate([[0], np.cumsum(valid.sum(1))]).astype(np.int32)
    vals = np.broadcast_to(rng.standard_normal(count), cols.shape) if constant \
        else rng.standard_normal(cols.shape)
    return gen.Csr(rp, cols[valid].astype(np.int32), vals[valid].copy(), n, n)


def _case(name):
    if name == "gauge":
        return gen.lattice_gauge(101)
    if name == "lap2d":
        return gen.laplacian_2d(90)
    if name == "varcoef":
        return gen.varcoef_poisson_3d(20, seed=3)[0]
    kind, count = name.split("_")
    return _diagonals(20_003, int(count), 0.6 if kind == "ragged" else 1.0, kind == "const")


@pytest.mark.parametrize("name", ["gauge", "lap2d", "varcoef", "full_3", "full_9", "full_10",
                                  "full_12", "full_13", "full_16", "const_9", "const_16",
                                  "ragged_3", "ragged_8", "ragged_9", "ragged_16"])
def test_products_on_both_sides(kspmv, oracle, name):
    A = _case(name)
    M = kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, A.nrows, A.ncols)
    rng = np.random.default_rng(3)
    for k in (1, 2, 9, 33, 50, 57, 63, 64, 65, 66, 100, 113, 127, 128, 130):
        X = rng.uniform(-1, 1, (A.ncols, k))
        Y = torch.full((A.nrows, k), float("nan"), dtype=torch.float64, device="cuda")
        kspmv.batch_spmv(M, torch.from_numpy(X).cuda(), Y)
        got = Y.cpu().numpy()
        # every (row, column) is summed serially in CSR order
        for c in {0, k // 2, k - 1}:
            want = oracle.spmv(A.row_ptr, A.col_idx, A.values, np.ascontiguousarray(X[:, c]))
            assert np.array_equal(got[:, c], want), (name, k, c)
        assert np.isfinite(got).all()
