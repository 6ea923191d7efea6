"""The SpMV on ten to thirteen diagonals, around the step between two instances
of its kernel, with rows that lack some of them: the oracle's bits in every
precision."""
import numpy as np
import pytest

from num_b200 import generators as gen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

OFFS = [-900, -500, -64, -33, -2, -1, 0, 1, 2, 31, 64, 500, 999]


@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
@pytest.mark.parametrize("n", [1001, 160_003])  # one row per thread, and two
@pytest.mark.parametrize("count", [10, 11, 12, 13])
@pytest.mark.parametrize("keep", [1.0, 0.6])
def test_counts_of_diagonals(kspmv, oracle, keep, count, n, precision):
    rng = np.random.default_rng(count)
    i = np.arange(n, dtype=np.int64)
    cols = i[:, None] + np.array(OFFS[13 - count:])
    valid = (cols >= 0) & (cols < n) & (rng.random((n // 32 + 1, count)) < keep)[i // 32]
    rp = np.concatenate([[0], np.cumsum(valid.sum(1))]).astype(np.int32)
    # eighths, exact in every precision: the sums too
    vals = rng.integers(-16, 17, cols.shape) / 8.0
    A = gen.Csr(rp, cols[valid].astype(np.int32), vals[valid], n, n)
    x = rng.integers(-16, 17, n) / 8.0
    M = kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, n, n, precision=precision)
    xt = torch.tensor(x, dtype=torch.float64 if precision == "fp64" else torch.float32,
                      device="cuda")
    y = torch.full_like(xt, float("nan"))
    kspmv.spmv(M, xt, y)
    want = oracle.spmv(A.row_ptr, A.col_idx, A.values, x)
    assert np.array_equal(y.cpu().numpy().astype(np.float64), want)
