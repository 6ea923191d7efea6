"""The row-block kernel reading x through L1 (matrices whose rows share lines of
x) and past it, against the per-warp gather kernel: both add a row's products
in CSR order, so the same bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _csr(n, ncols, half, extra, seed):
    """Rows of 2 * half + 1 consecutive columns and `extra` random ones."""
    rng = np.random.default_rng(seed)
    start = np.clip(np.arange(n) * ncols // n - half, 0, ncols - 2 * half - 1)
    cols = np.concatenate([start[:, None] + np.arange(2 * half + 1),
                           rng.integers(0, ncols, (n, extra))], 1) if half >= 0 else \
        rng.integers(0, ncols, (n, extra))
    cols.sort(1)
    keep = np.concatenate([np.ones((n, 1), bool), np.diff(cols, axis=1) > 0], 1)
    rp = np.concatenate([[0], np.cumsum(keep.sum(1))]).astype(np.int32)
    return rp, cols[keep].astype(np.int32), rng.standard_normal(int(keep.sum()))


# near: a band with random entries; far: random entries only; mixed: 3/4 near
# on either side of the rule; columns up to the last ones of x (ragged widths)
@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
@pytest.mark.parametrize("n,ncols,half,extra", [
    (5000, 5000, 6, 2), (5003, 4999, 3, 4), (4097, 4098, 1, 6), (3001, 20_011, 4, 3),
    (2000, 60_001, -1, 9), (70, 4001, 8, 8)])
def test_row_blocks_equal_the_gather_kernel(kspmv, n, ncols, half, extra, precision):
    A = kspmv.upload_csr(*_csr(n, ncols, half, extra, n), n, ncols, precision=precision)
    dt = torch.float64 if precision == "fp64" else torch.float32
    g = torch.Generator(device="cuda").manual_seed(n)
    for shift in (0, 1):  # 16-byte aligned x, and x without windows
        x = torch.randn(ncols + 1, dtype=dt, device="cuda", generator=g)[shift:ncols + shift]
        ys = []
        for kernel, tile in (("gather", 2048), ("blocks", 1024), ("blocks", 2048),
                             ("blocks", 4096)):
            kspmv.tune(A, kernel=kernel, tile=tile, stages=2)
            y = torch.full((n,), 7.0, dtype=dt, device="cuda")
            kspmv.spmv(A, x, y)
            ys.append(y)
        for y in ys[1:]:
            assert torch.equal(y, ys[0])
