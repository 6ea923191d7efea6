"""Uploads on both sides of the size up to which the arrays go up as one image
(512 KB): the arrays come back as they were, and the row-block kernel, which
reads the padding of each array, gives the oracle's bits."""
import numpy as np
import pytest

from num_b200 import generators as gen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

_VALUE = {"fp64": 8, "fp32": 4, "bf16": 2}


def _tridiag(n):
    i = np.arange(n, dtype=np.int64)
    cols = np.stack([i - 1, i, i + 1], 1)
    valid = (cols >= 0) & (cols < n)
    rp = np.concatenate([[0], np.cumsum(valid.sum(1))]).astype(np.int32)
    ci = cols[valid].astype(np.int32)
    # sixteenths: exact in every precision
    return gen.Csr(rp, ci, ((np.arange(ci.size) % 61) - 30) / 16.0, n, n)


def _image_bytes(n, es):
    up = lambda b: (b + 255) & ~255
    nnz_pad = ((3 * n - 2 + 7) & ~7) + 8
    return up(4 * (n + 9)) + up(4 * nnz_pad) + es * nnz_pad


@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
@pytest.mark.parametrize("side", ["one", "small", "last", "first", "large"])
def test_upload_both_ways(kspmv, oracle, precision, side):
    es = _VALUE[precision]
    last = max(n for n in range(13_000, 24_000) if _image_bytes(n, es) <= 512 << 10)
    A = _tridiag({"one": 1, "small": 7, "last": last, "first": last + 1, "large": 40_000}[side])
    M = kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, A.nrows, A.ncols, precision=precision)
    rp, ci, v = kspmv.download_csr(M)
    assert np.array_equal(rp, A.row_ptr) and np.array_equal(ci, A.col_idx)
    if precision == "bf16":
        v = np.asarray(v).view(np.uint16).astype(np.uint32) << 16
        v = v.view(np.float32)
    assert np.array_equal(np.asarray(v, np.float64), A.values)
    # eighths: products and sums are exact in 32 bits too
    x = ((np.arange(A.ncols) % 17) - 8) / 8.0
    xt = torch.tensor(x, dtype=torch.float64 if precision == "fp64" else torch.float32,
                      device="cuda")
    yt = torch.empty_like(xt)
    want = oracle.spmv(A.row_ptr, A.col_idx, A.values, x)
    for kernel in ("auto", "blocks"):
        kspmv.tune(M, kernel=kernel)
        yt.fill_(float("nan"))
        kspmv.spmv(M, xt, yt)
        assert np.array_equal(yt.cpu().numpy().astype(np.float64), want)


def test_upload_without_nonzeros(kspmv):
    M = kspmv.upload_csr(np.zeros(301, np.int32), np.zeros(0, np.int32), np.zeros(0), 300, 5)
    y = torch.full((300,), float("nan"), dtype=torch.float64, device="cuda")
    kspmv.spmv(M, torch.ones(5, dtype=torch.float64, device="cuda"), y)
    assert torch.count_nonzero(y).item() == 0


@pytest.mark.parametrize("dim,L", [(2, 1), (2, 2), (2, 3), (2, 17), (3, 1), (3, 2), (3, 3), (3, 9)])
@pytest.mark.parametrize("precision", ["fp64", "fp32", "bf16"])
def test_assembled_laplacian_has_the_uploaded_ones_form(kspmv, oracle, dim, L, precision):
    import ctypes as C

    from num_b200 import _lib
    A = gen.laplacian_2d(L) if dim == 2 else gen.laplacian_3d(L)
    handles = [kspmv.laplacian(dim, L, precision=precision),
               kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, A.nrows, A.ncols,
                                precision=precision)]
    x = ((np.arange(A.ncols) % 17) - 8) / 8.0
    want = oracle.spmv(A.row_ptr, A.col_idx, A.values, x)
    seen = []
    for M in handles:
        nd, b = C.c_int32(), C.c_int64()
        _lib.check(_lib.load().nm_csr_diagonals(M._h, C.byref(nd), C.byref(b)))
        seen.append((nd.value, b.value))
        xt = torch.tensor(x, dtype=torch.float64 if precision == "fp64" else torch.float32,
                          device="cuda")
        y = torch.full_like(xt, float("nan"))
        kspmv.spmv(M, xt, y)
        assert np.array_equal(y.cpu().numpy().astype(np.float64), want)
    assert seen[0] == seen[1] and seen[0][0] == (2 * dim + 1 if L > 1 else 1)
