"""nm_csr_diagonals: whether the plain SpMV runs a matrix along its diagonals,
by the library's own rules, and the bytes of the matrix it then reads."""
import ctypes as C

import numpy as np
import pytest

from num_b200 import _lib
from num_b200 import generators as gen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _query(M):
    nd, b = C.c_int32(-1), C.c_int64(-1)
    _lib.check(_lib.load().nm_csr_diagonals(M._h, C.byref(nd), C.byref(b)))
    return nd.value, b.value


def _upload(kspmv, A, **kw):
    return kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, A.nrows, A.ncols, **kw)


def test_diagonals_by_the_librarys_rules(kspmv):
    lap = gen.laplacian_2d(40)
    M = _upload(kspmv, lap)
    assert _query(M) == (5, lap.nrows)  # masks of a byte, no values
    kspmv.tune(M, kernel="blocks")
    assert _query(M) == (0, 0)
    var = gen.varcoef_poisson_3d(12, seed=3)[0]
    for precision, size in (("fp64", 8), ("fp32", 4), ("bf16", 2)):
        assert _query(_upload(kspmv, var, precision=precision)) == \
            (7, var.nrows + size * var.nnz)
    # nine diagonals, of which nearly every 32 rows of this small grid have
    # seven or more: 32-row pieces with too many absent values
    gauge = gen.lattice_gauge(40)
    row = np.repeat(np.arange(gauge.nrows), np.diff(gauge.row_ptr))
    pieces = len(set(zip((row // 32).tolist(), (gauge.col_idx - row).tolist())))
    assert 32 * pieces > gauge.nnz * 5 // 4 + 32 * 16
    assert _query(_upload(kspmv, gauge)) == (0, 0)
    # five diagonals, but a row's columns do not ascend
    order = np.concatenate([np.arange(lap.row_ptr[i], lap.row_ptr[i + 1])[::-1]
                            for i in range(lap.nrows)])
    back = gen.Csr(lap.row_ptr, lap.col_idx[order], lap.values[order], lap.nrows, lap.ncols)
    assert _query(_upload(kspmv, back)) == (0, 0)
    assert _lib.load().nm_csr_diagonals(None, None, None) == _lib.NM_ERR_INVALID
