"""The diagonal form's copy of values that vary, on a device whose memory is
nearly all in use: it is made only out of memory that is plentiful, and the CSR
arrays serve alone where it is not, with the same bits."""
import numpy as np
import pytest

from num_b200 import generators as gen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _seven(n):
    """Seven diagonals of varying values, diagonally dominant."""
    offs = np.array([-9000, -90, -1, 0, 1, 90, 9000])
    i = np.arange(n, dtype=np.int64)
    cols = i[:, None] + offs
    valid = (cols >= 0) & (cols < n)
    # symmetric: by the sum of row and column
    vals = -1.0 - ((i[:, None] + cols) % 7) / 8.0
    vals[:, 3] = 16.0
    rp = np.concatenate([[0], np.cumsum(valid.sum(1))]).astype(np.int32)
    return gen.Csr(rp, cols[valid].astype(np.int32), vals[valid], n, n)


@pytest.fixture
def nearly_full():
    """Fills the device until about `left` bytes are free."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []

    def fill(left):
        free = torch.cuda.mem_get_info()[0]
        held.append(torch.empty(free - left, dtype=torch.uint8, device="cuda"))
    yield fill
    held.clear()
    torch.cuda.empty_cache()


N = 1_300_000  # 73 MB of values by diagonal, 114 MB of CSR arrays


def test_upload_copies_values_only_out_of_plenty(kspmv, oracle, nearly_full):
    A = _seven(N)
    x = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, N)).cuda()
    y = torch.empty_like(x)
    csr = 12 * A.nnz + 4 * N
    copy = 8 * 7 * N
    used = []
    for left in (None, csr + 2 * copy):
        if left is not None:
            nearly_full(left)
        before = torch.cuda.mem_get_info()[0]
        M = kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, N, N)
        used.append(before - torch.cuda.mem_get_info()[0])
        y.fill_(float("nan"))
        kspmv.spmv(M, x, y)
        assert np.array_equal(y.cpu().numpy(),
                              oracle.spmv(A.row_ptr, A.col_idx, A.values, x.cpu().numpy()))
        del M
    assert used[0] >= csr + copy  # with the copy ...
    assert used[1] < csr + copy   # ... and without: it would take half of what is left


def test_upload_where_only_the_csr_arrays_fit(kspmv, oracle, nearly_full):
    # 56 MB of values by diagonal, below what is asked about first
    n = 1_000_000
    A = _seven(n)
    x = torch.from_numpy(np.random.default_rng(4).uniform(-1, 1, n)).cuda()
    y = torch.full_like(x, float("nan"))
    csr, copy = 12 * A.nnz + 4 * n, 8 * 7 * n
    nearly_full(csr + copy // 2)
    M = kspmv.upload_csr(A.row_ptr, A.col_idx, A.values, n, n)
    kspmv.spmv(M, x, y)
    assert np.array_equal(y.cpu().numpy(),
                          oracle.spmv(A.row_ptr, A.col_idx, A.values, x.cpu().numpy()))


def test_engine_copies_values_only_out_of_plenty(kspmv, nearly_full):
    from num_b200.solver import BatchSolver
    A = _seven(2 * N)
    b = np.random.default_rng(2).standard_normal(2 * N)
    copy = 4 * (A.nnz + A.nnz // 8)  # 9/8 of the capacity in inner values, 82 MB
    out = []
    for full in (False, True):
        S = BatchSolver(max_rows=2 * N + 8, max_nnz=A.nnz + 32, max_systems=1, precision="fp32")
        if full:
            nearly_full(2 * copy)
        before = torch.cuda.mem_get_info()[0]
        s = S.admit(A, b)
        took = before - torch.cuda.mem_get_info()[0]
        assert took < copy if full else took >= copy
        while s in S.active:
            S.step(32)
        out.append(S.take(s))
        del S
    (x, i), (y, j) = out
    assert i["converged"] and i["iters"] == j["iters"] and np.array_equal(x, y)


def test_row_subsets_hold_no_values_by_diagonal(kspmv):
    """A rank's slice, and its interior and boundary rows as matrices of their
    own: only the slice is multiplied along its diagonals."""
    import ctypes as C

    from num_b200 import _lib
    A = _seven(N)
    lib = _lib.load()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    h = C.c_void_p()
    _lib.check(lib.nm_dist_create(A.row_ptr.ctypes.data, A.col_idx.ctypes.data,
                                  A.values.ctypes.data, N, N, 0, 2, C.byref(h)))
    used = before - torch.cuda.mem_get_info()[0]
    lib.nm_dist_destroy(h)
    csr, copy = 6 * A.nnz + 2 * N, 4 * 7 * N  # of half of the rows
    assert 2 * csr + copy <= used < 2 * csr + 1.5 * copy
