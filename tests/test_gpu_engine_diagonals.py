"""Engine systems on eight diagonals, the most their form holds, and systems
that find no room for their values by diagonal and run from their CSR arrays:
the bits of the persistent step."""
import numpy as np
import pytest

from num_b200 import generators as gen

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _on_diagonals(n, offs, constant, every=1):
    """Symmetric and dominant on the diagonals `offs` (0 among them), entries
    beside the main one only between rows that are multiples of `every`."""
    offs = np.array(sorted(offs))
    i = np.arange(n, dtype=np.int64)
    cols = i[:, None] + offs
    valid = (cols >= 0) & (cols < n)
    off = offs != 0
    valid[:, off] &= (i[:, None] % every == 0) & (cols[:, off] % every == 0)
    vals = np.full(cols.shape, -1.0) if constant else -1.0 - ((i[:, None] + cols) % 7) / 8.0
    vals[:, ~off] = 2.0 * len(offs)
    rp = np.concatenate([[0], np.cumsum(valid.sum(1))]).astype(np.int32)
    return gen.Csr(rp, cols[valid].astype(np.int32), vals[valid].copy(), n, n)


def _solve(nmlib, systems, persistent, max_nnz, precision="fp32"):
    from num_b200.solver import BatchSolver
    rng = np.random.default_rng(13)
    systems = [(A, rng.standard_normal(A.nrows)) for A in systems]
    nmlib.nm_solver_set_persistent(persistent)
    try:
        S = BatchSolver(max_rows=sum(A.nrows + 8 for A, _ in systems), max_nnz=max_nnz,
                        max_systems=len(systems), precision=precision)
        return [(x, i["iters"], i["residual"])
                for x, i in S.solve(systems, max_iter=150, chunk=32)]
    finally:
        nmlib.nm_solver_set_persistent(0)


def _same(a, b):
    for (x, it, res), (y, jt, sres) in zip(a, b):
        assert it == jt and res == sres and np.array_equal(x, y)


# seven and one that only one side of the matrix has; with all of them a block
# of 256 rows holds 2,048 nonzeros, the most a block may
@pytest.mark.parametrize("precision", ["fp32", "fp64", "bf16"])
@pytest.mark.parametrize("constant", [True, False])
def test_eight_diagonals(kspmv, nmlib, constant, precision):
    A = _on_diagonals(131_073, [-500, -40, -1, 0, 1, 40, 500], constant)
    # an entry of value 0 beside each row's last: the eighth diagonal
    S = A.to_scipy().tocoo()
    i = np.arange(A.nrows - 777)
    rows, cols = np.concatenate([S.row, i]), np.concatenate([S.col, i + 777])
    vals = np.concatenate([S.data, np.zeros(i.size)])
    order = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=A.nrows))]).astype(np.int32)
    B = gen.Csr(rp, cols[order].astype(np.int32), vals[order], A.nrows, A.ncols)
    assert np.diff(B.row_ptr).max() == 8
    nnz = B.nnz + 32
    _same(_solve(nmlib, [B], 0, nnz, precision), _solve(nmlib, [B], 1, nnz, precision))


def test_no_room_for_values_by_diagonal(kspmv, nmlib):
    # 7 n values for each of two systems, of which the second has 2.5 n
    # nonzeros, in 9/8 of (7 + 2.5) n: the second runs from its CSR arrays; with
    # more room, by its diagonals
    full = _on_diagonals(140_000, [-500, -40, -1, 0, 1, 40, 500], False)
    thin = _on_diagonals(140_000, [-800, -400, -8, 0, 8, 400, 800], False, every=4)
    tight = full.nnz + thin.nnz + 64
    assert 7 * thin.nrows > tight + tight // 8 + 64 - 7 * full.nrows
    a = _solve(nmlib, [full, thin], 0, tight)
    _same(a, _solve(nmlib, [full, thin], 0, 2 * tight))
    _same(a, _solve(nmlib, [full, thin], 1, tight))
