"""arena_for's capacities stay within the budget together with the inner values
by diagonal that the engine may allocate later (9/8 of max_nnz)."""
import pytest

from num_b200.solver import arena_bytes, arena_for


@pytest.mark.parametrize("precision,value", [("fp64", 8), ("fp32", 4), ("bf16", 2)])
@pytest.mark.parametrize("budget", [1e6, 1e9, 16e9, 64e9, 160e9])
def test_budget_holds_the_values_by_diagonal(precision, value, budget):
    for nnz_per_row in (1, 5, 8, 64):
        rows, nnz = arena_for(budget, nnz_per_row, precision)
        assert arena_bytes(rows, nnz, precision) + value * (nnz + nnz // 8 + 64) <= budget
