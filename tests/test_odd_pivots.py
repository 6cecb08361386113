"""Pivots that are zero, infinite or not a number: the mixed-precision factorization raises or passes
them and never refuses a matrix (its refined solve reports what it cannot solve)."""
import numpy as np
import pytest

from tensors_b200.cholesky import CholeskyDecomposition, TBError

pytestmark = pytest.mark.gpu


def _dense(n, seed):
    G = np.random.default_rng(seed).standard_normal((n, n)) / np.sqrt(n)
    A = np.eye(n) + 0.25 * (G @ G.T)
    return A, np.arange(0, n * n + 1, n, dtype=np.int64), np.tile(np.arange(n, dtype=np.int32), n)


@pytest.mark.parametrize("n", [2, 14, 40, 70])
@pytest.mark.parametrize("value", [0.0, np.nan, np.inf])
@pytest.mark.parametrize("schedule", ["levels", "task_graph_all"])
def test_mixed_factorization_refuses_no_pivot(n, value, schedule):
    A, outer, inner = _dense(n, n)
    for row in sorted({0, n // 2, n - 1}):
        B = A.copy()
        B[row, :] = B[:, row] = 0.0                          # alone: its floor is the entry's own
        B[row, row] = value
        c = CholeskyDecomposition(outer, inner)
        c.SetPrecision("mixed")
        c.SetSchedule(schedule)
        assert c.NumericFactorization(B.ravel()) == 0
        with pytest.raises(TBError):
            c.Solve(np.ones(n))
        assert c.NumericFactorization(A.ravel()) == 0        # the handle goes on
        assert np.linalg.norm(A @ c.Solve(np.ones(n)) - 1.0) < 1e-10


@pytest.mark.parametrize("n", [2, 8, 14, 40, 64])
@pytest.mark.parametrize("schedule", ["levels", "task_graph_all"])
def test_infinite_pivot_eliminates_its_row_alone(n, schedule):
    # inside one panel: the row of U is scaled to zero and the other rows factor as without it
    A, outer, inner = _dense(n, n + 1)
    for row in sorted({0, n // 2, n - 1}):
        B = A.copy()
        B[row, row] = np.inf
        c = CholeskyDecomposition(outer, inner)
        c.SetSchedule(schedule)
        assert c.NumericFactorization(B.ravel()) == 0
        U, p = c.GetU().toarray(), np.asarray(c.GetPermutation())
        at = int(np.where(p == row)[0][0])
        assert not U[at, at + 1:].any()
        keep = np.delete(np.arange(n), at)
        R = U[np.ix_(keep, keep)]
        # rows before it are finite multiples; the bound of Cholesky's backward error for the rest
        assert np.abs(R.T @ R - A[np.ix_(p[keep], p[keep])]).max() <= 2 * (n + 2) * 2.0 ** -53 * np.abs(A).max()
