"""The panel factorization (64 x 64 diagonal blocks by 8 x 8 tiles) at the sizes where tiles and
panels end: dense matrices, which are one front of ceil(n / 64) panels."""
import numpy as np
import pytest

from tensors_b200.cholesky import CholeskyDecomposition

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 7, 8, 9, 16, 17, 31, 56, 57, 63, 64, 65, 72, 127, 129]


def _dense(n, seed):
    """Well-conditioned SPD matrix (kappa < 4) and its full pattern."""
    G = np.random.default_rng(seed).standard_normal((n, n)) / np.sqrt(n)
    A = np.eye(n) + 0.25 * (G @ G.T)
    return A, np.arange(0, n * n + 1, n, dtype=np.int64), np.tile(np.arange(n, dtype=np.int32), n)


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_dense_factor_at_tile_and_panel_edges(n, precision):
    A, outer, inner = _dense(n, n)
    c = CholeskyDecomposition(outer, inner)
    c.SetPrecision(precision)
    assert c.NumericFactorization(A.ravel()) == 0
    U = c.GetU().toarray()
    # Cholesky's backward error: |U^T U - A| <= (n + 2) u |U|^T |U|, here |U|^T |U| <= n max a_ii;
    # twice that for the products with explicit 8 x 8 and 64 x 64 inverses (kappa(U) < 2)
    unit = 2.0 ** -53 if precision == "fp64" else 2.0 ** -24
    assert np.abs(U.T @ U - A).max() <= 2 * (n + 2) * unit * np.abs(A).max() * min(n, 4)
    assert not np.tril(U, -1).any()
    B = np.random.default_rng(n + 1).standard_normal((n, 3))
    X = c.Solve(B)
    expect = np.linalg.solve(A, B)
    assert np.abs(X - expect).max() <= 1e-11 * np.abs(expect).max()


@pytest.mark.parametrize("row", [0, 3, 8, 21, 63, 64, 70])
def test_first_failing_row_is_reported_anywhere_in_a_panel(row):
    n = 80
    A, outer, inner = _dense(n, 5)
    A[row, row] = -1.0
    c = CholeskyDecomposition(outer, inner)
    # the first row of a dense matrix is a 1 x 1 supernode of its own, which takes sqrt(|a|) and
    # never fails (Multifrontal.hpp:471); the others are one supernode
    sn = int(c.RowToSN()[row])
    single = np.diff(c.SN_RowPointers())[sn] == 1
    assert single == (row == 0)
    assert c.NumericFactorization(A.ravel()) == (0 if single else 1)
    if not single:
        assert c.FailedSupernode() == sn and not c.NumericallyGoodQ()


@pytest.mark.parametrize("rows", [(1,), (7, 9), (8, 40, 63), (64, 65)])
def test_raised_pivots_in_any_tile(rows):
    # row r equals row r - 1 up to 1e-9 of its diagonal: its pivot (~1e-9) falls below the mixed
    # path's floor (1e-5 of the diagonal) and is raised; all others stay (kappa < 4 without these rows)
    n = 80
    A, outer, inner = _dense(n, 9)
    for r in rows:
        A[r, :] = A[r - 1, :]
        A[:, r] = A[:, r - 1]
        A[r, r] = A[r - 1, r - 1] * (1.0 + 1e-9)
    c = CholeskyDecomposition(outer, inner)
    c.SetPrecision("mixed")
    assert c.NumericFactorization(A.ravel()) == 0
    assert c.PerturbedPivots() == len(rows)
    assert np.isfinite(c.GetU().toarray()).all()
