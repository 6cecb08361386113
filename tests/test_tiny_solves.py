"""Solve steps of tiny fronts (at most 8 rows and 16 rest rows), a warp each in launches of many
tasks: fronts of 1 to 9 rows with 0 to 17 rest rows side by side, both sides of both limits, for
widths with and without full 8- and 16-column tiles, by their residuals."""
from __future__ import annotations

import numpy as np
import pytest

from tensors_b200.cholesky import CholeskyDecomposition


def _arrow(rows, rest, copies, seed):
    """Blocks of `rows` unknowns, each coupled to `rest` of the last 17: one front a block."""
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    n = rows * copies + 17
    I, J, V = [], [], []
    for b in range(copies):
        blk = np.arange(b * rows, (b + 1) * rows)
        cols = rows * copies + np.sort(rng.choice(17, rest, replace=False))
        idx = np.concatenate([blk, cols])
        g = rng.standard_normal((rows, idx.size)) * 0.1
        for r in range(rows):
            I.append(np.full(idx.size, blk[r])); J.append(idx); V.append(g[r])
    I.append(np.repeat(np.arange(n - 17, n), 17)); J.append(np.tile(np.arange(n - 17, n), 17)); V.append(np.full(17 * 17, 0.01))
    A = sp.csr_matrix((np.concatenate(V), (np.concatenate(I), np.concatenate(J))), shape=(n, n))
    # diagonally dominant: condition number below 10
    A = A + A.T
    A = A + sp.diags(2.0 * np.abs(A).sum(axis=1).A1 + 1.0)
    A = A.tocsr(); A.sort_indices()
    return A


@pytest.mark.parametrize("rows,rest", [(1, 0), (3, 6), (8, 16), (9, 17)])
def test_plans_are_checked(rows, rest):
    A = _arrow(rows, rest, 1100, 1)
    c = CholeskyDecomposition(A.indptr.astype(np.int32), A.indices.astype(np.int32), np.arange(A.shape[0], dtype=np.int32))
    c.SymbolicFactorization()
    c.CheckPlan()


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("rows,rest", [(1, 0), (1, 6), (3, 17), (7, 8), (8, 1), (8, 16), (9, 17)])
@pytest.mark.parametrize("k", [1, 9, 24, 65])
def test_tiny_fronts_solve(rows, rest, k, precision):
    A = _arrow(rows, rest, 1100, 7 * rows + rest)
    n = A.shape[0]
    c = CholeskyDecomposition(A.indptr.astype(np.int32), A.indices.astype(np.int32), np.arange(n, dtype=np.int32))
    if precision == "mixed":
        c.SetPrecision("mixed")
        c.SetRefinement(1e-13, 30)
    assert c.NumericFactorization(A.data, 0.0) == 0
    b = np.random.default_rng(k).standard_normal((n, k))
    x = c.Solve(b).reshape(n, k)
    if precision == "mixed":
        # the refinement's own target, per column in the 2-norm (and the rounding of this residual)
        assert (np.linalg.norm(A @ x - b, axis=0) / np.linalg.norm(b, axis=0)).max() < 2e-13
    else:
        # backward error of a stable solve with condition number below 10: a few dozen roundings
        assert np.abs(A @ x - b).max() / np.abs(b).max() < 1e-12
        y = c.UpperSolve(c.LowerSolve(b)).reshape(n, k)
        assert np.abs(y - x).max() / np.abs(x).max() < 1e-12
