"""Fronts of 65 to 255 rows beside a front of 256 rows or more step by super-panels.  Where such a
block's rows are nearly dependent its inverse is not used: each sweep's residual stays that of panel
steps, which the same block takes when it is alone."""
import numpy as np
import pytest
import scipy.sparse as sp

from tensors_b200.cholesky import CholeskyDecomposition

SIZES = (300, 200, 130, 65, 192, 40, 3, 1)


def _near(n, gap, seed):
    """Every third row within `gap` (squared) of the one before it."""
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((n, n + 4))
    for r in range(2, n, 3):
        G[r] = G[r - 1] + np.sqrt(gap) * rng.standard_normal(n + 4)
    A = G @ G.T
    return (A + A.T) / 2


def _well(n, seed):
    G = np.random.default_rng(seed).standard_normal((n, n)) / np.sqrt(n)
    return np.eye(n) + 0.25 * (G @ G.T)


def _blocks(gap):
    return [_near(n, gap, n) if n in (200, 130, 65) else _well(n, n) for n in SIZES]      # 192: uses its inverse


def _handle(blocks, precision="fp64"):
    S = sp.block_diag([sp.coo_array(b) for b in blocks], format="csr")
    S.sort_indices()
    c = CholeskyDecomposition(S.indptr.astype(np.int64), S.indices.astype(np.int32), np.arange(S.shape[0], dtype=np.int32))
    c.SetPrecision(precision)
    return c, S.data


def test_plan_guards_the_fronts_below_256_rows():
    c, _ = _handle(_blocks(1e-6))
    c.SymbolicFactorization()
    c.CheckPlan()
    st = c.PlanStats()
    assert st["super_panels"] == 5 and st["levels"] == 1          # 300, 200, 192, 130 and 65 rows
    for block in _blocks(1e-6)[1:]:
        c, _ = _handle([block])
        c.SymbolicFactorization()
        assert c.PlanStats()["super_panels"] == 0                 # alone: panel steps


def _residuals(blocks, precision, k, upper):
    """Per block |b - M x| / |x| of one sweep, M = U or U^T the block's own factor."""
    c, values = _handle(blocks, precision)
    assert c.NumericFactorization(values) == 0
    p = np.asarray(c.GetPermutation())
    where = np.argsort(p)                                        # caller's row -> factor's row
    U = c.GetU().toarray()
    M = (U if upper else U.T).astype(np.longdouble)
    rhs, begin, at = np.empty((len(p), k)), 0, []
    for block in blocks:
        rows = np.sort(where[begin:begin + len(block)])
        begin += len(block)
        assert rows[-1] - rows[0] == len(block) - 1
        at.append(slice(rows[0], rows[-1] + 1))
        rhs[at[-1]] = (M[at[-1], at[-1]] @ np.random.default_rng(len(block)).standard_normal((len(block), k))).astype(np.float64)
    b = np.empty_like(rhs)
    b[p] = rhs
    x = (c.UpperSolve(b) if upper else c.LowerSolve(b)).reshape(rhs.shape)[p]
    return [np.linalg.norm((rhs[s] - M[s, s] @ x[s]).astype(np.float64)) / np.linalg.norm(x[s]) for s in at]


@pytest.mark.gpu
@pytest.mark.parametrize("gap,precision", [(1.0, "fp64"), (1e-4, "fp64"), (1e-6, "fp64"), (1e-2, "mixed")])
@pytest.mark.parametrize("k", [1, 8, 16, 33, 65])
@pytest.mark.parametrize("upper", [False, True])
def test_residual_of_each_sweep_is_that_of_panel_steps(gap, precision, k, upper):
    blocks = _blocks(gap)
    together = _residuals(blocks, precision, k, upper)
    for n, block, residual in list(zip(SIZES, blocks, together))[1:]:
        alone, = _residuals([block], precision, k, upper)
        # the same operations on the same factor up to the order of sums: a factor of 4 for what that
        # changes, and a few roundings at the block's scale where the residual happens to be small
        assert residual <= 4 * alone + 8 * 2.0 ** -53 * np.sqrt(np.abs(block).sum(axis=1).max())
