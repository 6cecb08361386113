"""A factor swapped in and out of a decomposition whose solves use super-panel inverses (fronts of 256
rows and more): the inverses go with the factor they belong to."""
import numpy as np
import pytest

from tensors_b200 import matrices as M
from tensors_b200 import ordering as O
from tensors_b200.cholesky import CholeskyDecomposition, NumericalFactorization

pytestmark = pytest.mark.gpu


def _residual(A, x, b):
    return np.linalg.norm(b - A.to_scipy() @ x) / np.linalg.norm(b)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_solves_after_swaps(precision):
    A = M.grid_laplacian_3d(23, 0x5EED0081, 1e-2)
    A2 = M.grid_laplacian_3d(23, 0x5EED0082, 1e-2)           # same pattern, other values
    perm = O.nested_dissection(A)
    h = CholeskyDecomposition(A.outer, A.inner, perm)
    h.SetPrecision(precision)
    h.SetRefinement(1e-12, 30)
    h.SymbolicFactorization()
    assert h.PlanStats()["super_panels"] > 0
    b = np.random.default_rng(81).standard_normal((A.n, 3))
    bound = 1e-11                                            # cond(A) is about 1e3; the refinement's target 1e-12
    f = NumericalFactorization()
    assert h.NumericFactorization(A.values, 0.0) == 0
    assert _residual(A, h.Solve(b), b) < bound
    h.SwapNumericalFactorization(f)                          # f <- A's factor
    assert h.NumericFactorization(A2.values, 0.0) == 0
    assert _residual(A2, h.Solve(b), b) < bound
    steps = h.RefinementInfo()[0] if precision == "mixed" else 0
    h.SwapNumericalFactorization(f)                          # h <- A's factor, f <- A2's
    assert _residual(A, h.Solve(b), b) < bound
    if precision == "mixed":
        assert h.RefinementInfo()[0] <= steps + 1 and h.PrecisionInUse()[0] == "mixed"
    fresh = CholeskyDecomposition(A.outer, A.inner, perm)    # a handle that never factored
    fresh.SwapNumericalFactorization(f)
    assert _residual(A2, fresh.Solve(b), b) < bound
    # the two handles go on with their own storage
    assert h.NumericFactorization(A2.values, 0.0) == 0 and fresh.NumericFactorization(A.values, 0.0) == 0
    assert _residual(A2, h.Solve(b), b) < bound and _residual(A, fresh.Solve(b), b) < bound
