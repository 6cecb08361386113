"""A level that holds super-panels and one-panel fronts with rest rows: the one-panel fronts' step
runs inside the level's diagonal launches, forward and back, beside fronts with two and more
super-panels."""
import numpy as np
import pytest
from plan_lists import SUPER_DIAG, plan_lists
from test_front_classes import _blocks_and_tail

from tensors_b200 import _lib
from tensors_b200.cholesky import CholeskyDecomposition

# with fronts of two super-panels (520 rows), of one, below 256 rows, and of one panel; tails of odd and
# even width, within and beyond a chunk of 64
CASES = {"two super-panels": ([520, 300, 130, 65, 40, 20, 3, 1], 70), "one": ([300, 130, 65, 40, 20, 3, 1], 33),
         "no tail to speak of": ([300, 64, 7], 1)}
BELOW = ([250, 130, 65, 40, 20, 3, 1], 33)                   # no front of 256 rows: panel steps


@pytest.mark.parametrize("case", sorted(CASES))
def test_plan(case):
    S = _blocks_and_tail(*CASES[case])
    p = plan_lists(S.indptr, S.indices)
    for name in ("lower_super", "upper_super"):
        shared = [x for x in p[name] if x["kind"] == SUPER_DIAG and x["tc_count"] > 0]
        assert shared
        tasks = [t for x in shared for t in p["rest_tasks"][x["tc_first"]:x["tc_first"] + x["tc_count"]]]
        assert all(t[0] <= 64 for t in tasks) and any(t[1] > 0 and t[4] > max(t[3], 0) for t in tasks)


def test_plan_below_the_line():
    S = _blocks_and_tail(*BELOW)
    c = CholeskyDecomposition(S.indptr.astype(np.int64), S.indices.astype(np.int32))
    c.SymbolicFactorization()
    assert c.PlanStats()["super_panels"] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("k", [1, 2, 8, 17, 32, 33, 64, 65, 129])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sweeps(case, k, precision):
    import torch

    S = _blocks_and_tail(*CASES[case], seed=k)
    n = S.shape[0]
    c = CholeskyDecomposition(S.indptr.astype(np.int64), S.indices.astype(np.int32))
    c.SetPrecision(precision)
    c.SetRefinement(1e-13, 30)
    assert c.NumericFactorization(S.data) == 0
    b = np.random.default_rng(k).standard_normal((n, k))
    # condition number below 10: a few dozen roundings, or the refinement's target
    x = c.Solve(b).reshape(n, k)
    assert (np.linalg.norm(b - S @ x, axis=0) / np.linalg.norm(b, axis=0)).max() < 2e-13
    U, p = c.GetU(), np.asarray(c.GetPermutation())
    y = c.LowerSolve(b).reshape(n, k)
    assert np.linalg.norm(U.T @ y[p] - b[p]) / np.linalg.norm(b) < 1e-13
    z = c.UpperSolve(b).reshape(n, k)
    assert np.linalg.norm(U @ z[p] - b[p]) / np.linalg.norm(b) < 1e-13
    if precision == "fp64":
        # the panel-step sweeps of the no-allocation solve on the same factor
        B = torch.tensor(b, device="cuda")
        X = torch.zeros_like(B)
        assert _lib.lib().tb_chol_solve_device_noalloc(c.handle, 1.0, B.data_ptr(), k, 0.0, X.data_ptr(), k, k) == 0
        torch.cuda.synchronize()
        assert np.abs(X.cpu().numpy().reshape(n, k) - x).max() / np.abs(x).max() < 1e-13
