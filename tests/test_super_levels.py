"""Levels that solve by super-panels: when the largest front of a level has 256 pivot rows, every
front of more than one panel there steps by super-panels and the one-panel fronts' step runs in the
level's first diagonal launch.  The sweeps are compared with the panel-step sweeps (those of the
no-allocation solve) on grids whose fronts end inside 64-row panels and 64-column chunks, for
widths with 16-byte rows and without (an odd leading dimension), and for the widths' last columns."""
from __future__ import annotations

import numpy as np
import pytest

from tensors_b200 import _lib
from tensors_b200 import matrices as M
from tensors_b200 import ordering as O
from tensors_b200.cholesky import CholeskyDecomposition


def _banded(n, w):
    import scipy.sparse as sp

    rng = np.random.default_rng(0x5EED0071)
    S = sp.random(n, n, density=2.0 / n, random_state=rng, format="csr")
    D = sp.block_diag([sp.csr_matrix(np.ones((m, m))) for m in (w, 130, 65, 40, n - w - 235)], format="csr")
    A = ((S + S.T) * 0.1 + D + sp.identity(n) * (4.0 * n)).tocsr()
    A.sort_indices()
    return A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, np.arange(n, dtype=np.int32), A


def _grid():
    A = M.grid_laplacian_3d(23, 0x5EED0072, 1e-2)            # top separator 23 x 23 = 529 rows: 512 + 17
    return A.outer, A.inner, A.values, O.nested_dissection(A), A.to_scipy()


# fronts of 300 (four panels and 44 rows), 130, 65 and 40 rows side by side; the same with the largest below the line
CASES = {"blocks300": lambda: _banded(700, 300), "blocks250": lambda: _banded(700, 250), "grid23": _grid}


@pytest.mark.parametrize("case", sorted(CASES))
def test_plan_is_checked(case):
    outer, inner, _, perm, _ = CASES[case]()
    c = CholeskyDecomposition(outer, inner, perm)
    c.SymbolicFactorization()
    c.CheckPlan()
    st = c.PlanStats()
    if case == "grid23":
        assert st["super_panels"] == 2                       # the root: 512 and 17 rows (its halves have 253)
        assert st["lower_launches_super"] < st["lower_launches"]


@pytest.mark.gpu
@pytest.mark.parametrize("case", sorted(CASES))
@pytest.mark.parametrize("k", [1, 16, 33, 64, 65, 66])
def test_sweeps_agree_with_panel_steps(case, k):
    import torch

    outer, inner, values, perm, S = CASES[case]()
    n = S.shape[0]
    c = CholeskyDecomposition(outer, inner, perm)
    assert c.NumericFactorization(values, 0.0) == 0
    b = np.random.default_rng(k).standard_normal((n, k))
    B = torch.tensor(b, device="cuda")
    X1, X2 = torch.zeros_like(B), torch.zeros_like(B)
    lib = _lib.lib()
    assert lib.tb_chol_solve_device(c.handle, 1.0, B.data_ptr(), k, 0.0, X1.data_ptr(), k, k) == 0
    assert lib.tb_chol_solve_device_noalloc(c.handle, 1.0, B.data_ptr(), k, 0.0, X2.data_ptr(), k, k) == 0
    torch.cuda.synchronize()
    # rounding of two orders of the same sums: cond(A) (about 1e3 for the grid) x n eps = 1e3 x 1e4 x 1e-16
    assert float((X1 - X2).abs().max() / X2.abs().max()) < 1e-9
    x = X1.cpu().numpy()
    assert np.linalg.norm(b - S @ x) / np.linalg.norm(b) < 1e-11
    # forward and back sweeps alone, and the whole solve once more on used buffers
    assert np.linalg.norm(c.UpperSolve(c.LowerSolve(b)) - x) / np.linalg.norm(x) < 1e-11
    assert np.linalg.norm(c.Solve(b) - x) / np.linalg.norm(x) < 1e-11
