"""Fronts with many children: a few wide ones (more than 80 rows, more than 64k entries of child
update matrices) keep the extend-add by parent rows, which spreads their rows over the chip; narrow
ones, and many wide ones in a level, are taken whole.  Factors are the same bits either way."""
import numpy as np
import pytest
import scipy.sparse as sp
from plan_lists import FRONT, plan_lists

from tensors_b200.cholesky import CholeskyDecomposition


def _groups(leaf, count, sep, top, groups):
    """`groups` separators of `sep` rows, each with `count` leaf blocks of `leaf` rows below it, all
    coupled to the last `top` rows."""
    g = leaf * count + sep
    low = sp.block_diag([sp.coo_array(np.ones((leaf, leaf)))] * count)
    edge = sp.coo_array(np.ones((leaf * count, sep)))
    group = sp.block_array([[low, edge], [edge.T, sp.coo_array(np.ones((sep, sep)))]])
    edge = sp.coo_array(np.ones((g * groups, top)))
    S = sp.block_array([[sp.block_diag([group] * groups), edge], [edge.T, sp.coo_array(np.ones((top, top)))]], format="csr")
    S.sort_indices()
    return S


def _values(S):
    """Diagonally dominant."""
    n = S.shape[0]
    rows = np.repeat(np.arange(n), np.diff(S.indptr))
    v = -np.random.default_rng(n).random(S.nnz)
    T = sp.csr_array((v, S.indices, S.indptr), shape=S.shape)
    v = ((T + T.T) * 0.5).tocsr().data
    v[rows == S.indices] = np.diff(S.indptr) + 1.0
    return v


@pytest.mark.parametrize("groups,count,sep,top,whole", [
    (3, 16, 8, 200, False),      # children of 208 rows: 16 x 21,736 entries
    (12, 8, 8, 200, False),
    (40, 8, 8, 200, True),       # enough such fronts to fill the chip
    (3, 4, 8, 100, True),        # 4 x 5,886 entries
    (3, 64, 8, 56, True),        # 64 rows: whole with any number of children
    (3, 512, 3, 14, True),
])
def test_choice(groups, count, sep, top, whole):
    S = _groups(3, count, sep, top, groups)
    p = plan_lists(S.indptr, S.indices)
    # (a separator takes its last leaves in, and the last separator merges with the top rows)
    separators = [f for f in p["fronts"] if f[2] == 1 and f[1] == top]
    assert len(separators) == groups - 1
    assert all(bool(f[4]) == whole for f in separators)
    assert any(launch["kind"] == FRONT for launch in p["whole"])
    children = max(t[2] for t in p["front_tasks"] if t[1] in (0, top) or not whole)
    assert children >= count - 2 if whole else children == 0


@pytest.mark.gpu
@pytest.mark.parametrize("groups,count,sep,top", [(3, 16, 8, 200), (40, 8, 8, 200), (3, 64, 8, 56), (3, 17, 3, 14), (2, 33, 3, 14)])
def test_factor_bits_do_not_depend_on_the_choice(groups, count, sep, top):
    S = _groups(3, count, sep, top, groups)
    v = _values(S)
    factors = []
    for schedule in ("levels", "task_graph_all"):
        c = CholeskyDecomposition(S.indptr.astype(np.int64), S.indices.astype(np.int32))
        c.SetSchedule(schedule)
        assert c.NumericFactorization(v) == 0
        factors.append(c.FactorValues())
    assert np.array_equal(factors[0][0], factors[1][0]) and np.array_equal(factors[0][1], factors[1][1])
    b = np.random.default_rng(1).standard_normal(S.shape[0])
    A = sp.csr_array((v, S.indices, S.indptr), shape=S.shape)
    x = c.Solve(b)
    # diagonally dominant: condition number below 1e3
    assert np.linalg.norm(b - A @ x) / np.linalg.norm(b) < 1e-12
