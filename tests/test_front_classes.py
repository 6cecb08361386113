"""Launch classes of the small fronts (128, 256 and 384 threads, several launches a level) and batches
of their children (16 at a time), with what the plan chose asserted and the factor compared bit for
bit with the task graph's separate kernels; fronts of different panel counts side by side."""
import numpy as np
import pytest
import scipy.sparse as sp
from plan_lists import FRONT, SOLVE, plan_lists

from tensors_b200.cholesky import CholeskyDecomposition


def _blocks_and_tail(sizes, tail, seed=0):
    """Dense blocks of `sizes` rows, each coupled to a dense tail; diagonally dominant values."""
    D = sp.block_diag([sp.coo_array(np.ones((m, m))) for m in sizes])
    edge = sp.coo_array(np.ones((sum(sizes), tail)))
    S = sp.block_array([[D, edge], [edge.T, sp.coo_array(np.ones((tail, tail)))]], format="csr")
    S.sort_indices()
    n = S.shape[0]
    rows = np.repeat(np.arange(n), np.diff(S.indptr))
    T = sp.csr_array((-np.random.default_rng(seed).random(S.nnz), S.indices, S.indptr), shape=S.shape)
    v = ((T + T.T) * 0.5).tocsr().data
    v[rows == S.indices] = np.diff(S.indptr) + 1.0
    return sp.csr_array((v, S.indices, S.indptr), shape=S.shape)


# sizes, tail -> thread classes of the launches with small fronts, lowest level first
CLASSES = {
    "many near the smallest class's limit": ([8] * 2040, 120, [128]),             # 71 KB of 74
    "many, all classes": ([8] * 1990 + [16, 24, 40, 64] * 5, 112, [384, 256, 128]),
    "two classes": ([48] * 90 + [8] * 90, 130, [384, 256]),
    "few, one launch": ([48] * 70 + [8] * 70, 130, [384]),
    "children in batches of 16": ([3] * 35, 20, [256]),
}


@pytest.mark.parametrize("case", sorted(CLASSES))
def test_classes(case):
    sizes, tail, threads = CLASSES[case]
    S = _blocks_and_tail(sizes, tail)
    p = plan_lists(S.indptr, S.indices)
    launches = [x for x in p["whole"] if x["kind"] == FRONT and x["level"] == 0]
    assert [x["tc_count"] for x in launches] == threads
    assert len(p["whole"]) < len(p["factor"])
    if case == "children in batches of 16":
        assert max(t[2] for t in p["front_tasks"]) > 32      # three batches, the root taken whole


@pytest.mark.parametrize("rows,tail,tiny", [(2, 6, True), (3, 16, True), (8, 16, True), (9, 16, False), (8, 17, False)])
def test_tiny_solve_tasks(rows, tail, tiny):
    S = _blocks_and_tail([rows] * 300, tail)
    p = plan_lists(S.indptr, S.indices)
    leaves = sum(1 for f in p["fronts"] if f[2] == 0 and f[0] == rows)
    for name in ("lower", "upper"):
        warps = sum(x["small_count"] for x in p[name] if x["kind"] == SOLVE and x["level"] == 0)
        assert (warps >= leaves and leaves > 250) if tiny else warps == 0


@pytest.mark.gpu
@pytest.mark.parametrize("case", sorted(CLASSES))
def test_factor_bits_of_every_class(case):
    sizes, tail, _ = CLASSES[case]
    S = _blocks_and_tail(sizes, tail)
    factors = []
    for schedule in ("levels", "task_graph_all"):
        c = CholeskyDecomposition(S.indptr.astype(np.int64), S.indices.astype(np.int32))
        c.SetSchedule(schedule)
        for _ in range(2):
            assert c.NumericFactorization(S.data) == 0
        factors.append(c.FactorValues())
    assert np.array_equal(factors[0][0], factors[1][0]) and np.array_equal(factors[0][1], factors[1][1])
    b = np.random.default_rng(3).standard_normal((S.shape[0], 2))
    x = c.Solve(b)
    # diagonally dominant by half: condition number below 10
    assert np.linalg.norm(b - S @ x) / np.linalg.norm(b) < 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("defer", [1, 2, 3, 4])
@pytest.mark.parametrize("tail", [1, 70])
def test_panel_counts_side_by_side(defer, tail):
    # fronts of 1, 2, 3 and 5 panels (some cut short) in one level: every front's pending rows and
    # look-ahead parts end at another step
    S = _blocks_and_tail([300, 190, 128, 60, 257, 65, 3], tail, seed=defer)
    n = S.shape[0]
    A = S.toarray()
    factors = []
    for graph in (True, False):
        c = CholeskyDecomposition(S.indptr.astype(np.int64), S.indices.astype(np.int32))
        c.SetPlanOptions(defer, 1, 256)
        c.SetUseGraph(graph)
        assert c.NumericFactorization(S.data) == 0
        factors.append(c.GetU().toarray())
        U, p = factors[-1], np.asarray(c.GetPermutation())
        # Cholesky's backward error (n + 2) u |U^T| |U|, |U^T| |U| <= max a_ii, twice that for products
        # with explicit inverses of well-conditioned blocks
        assert np.abs(U.T @ U - A[np.ix_(p, p)]).max() <= 2 * (n + 2) * 2.0 ** -53 * np.abs(A).max()
    assert np.array_equal(factors[0], factors[1])
