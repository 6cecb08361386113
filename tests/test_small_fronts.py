"""Small fronts taken whole by one CTA (front_kernel): the sizes where its classes, row blocks and
children's chunks end, against the oracle, and the plan's choice on the host."""
import os
import sys

import numpy as np
import pytest

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "oracle"))
import oracle  # noqa: E402

from tensors_b200 import matrices as M, ordering as O
from tensors_b200.cholesky import CholeskyDecomposition


def _star_of_cliques(leaf, cut, count, seed):
    """`count` dense blocks of `leaf` rows, each joined to all of one dense block of `cut` rows that
    is ordered last: leaf fronts of n0 = leaf, n1 = cut, and a root with `count` children."""
    n = leaf * count + cut
    rows, cols = [], []
    for b in range(count):
        i = np.arange(b * leaf, (b + 1) * leaf)
        j = np.concatenate([i, np.arange(leaf * count, n)])
        rows.append(np.repeat(i, len(j)))
        cols.append(np.tile(j, len(i)))
    r, c = np.concatenate(rows), np.concatenate(cols)
    k = np.arange(leaf * count, n)
    r, c = np.concatenate([r, c, np.repeat(k, cut)]), np.concatenate([c, r, np.tile(k, cut)])
    v = np.random.default_rng(seed).standard_normal(len(r))
    S = M.from_coo(n, r, c, v).to_scipy()
    S = S + S.T
    d = np.asarray(abs(S).sum(axis=1)).ravel() + 1.0
    S.setdiag(d)                                         # diagonally dominant: SPD, kappa modest
    S.sort_indices()
    return n, S.indptr.astype(np.int64), S.indices.astype(np.int32), S.data.copy(), S


# (leaf rows, cut rows, children): one tile and one column; row and tile remainders; chunk ends of the
# children (32 columns, 16 children a batch); the largest of each shared-memory class and just beyond
SIZES = [(1, 1, 2), (7, 9, 3), (8, 8, 17), (31, 33, 2), (32, 64, 35), (33, 65, 4), (64, 63, 2), (64, 130, 3), (40, 150, 2),
         (64, 140, 2), (16, 200, 3), (65, 30, 2)]


@pytest.mark.gpu
@pytest.mark.parametrize("leaf,cut,count", SIZES)
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_factor_and_solution_match_the_oracle(leaf, cut, count, precision):
    n, outer, inner, vals, S = _star_of_cliques(leaf, cut, count, leaf + cut)
    c = CholeskyDecomposition(outer, inner)
    c.SetPrecision(precision)
    assert c.NumericFactorization(vals) == 0
    ref = oracle.OracleCholesky(n, outer, inner, None)
    assert ref.factor(vals, 0.0) == 0
    tri, rec = c.FactorValues()
    to, ro = ref.factor_values()
    # both factors are backward stable and the matrix is strictly diagonally dominant (kappa < 1e3):
    # they agree to n kappa u
    tol = n * 1e3 * (2.0 ** -53 if precision == "fp64" else 2.0 ** -24 / 32)
    assert np.abs(tri - to).max() <= tol * np.abs(to).max()
    assert len(ro) == 0 or np.abs(rec - ro).max() <= tol * np.abs(to).max()
    B = np.random.default_rng(3).standard_normal((n, 2))
    X = c.Solve(B)
    assert np.abs(X - ref.solve(B)).max() <= 1e-10 * np.abs(X).max()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["mesh", "grid3d"])
def test_every_schedule_factors_small_and_large_fronts_alike(kind):
    A = M.mesh_laplacian(4000, 3, 1e-2, relative=True) if kind == "mesh" else M.grid_laplacian_3d(13, 4, 1e-2)
    p = O.nested_dissection(A, 16)
    out = []
    for schedule in ("levels", "task_graph", "task_graph_all"):
        c = CholeskyDecomposition(A.outer, A.inner, p)
        c.SetSchedule(schedule)
        for _ in range(2):
            assert c.NumericFactorization(A.values) == 0
        out.append(c.FactorValues())
    for t, r in out[1:]:
        assert np.array_equal(t, out[0][0]) and np.array_equal(r, out[0][1])


def test_plan_of_small_fronts_passes_the_check():
    for A in (M.grid_laplacian_2d(40, 0.0), M.grid_laplacian_3d(12, 1), M.vector_laplacian_3d(6, 1)):
        c = CholeskyDecomposition(A.outer, A.inner, O.nested_dissection(A, 16))
        c.SymbolicFactorization()
        c.CheckPlan()
        st = c.PlanStats()
        # one launch per level of small fronts: never more launches than the separate kinds took
        assert st["factor_launches"] <= 5 * st["panel_tasks"] + 5 * st["levels"]
    for leaf, cut, count in SIZES:
        n, outer, inner, _, _ = _star_of_cliques(leaf, cut, count, 1)
        c = CholeskyDecomposition(outer, inner)
        c.SymbolicFactorization()
        c.CheckPlan()
