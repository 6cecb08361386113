"""The FP64 panel chain over several panels: pending updates applied by the potrf, the next panel's
other rows on their own stream, the trsm's chunks at the boundary of pivot and update rows.  Two dense
blocks of `rows` unknowns coupled to a dense tail, for every deferral of the trailing updates, with
captured graphs and with direct launches."""
import numpy as np
import pytest
import scipy.sparse as sp

from tensors_b200.cholesky import CholeskyDecomposition

pytestmark = pytest.mark.gpu


def _blocks(rows, tail, seed):
    """SPD, kappa < 4: the identity plus a quarter of a scaled Gram matrix without the blocks' coupling."""
    rng = np.random.default_rng(seed)
    n = 2 * rows + tail
    A = np.eye(n)
    for b in range(2):
        idx = np.r_[b * rows:(b + 1) * rows, 2 * rows:n]
        G = rng.standard_normal((idx.size, idx.size)) / np.sqrt(idx.size)
        A[np.ix_(idx, idx)] += 0.125 * (G @ G.T)
    return A


@pytest.mark.parametrize("rows,tail", [(65, 1), (128, 63), (193, 65), (257, 130), (330, 7), (450, 200)])
@pytest.mark.parametrize("defer", [1, 2, 3, 4])
def test_factor_over_several_panels(rows, tail, defer):
    A = _blocks(rows, tail, 10 * rows + tail)
    S = sp.csr_matrix(A)
    S.sort_indices()
    n = S.shape[0]
    c = CholeskyDecomposition(S.indptr.astype(np.int64), S.indices.astype(np.int32))
    c.SetPlanOptions(defer, 1, 256)
    factors = []
    for graph in (True, False):
        c.SetUseGraph(graph)
        assert c.NumericFactorization(S.data) == 0
        factors.append(c.GetU().toarray())
        U, p = factors[-1], c.GetPermutation()
        # as for one front (Cholesky's backward error, twice that for products with explicit inverses)
        assert np.abs(U.T @ U - A[np.ix_(p, p)]).max() <= 2 * (n + 2) * 2.0 ** -53 * np.abs(A).max() * 4
    assert np.array_equal(factors[0], factors[1])            # every entry's updates keep their order
    b = np.random.default_rng(n).standard_normal((n, 5))
    x = c.Solve(b)
    assert np.abs(x - np.linalg.solve(A, b)).max() <= 1e-11 * np.abs(x).max()
