"""FP64 factors of dense blocks with nearly dependent rows (condition numbers of 1e8 to 1e15): every
third row is within `gap` (squared) of the one before it, so that 8 x 8 diagonal tiles are nearly
singular.  Fronts taken whole, panels of 64 rows, and a panel after a well-conditioned one."""
import numpy as np
import pytest

from tensors_b200.cholesky import CholeskyDecomposition

pytestmark = pytest.mark.gpu


def _near(n, begin, gap, seed):
    rng = np.random.default_rng(seed)
    G = rng.standard_normal((n, n + 4))
    for r in range(begin + 2, n, 3):
        G[r] = G[r - 1] + np.sqrt(gap) * rng.standard_normal(n + 4)
    A = G @ G.T
    return (A + A.T) / 2


@pytest.mark.parametrize("n,begin,gap", [(n, b, g) for n, b in ((8, 0), (17, 0), (40, 0), (64, 0), (100, 64), (128, 64))
                                         for g in (1e-6, 1e-8, 1e-10, 1e-11) if g > 1e-11 or n <= 64])
@pytest.mark.parametrize("schedule", ["levels", "task_graph_all"])
def test_factor_is_backward_stable(n, begin, gap, schedule):
    outer, inner = np.arange(0, n * n + 1, n, dtype=np.int64), np.tile(np.arange(n, dtype=np.int32), n)
    c = CholeskyDecomposition(outer, inner)
    c.SetSchedule(schedule)
    for seed in range(6):
        A = _near(n, begin, gap, seed)
        # the smallest eigenvalue (about gap / 10) over the largest diagonal entry is above (n + 2) u
        # (u = 2^-53), so that a backward stable factorization runs through
        assert c.NumericFactorization(A.ravel()) == 0
        U = c.GetU().toarray().astype(np.longdouble)
        # Cholesky's bound |U^T U - A| <= (n + 2) u |U^T| |U| with |U^T| |U| <= max a_ii, twice that
        # for the tiles solved by their inverse (pivots of at least 1/16 of their diagonal entries)
        assert np.abs(U.T @ U - A).max() <= 2 * (n + 2) * 2.0 ** -53 * np.abs(A).max()
