"""The panel factorization reads a diagonal tile in every lane before one lane writes over it: the
factor of many blocks at once has the same bits in every run and under every schedule (panel launches
of 384 threads, small fronts of 128 to 384, the persistent kernel's 256)."""
import numpy as np
import pytest
import scipy.sparse as sp

from tensors_b200.cholesky import CholeskyDecomposition

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,count", [(8, 2100), (24, 400), (64, 160), (72, 90)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_factor_bits_repeat(rows, count, precision):
    rng = np.random.default_rng(rows)
    G = rng.standard_normal((rows, rows)) / np.sqrt(rows)
    S = sp.block_diag([sp.coo_array(np.eye(rows) + 0.25 * (G @ G.T))] * count, format="csr")
    S.sort_indices()
    values = S.data * (1.0 + 0.125 * rng.random(count).repeat(rows * rows))       # every block its own multiple
    first = None
    for schedule in ("levels", "task_graph_all"):
        c = CholeskyDecomposition(S.indptr.astype(np.int64), S.indices.astype(np.int32))
        c.SetPrecision(precision)
        if precision == "fp64":
            c.SetSchedule(schedule)
        for _ in range(8):
            assert c.NumericFactorization(values) == 0
            tri, _ = c.FactorValues()
            first = tri if first is None else first
            assert np.array_equal(tri, first)
