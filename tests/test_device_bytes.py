"""DeviceBytes counts what the handle holds on the device: the fronts, the panels' and super-panels'
inverses, the task arrays and the work vectors, against the change in the device's free memory."""
import numpy as np
import pytest
import scipy.sparse as sp

from tensors_b200.cholesky import CholeskyDecomposition

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_against_free_memory(precision):
    import torch

    rows, count = 300, 60                                        # every block a super-panel of 320 x 320 doubles
    rng = np.random.default_rng(1)
    G = rng.standard_normal((rows, rows)) / np.sqrt(rows)
    block = sp.coo_array(np.eye(rows) + 0.25 * (G @ G.T))
    S = sp.block_diag([block] * count, format="csr")
    S.sort_indices()
    b = rng.standard_normal((rows * count, 16))

    def used():
        c = CholeskyDecomposition(S.indptr.astype(np.int64), S.indices.astype(np.int32))
        c.SetPrecision(precision)
        c.SetUseGraph(False)
        c.SymbolicFactorization()
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        assert c.NumericFactorization(S.data) == 0
        c.Solve(b)
        torch.cuda.synchronize()
        return free - torch.cuda.mem_get_info()[0], c.DeviceBytes()

    torch.zeros(1, device="cuda")
    used()                                                       # kernels loaded, pools grown
    taken, counted = used()
    # arrays are taken from the device in pieces of 2 MB: a piece may hold several arrays, or be partly
    # used; below a tenth of the handle's 150 MB
    assert abs(taken - counted) < 0.1 * counted
