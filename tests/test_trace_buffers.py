"""The time-stamp buffers follow the plan: tracing is enabled on one plan and another schedule, other
plan options or another precision make the task lists longer afterwards."""
import numpy as np
import pytest

from tensors_b200 import matrices as M
from tensors_b200 import ordering as O
from tensors_b200.cholesky import CholeskyDecomposition, TBError

pytestmark = pytest.mark.gpu


def _changes(c):
    yield lambda: c.SetSchedule("task_graph_all")
    yield lambda: c.SetPlanOptions(1, 0, 256)
    yield lambda: c.SetSolveSchedule("task_graph_all")
    yield lambda: c.SetPrecision("mixed")
    yield lambda: c.SetPlanOptions(4, 2, 128)
    yield lambda: c.SetSchedule("task_graph")
    yield lambda: c.SetSupernodeStrategy(1)


def test_traces_after_plan_changes():
    A = M.grid_laplacian_3d(15, 0x5EED00A1, 1e-2)
    c = CholeskyDecomposition(A.outer, A.inner, O.nested_dissection(A))
    c.SetRefinement(1e-12, 30)
    assert c.NumericFactorization(A.values, 0.0) == 0
    c.SetTrace(True)                                         # sized for the level schedule's plan
    b = np.random.default_rng(1).standard_normal((A.n, 2))
    for change in _changes(c):
        change()
        assert c.NumericFactorization(A.values, 0.0) == 0
        x = c.Solve(b)
        assert np.linalg.norm(b - A.to_scipy() @ x) / np.linalg.norm(b) < 1e-11
        t, st = c.Trace(), c.PlanStats()
        assert len(t) == st["graph_tasks"]
        if st["graph_tasks"]:
            # taken, waits met, done: in order, every task on a CTA of the launch
            assert (t[:, 2] <= t[:, 3]).all() and (t[:, 3] <= t[:, 4]).all() and (t[:, 2] > 0).all()
            assert (t[:, 5] < st["graph_ctas"]).all()
        assert len(c.SolveTrace()) == 2 * st["solve_graph_tasks"]


def test_no_trace_of_a_plan_that_has_not_run():
    A = M.grid_laplacian_3d(12, 0x5EED00A2, 1e-2)
    c = CholeskyDecomposition(A.outer, A.inner, O.nested_dissection(A))
    assert c.NumericFactorization(A.values, 0.0) == 0
    c.SetTrace(True)
    c.SetSchedule("task_graph_all")
    c.PlanStats()                                            # the new plan exists, its factorization does not
    with pytest.raises(TBError):
        c.Trace()
