"""PlanStats is a host getter: after a level-schedule factorization it reports the ordered task
graph's duration without device work, so that it can be read inside a stream capture and takes no
device memory."""
import pytest

from tensors_b200 import matrices as M
from tensors_b200 import ordering as O
from tensors_b200.cholesky import CholeskyDecomposition

pytestmark = pytest.mark.gpu


def _handle():
    A = M.grid_laplacian_3d(20, 0x5EED0091, 1e-2)
    return A, CholeskyDecomposition(A.outer, A.inner, O.nested_dissection(A))


def test_read_inside_a_capture():
    import torch

    A, c = _handle()
    stream = torch.cuda.Stream()
    c.SetStream(stream)
    assert c.NumericFactorization(A.values, 0.0) == 0
    x = torch.zeros(4, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        x += 1
        stats = c.PlanStats()
    graph.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 1.0
    assert stats["graph_makespan_us"] > 0 and stats["graph_tasks"] > 0


def test_takes_no_device_memory_and_leaves_the_schedules_as_they_are():
    import torch

    A, c = _handle()
    assert c.NumericFactorization(A.values, 0.0) == 0
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    before = c.DeviceBytes()
    stats = c.PlanStats()
    assert c.DeviceBytes() == before and torch.cuda.mem_get_info()[0] == free
    tri, rec = c.FactorValues()
    # the graph that was ordered for the getter is the one the persistent launch then runs
    c.SetSchedule("task_graph")
    assert c.NumericFactorization(A.values, 0.0) == 0
    assert c.PlanStats()["graph_makespan_us"] == stats["graph_makespan_us"]
    tri2, rec2 = c.FactorValues()
    assert (tri == tri2).all() and (rec == rec2).all()
