"""Stage times count the kernels a solve launches: as many in all as the
solve's captured graph has kernel nodes, with and without z tables."""
import numpy as np
import pytest

from pascal_poisson_fft_b200 import PPF_FP32, PPF_FP64, PPF_MIXED
from pascal_poisson_fft_b200 import workloads as W

pytestmark = pytest.mark.gpu


# (shape, pbc, precision, whether the plan takes z tables)
@pytest.mark.parametrize("shape,pbc,precision,tables", [
    ((32, 24, 20), (1, 1, 0), PPF_FP64, True), ((256, 250, 200), (0, 0, 0), PPF_FP64, False),
    ((32, 24, 20), (1, 1, 0), PPF_MIXED, True), ((256, 160, 64), (1, 1, 0), PPF_MIXED, False),
    ((48, 40, 33), (1, 1, 1), PPF_MIXED, False), ((300, 180, 48), (0, 0, 0), PPF_FP32, False)])
def test_launches_are_those_of_the_graph(shape, pbc, precision, tables):
    import torch
    from cuda.bindings import runtime as rt
    import pascal_poisson_fft_b200 as ppf
    p = W.random_problem(np.random.default_rng(3), *shape, pbc)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda:0")
    plan = ppf.Plan(*shape, p.L1, p.L2, *p.pbc, precision=precision, max_sweeps=2)
    P = torch.zeros(plan.gshape, dtype=torch.float64, device="cuda:0")
    args = [t(p.f), P] + [t(p.metrics[k]) for k in ("dmx1", "dmx2", "dmx3", "dx3")]
    plan.solve(*args)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        plan.solve(*args)
    raw = rt.cudaGraph_t(graph.raw_cuda_graph())
    _, _, n = rt.cudaGraphGetNodes(raw)
    _, nodes, _ = rt.cudaGraphGetNodes(raw, n)
    kernels = sum(rt.cudaGraphNodeGetType(v)[1] == rt.cudaGraphNodeType.cudaGraphNodeTypeKernel for v in nodes)
    plan.stage_timing(True)
    for _ in range(3):
        plan.solve(*args)
    stages = plan.stage_times()
    plan.stage_timing(False)
    assert sum(v[1] for v in stages.values()) == 3 * kernels
    assert (stages["z-coefficients"][1] == 0) == tables
