"""Overlapped kernel launches of a solve: the same bits as the solve captured
into a CUDA graph (which does without) and as solves running beside one
another on several streams."""
import numpy as np
import pytest

from pascal_poisson_fft_b200 import PPF_FP64, PPF_MIXED
from pascal_poisson_fft_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _setup(shape, pbc, precision, seed):
    import torch
    import pascal_poisson_fft_b200 as ppf
    p = W.random_problem(np.random.default_rng(seed), *shape, pbc)
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda:0")
    plan = ppf.Plan(*shape, p.L1, p.L2, *p.pbc, precision=precision, max_sweeps=2)
    P = torch.zeros(plan.gshape, dtype=torch.float64, device="cuda:0")
    args = [t(p.metrics[k]) for k in ("dmx1", "dmx2", "dmx3", "dx3")]
    f = t(p.f)
    return P, lambda: plan.solve(f, P, *args)


CASES = [((32, 48, 20), (1, 1, 0), PPF_FP64), ((50, 30, 17), (0, 1, 0), PPF_MIXED), ((64, 64, 33), (1, 0, 1), PPF_FP64)]


@pytest.mark.parametrize("case", CASES)
def test_captured_solve_is_the_same(case):
    import torch
    P, solve = _setup(*case, 11)
    solve()
    torch.cuda.synchronize()
    ref = P.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        solve()
    P.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(P, ref)


def test_solves_on_several_streams():
    import torch
    jobs = [_setup(*c, 20 + k) for k, c in enumerate(CASES)]
    for _, solve in jobs:
        solve()
    torch.cuda.synchronize()
    refs = [P.clone() for P, _ in jobs]
    streams = [torch.cuda.Stream() for _ in jobs]
    for _ in range(20):
        for (_, solve), s in zip(jobs, streams):
            with torch.cuda.stream(s):
                solve()
    torch.cuda.synchronize()
    assert all(torch.equal(P, r) for (P, _), r in zip(jobs, refs))
