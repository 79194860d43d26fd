"""Overlapped launches of solves without z tables, where ordinary launches and
the auxiliary stream of the low wavenumbers stand between the overlapped ones:
the same bits as the captured solve, which has none, also when repeated."""
import pytest

from pascal_poisson_fft_b200 import PPF_FP32, PPF_FP64, PPF_MIXED
from test_gpu_streams import _setup

pytestmark = pytest.mark.gpu

# cyclic z; the streamed z solve beside the low wavenumbers; one thread per
# system beside them; run-time lengths; FP64 with checkpoints
CASES = [((48, 40, 33), (1, 1, 1), PPF_MIXED), ((256, 160, 64), (1, 1, 0), PPF_MIXED),
         ((128, 128, 200), (1, 1, 0), PPF_MIXED), ((300, 180, 48), (0, 0, 0), PPF_FP32),
         ((256, 250, 200), (0, 0, 0), PPF_FP64)]


@pytest.mark.parametrize("case", CASES)
def test_captured_solve_is_the_same(case):
    import torch
    P, solve = _setup(*case, 31)
    solve()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        solve()
    P.zero_()
    graph.replay()
    torch.cuda.synchronize()
    ref = P.clone()
    for _ in range(10):
        P.zero_()
        solve()
        torch.cuda.synchronize()
        assert torch.equal(P, ref)
