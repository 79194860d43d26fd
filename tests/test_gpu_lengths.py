"""Run-time transform lengths: every radix of the schedules, odd half-lengths,
the shortest lines and tiles with a ragged last line or column, in each pair
of boundary conditions, against the oracle with the tolerances of the other
parity tests."""
import numpy as np
import pytest

from _util import gpu_solve, oracle_solve, rel_l2
from pascal_poisson_fft_b200 import PPF_FP64, PPF_MIXED
from pascal_poisson_fft_b200 import workloads as W

pytestmark = pytest.mark.gpu
LENGTHS = [(2, 2), (4, 6), (10, 18), (18, 10), (50, 54), (54, 60), (90, 96), (150, 100), (162, 90), (192, 48),
           (250, 36), (360, 162)]


@pytest.mark.parametrize("pbc", [(1, 1, 0), (1, 0, 0), (0, 1, 0), (0, 0, 0)])
@pytest.mark.parametrize("n1m,n2m", LENGTHS)
def test_lengths(n1m, n2m, pbc):
    p = W.random_problem(np.random.default_rng(n1m + n2m), n1m, n2m, 5, pbc)
    R = oracle_solve(p)
    assert rel_l2(gpu_solve(p, precision=PPF_FP64), R) < 1e-12
    assert rel_l2(gpu_solve(p, precision=PPF_MIXED, max_sweeps=3), R) < 1e-10
