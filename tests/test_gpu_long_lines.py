"""The longest transform lines a plan accepts, run-time tiles of up to 98 KB
with their padding: 2048 and other long lengths in each direction, against the
oracle.  FP64 with the tolerance of the other parity tests.  A mixed solve ends
where the rounding of its FP64 residual does: eps times the largest eigenvalue
over the smallest, at most 4 n^2 / pi^2 eps = 2e-10 a direction at n = 2048."""
import numpy as np
import pytest

from _util import gpu_solve, oracle_solve, rel_l2
from pascal_poisson_fft_b200 import PPF_FP64, PPF_MIXED
from pascal_poisson_fft_b200 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pbc", [(1, 1, 0), (1, 0, 0), (0, 1, 0), (0, 0, 0)])
@pytest.mark.parametrize("n1m,n2m", [(2048, 18), (20, 2048), (2000, 1944), (1620, 1350)])
def test_fp64(n1m, n2m, pbc):
    p = W.random_problem(np.random.default_rng(n1m + n2m), n1m, n2m, 4, pbc)
    assert rel_l2(gpu_solve(p, precision=PPF_FP64), oracle_solve(p)) < 1e-12


@pytest.mark.parametrize("pbc", [(1, 1, 0), (0, 0, 0)])
@pytest.mark.parametrize("n1m,n2m", [(1000, 2048), (1024, 30), (960, 2000)])
def test_mixed(n1m, n2m, pbc):
    p = W.random_problem(np.random.default_rng(n1m + n2m), n1m, n2m, 4, pbc)
    assert rel_l2(gpu_solve(p, precision=PPF_MIXED, max_sweeps=3), oracle_solve(p)) < 4e-10
