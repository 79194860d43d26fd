"""The z solve from tables of its right-hand-side-independent half, which
small and mid-size grids take: chunk edges (16 rows), the smallest and tall
columns (d' kept in shared memory or checkpointed), every spectrum kind and
the cyclic sequence, against the oracle with the tolerances of the other
parity tests."""
import numpy as np
import pytest

from _util import gpu_solve, oracle_solve, rel_l2
from pascal_poisson_fft_b200 import PPF_FP64, PPF_MIXED
from pascal_poisson_fft_b200 import workloads as W

pytestmark = pytest.mark.gpu
KINDS = [(1, 1, 0), (1, 0, 0), (0, 1, 0), (0, 0, 0), (1, 1, 1), (0, 0, 1)]


@pytest.mark.parametrize("nz", [3, 4, 15, 16, 17, 32, 33, 49])
@pytest.mark.parametrize("pbc", KINDS)
def test_chunk_edges(nz, pbc):
    p = W.random_problem(np.random.default_rng(nz), 20, 12, nz, pbc, beta=0.0 if pbc[2] else 1.0)
    R = oracle_solve(p)
    assert rel_l2(gpu_solve(p, precision=PPF_FP64), R) < 1e-12
    assert rel_l2(gpu_solve(p, precision=PPF_MIXED, max_sweeps=3), R) < 1e-10


@pytest.mark.parametrize("shape,pbc", [((8, 6, 700), (1, 1, 0)), ((8, 6, 1024), (1, 1, 0)), ((96, 80, 300), (1, 1, 0)),
                                       ((96, 80, 300), (0, 0, 1))])
def test_tall_columns(shape, pbc):
    p = W.random_problem(np.random.default_rng(shape[2]), *shape, pbc)
    assert rel_l2(gpu_solve(p, precision=PPF_FP64), oracle_solve(p)) < 1e-12
