"""Variants taken only where there are more blocks than fit at once: the z
tables with d' checkpointed instead of kept (cyclic FP64, and FP32 spectra),
and short tridiagonal lines on chip in several waves; against the oracle with
the tolerances of the other parity tests."""
import numpy as np
import pytest

from _util import gpu_solve, oracle_solve, rel_l2
from oracle import oracle as O
from pascal_poisson_fft_b200 import PPF_FP64, PPF_MIXED
from pascal_poisson_fft_b200 import workloads as W
from test_gpu_tdma import _gpu

pytestmark = pytest.mark.gpu


# a block a 32 real columns; of 148 SMs each holds as many as 227 KB of shared
# memory allows with d' of every level kept: 200 levels four (592 blocks), 400
# two (296), 128 of FP32 spectra six (888)
@pytest.mark.parametrize("shape,pbc,precision,tol", [
    ((160, 128, 200), (1, 1, 1), PPF_FP64, 1e-12),   # 768 blocks
    ((150, 180, 201), (0, 0, 1), PPF_FP64, 1e-12),   # 900
    ((90, 100, 400), (0, 1, 1), PPF_FP64, 1e-12),    # 306
    ((150, 180, 128), (1, 1, 0), PPF_MIXED, 1e-10)])   # 900
def test_checkpointed_tables(shape, pbc, precision, tol):
    p = W.random_problem(np.random.default_rng(shape[2]), *shape, pbc)
    assert rel_l2(gpu_solve(p, precision=precision, max_sweeps=3), oracle_solve(p)) < tol


# four resident blocks of 32 systems an SM are 18 944 systems
@pytest.mark.parametrize("n_sys,n_row,cyclic", [(300000, 32, False), (150001, 40, False), (200003, 24, False),
                                                (300000, 40, True), (100001, 101, True)])
def test_lines_in_several_waves(n_sys, n_row, cyclic):
    rng = np.random.default_rng(n_sys)
    a = rng.uniform(-1, 1, (n_row, n_sys)); c = rng.uniform(-1, 1, (n_row, n_sys))
    b = (np.abs(a) + np.abs(c) + rng.uniform(0.2, 2, (n_row, n_sys))) * rng.choice([-1.0, 1.0], (n_row, n_sys))
    d = rng.standard_normal((n_row, n_sys))
    got = _gpu(a, b, c, d, cyclic)
    ref = [v.copy() for v in (a, b, c, d)]
    O.tdma_many(*ref, cyclic=cyclic)
    assert np.linalg.norm(got - ref[3]) / np.linalg.norm(ref[3]) < 1e-13
