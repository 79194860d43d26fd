"""Tridiagonal systems whose factors stay on chip: chunk edges of the
elimination (8 rows) and the substitution (16), the shortest column taken,
ragged last warps, d' in shared memory or in place, one wave and several,
against the oracle with the tolerance of the other tests."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_tdma import _gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_sys,n_row", [(33, 24), (31, 25), (1, 31), (65, 32), (64, 33), (100, 40), (97, 41), (40, 440),
                                         (37, 880), (6000, 118), (9500, 230), (60000, 48)])
@pytest.mark.parametrize("cyclic", [False, True])
def test_against_oracle(n_sys, n_row, cyclic):
    rng = np.random.default_rng(n_sys + n_row)
    a = rng.uniform(-1, 1, (n_row, n_sys)); c = rng.uniform(-1, 1, (n_row, n_sys))
    b = (np.abs(a) + np.abs(c) + rng.uniform(0.2, 2, (n_row, n_sys))) * rng.choice([-1.0, 1.0], (n_row, n_sys))
    d = rng.standard_normal((n_row, n_sys))
    got = _gpu(a, b, c, d, cyclic)
    ref = [v.copy() for v in (a, b, c, d)]
    O.tdma_many(*ref, cyclic=cyclic)
    assert np.linalg.norm(got - ref[3]) / np.linalg.norm(ref[3]) < 1e-13
