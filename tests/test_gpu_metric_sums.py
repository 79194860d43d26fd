"""Plane sums of the z-metric gradient where they cancel: the terms df (u_{k+1}
- u_k) are of one sign in the lower half of every plane and of the other in the
upper half, as a large-scale field's are.  The gradient with respect to dmx3 is
compared with the same sums in extended precision of the df the call returned.
A sum that runs over the whole plane in every thread and block rounds like a
random walk, about eps sqrt(N) times a term (8 times that is allowed); one over
contiguous pieces of 4096 cells first grows to thousands of terms (over 100
times as far)."""
import numpy as np
import pytest

from pascal_poisson_fft_b200 import PPF_FP64
from pascal_poisson_fft_b200 import workloads as W
from test_gpu_adjoint import _gpu_adjoint

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n1m,n2m", [(256, 256), (512, 384), (360, 250)])
def test_cancelling_plane_sums(n1m, n2m):
    import pascal_poisson_fft_b200 as ppf
    rng = np.random.default_rng(n1m)
    nz, at = 8, 3   # u steps between the levels `at` and `at` + 1 alone
    p = W.random_problem(rng, n1m, n2m, nz, (1, 1, 0), beta=1.0)
    m = p.metrics
    plan = ppf.Plan(n1m, n2m, nz, p.L1, p.L2, *p.pbc, precision=PPF_FP64)
    xc = 2.0 * np.pi * (np.arange(n1m) + 0.5) / n1m
    g = np.broadcast_to(np.cos(xc), p.shape).copy()
    half = np.where(np.arange(n2m) < n2m // 2, 1.0, -1.0)[:, None]
    df = _gpu_adjoint(p, g, plan=plan)
    err, bound = [], []
    for _ in range(4):
        step = half * np.sign(df[at]) * np.exp(0.7 * rng.standard_normal((n2m, n1m)))
        u = np.zeros((nz + 2, n2m + 2, n1m + 2))
        u[at + 2:nz + 1, 1:-1, 1:-1] = step
        got_df, _, ddmx3 = _gpu_adjoint(p, g, u=u, plan=plan)
        assert np.array_equal(got_df, df)
        lower, upper = (df[k].astype(np.longdouble) * step for k in (at, at + 1))
        # dJ/dap_at = -sum df_at step, dJ/dam_{at+1} = sum df_{at+1} step
        j = at + 2
        ap, am = (1.0 / m["dx3"][k + 1] / m["dmx3"][j] for k in (at, at + 1))
        want = (ap * lower.sum() - am * upper.sum()) / m["dmx3"][j]
        rms = float(max(np.sqrt((lower ** 2).mean()), np.sqrt((upper ** 2).mean())))
        err.append(float(ddmx3[j] - want))
        bound.append((ap + am) / m["dmx3"][j] * np.finfo(float).eps * np.sqrt(n1m * n2m) * rms)
    assert np.sqrt(np.mean(np.square(err))) < 8.0 * np.mean(bound), (err, bound)
