"""Calls of different sizes from two host threads at once, on streams of their
own: a kernel's limit of dynamic shared memory belongs to the function, so one
thread's call must not lower it under the other's.  Pairs that share a kernel:
tridiagonal lines kept on chip and not, plans by z tables, by the streamed and
low-|k| z kernels, and by run-time transform tiles.  Each thread's results have
the bits of the same calls made alone."""
import threading

import numpy as np
import pytest

from pascal_poisson_fft_b200 import PPF_FP64, PPF_MIXED
from pascal_poisson_fft_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _lines(n_sys, n_row, cyclic):
    import torch
    import pascal_poisson_fft_b200 as ppf
    rng = np.random.default_rng(n_row)
    t = lambda v: torch.as_tensor(v, dtype=torch.float64, device="cuda:0")
    a, c = (t(rng.uniform(-1, 1, (n_row, n_sys))) for _ in range(2))
    b, rhs = 3.0 + a.abs() + c.abs(), t(rng.standard_normal((n_row, n_sys)))
    d, zero = torch.empty_like(rhs), torch.zeros_like(rhs)
    solve = ppf.tdma_cycl_many if cyclic else ppf.tdma_many
    fn = ppf.lib().ppf_tdma_cycl_many if cyclic else ppf.lib().ppf_tdma_many

    def call():
        # the C calls back to back (a zero right-hand side stays zero), then
        # one whole call for the results
        ptrs, st = [v.data_ptr() for v in (a, b, c, zero)], torch.cuda.current_stream().cuda_stream
        for _ in range(200):
            if fn(*ptrs, n_sys, n_row, st) != 0:
                raise RuntimeError(ppf.lib().ppf_last_error().decode())
        d.copy_(rhs)
        solve(a, b, c, d)
    return d, call


def _plan(shape, pbc, precision, sweeps=1):
    import torch
    import pascal_poisson_fft_b200 as ppf
    p = W.random_problem(np.random.default_rng(shape[2]), *shape, pbc)
    t = lambda v: torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device="cuda:0")
    plan = ppf.Plan(*shape, p.L1, p.L2, *p.pbc, precision=precision, max_sweeps=sweeps)
    P = torch.zeros(plan.gshape, dtype=torch.float64, device="cuda:0")
    f, args = t(p.f), [t(p.metrics[k]) for k in ("dmx1", "dmx2", "dmx3", "dx3")]
    return P, lambda: plan.solve(f, P, *args)


PAIRS = {
    "lines_on_chip": (100, lambda: _lines(64, 30, False), lambda: _lines(64, 300, False)),
    "lines_on_chip_cyclic": (100, lambda: _lines(64, 30, True), lambda: _lines(64, 300, True)),
    "lines": (100, lambda: _lines(64, 900, False), lambda: _lines(64, 1000, False)),
    "lines_cyclic": (100, lambda: _lines(64, 500, True), lambda: _lines(64, 700, True)),
    "z_tables": (600, lambda: _plan((32, 24, 200), (1, 1, 0), PPF_FP64), lambda: _plan((32, 24, 300), (1, 1, 0), PPF_FP64)),
    "z_stream": (200, lambda: _plan((256, 160, 100), (1, 1, 0), PPF_MIXED),
                 lambda: _plan((256, 160, 160), (1, 1, 0), PPF_MIXED)),
    "run_time_tiles": (600, lambda: _plan((32, 1000, 6), (1, 1, 0), PPF_FP64),
                       lambda: _plan((32, 1500, 6), (1, 1, 0), PPF_FP64)),
}


@pytest.mark.parametrize("name", sorted(PAIRS))
def test_two_threads(name):
    import torch
    loops, *makes = PAIRS[name]
    jobs = [m() for m in makes]
    for _, call in jobs:
        call()
    torch.cuda.synchronize()
    refs = [out.clone() for out, _ in jobs]
    for out, _ in jobs:
        out.zero_()
    torch.cuda.synchronize()
    errors, start = [], threading.Barrier(2)

    def work(call):
        torch.cuda.set_device(0)
        with torch.cuda.stream(torch.cuda.Stream()):
            start.wait(60)
            try:
                for _ in range(loops):
                    call()
            except Exception as exc:
                errors.append(str(exc))

    threads = [threading.Thread(target=work, args=(call,)) for _, call in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join(300)
    torch.cuda.synchronize()
    assert not errors, errors[0]
    assert all(torch.equal(out, ref) for (out, _), ref in zip(jobs, refs))
