"""The calls a user of this package makes, as performance cases.

Every case goes through the public Python entry points (Plan, Batch,
autograd.PoissonSolve, tdma_many / tdma_cycl_many) on device arrays, the way a
flow solver, a parameter study, an inverse problem or a line-implicit time
stepper calls them.  listed() names the representative ones, draw() samples
the same ranges, exact() restates the outputs in plain float64 torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import pascal_poisson_fft_b200 as ppf
from pascal_poisson_fft_b200 import workloads as W
from pascal_poisson_fft_b200.autograd import PoissonSolve

TWO_PI = 2.0 * math.pi
PREC = {"fp64": ppf.PPF_FP64, "mixed": ppf.PPF_MIXED, "fp32": ppf.PPF_FP32}
MODES = 24


def _solve(name, n1m, n2m, n3m, px, py, pz, beta, precision, sweeps, kind="solve"):
    return {"name": name, "kind": kind, "n1m": n1m, "n2m": n2m, "n3m": n3m, "px": px, "py": py, "pz": pz,
            "beta": beta, "precision": precision, "sweeps": sweeps}


def listed():
    return [
        # the smallest grid of the configurations: a pressure solve inside a
        # small time-stepping loop, where launches and latency are the cost
        _solve("cube_64_fp64", 64, 64, 64, True, True, False, 0.0, "fp64", -1),
        # an odd, ragged grid (composite lengths, an odd level count) between
        # side walls in x, stretched towards the z walls
        _solve("ragged_100x90x33_fp64", 100, 90, 33, False, True, False, 1.5, "fp64", -1),
        # the mixed-precision method at its default two sweeps on a mid-size
        # channel grid
        _solve("channel_128_mixed", 128, 128, 128, True, True, False, 1.5, "mixed", -1),
        # periodic in all three directions (the cyclic z solver)
        _solve("periodic_160x128x96_fp64", 160, 128, 96, True, True, True, 0.0, "fp64", -1),
        # the cavity: walls on every side (DCT in x and y), stretched z
        _solve("cavity_256_fp64", 256, 256, 256, False, False, False, 2.0, "fp64", -1),
        # the large channel in the reference's precision
        _solve("channel_512_fp64", 512, 512, 512, True, True, False, 1.5, "fp64", -1),
        # the same grid by FP32 transforms and one FP64 refinement sweep
        _solve("channel_512_mixed", 512, 512, 512, True, True, False, 1.5, "mixed", 1),
        # a large FP32 solve of radix-3 lengths (a preconditioner's accuracy)
        _solve("slab_768x768x384_fp32", 768, 768, 384, True, True, False, 1.5, "fp32", -1),
        # a parameter study: many uneven problems, solved by one call
        {"name": "study_64_fp64", "kind": "batch", "count": 64, "grids": 4, "precision": "fp64", "sweeps": -1},
        # a smaller study by the mixed method
        {"name": "study_24_mixed", "kind": "batch", "count": 24, "grids": 11, "precision": "mixed", "sweeps": 2},
        # an inverse problem: the solve and its gradient with respect to the
        # right-hand side and the z metric, through torch.autograd
        _solve("inverse_256x256x128_fp64", 256, 256, 128, True, True, False, 2.0, "fp64", -1, kind="grad"),
        # a line-implicit step: batched tridiagonal systems given as arrays
        {"name": "lines_65536x256", "kind": "tdma", "n_sys": 65536, "n_row": 256, "cyclic": False},
    ]


def _smooth(lo, hi):
    """Even 2-3-5 products in [lo, hi] (the transform lengths a plan accepts)."""
    out = []
    for n in range(lo, hi + 1, 2):
        m = n
        for r in (2, 3, 5):
            while m % r == 0:
                m //= r
        if m == 1:
            out.append(n)
    return out


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _log_smooth(rng, lo, hi):
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(_smooth(lo, hi), key=lambda n: abs(n - x))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    what = rng.choice(["solve"] * 5 + ["grad", "batch", "tdma"])
    if what == "tdma":
        n_row = _log_int(rng, 16, 1024)
        n_sys = _log_int(rng, 1000, min(300000, (1 << 26) // n_row))
        return {"kind": "tdma", "n_sys": n_sys, "n_row": n_row, "cyclic": rng.random() < 0.5}
    if what == "batch":
        precision = rng.choice(["fp64", "mixed"])
        return {"kind": "batch", "count": rng.randint(4, 32), "grids": rng.randint(1, 10 ** 6),
                "precision": precision, "sweeps": rng.choice([1, 2]) if precision == "mixed" else -1}
    top = 1 << 24 if what == "grad" else 1 << 27   # cells
    while True:
        n1m, n2m, n3m = _log_smooth(rng, 32, 768), _log_smooth(rng, 32, 768), _log_int(rng, 24, 512)
        if n1m * n2m * n3m <= top:
            break
    precision = "fp64" if what == "grad" else rng.choice(["fp64", "fp64", "mixed", "fp32"])
    case = _solve("", n1m, n2m, n3m, rng.random() < 0.6, rng.random() < 0.6, what == "solve" and rng.random() < 0.15,
                  rng.choice([0.0, 1.0, 1.5, 2.0]), precision, rng.choice([1, 2]) if precision == "mixed" else -1,
                  kind=what)
    del case["name"]
    return case


# ---- problems ---------------------------------------------------------------

def _problem(case):
    pbc = (case["px"], case["py"], case["pz"])
    beta = 0.0 if pbc[2] else case["beta"]   # a periodic z axis is uniform
    return W.build_metrics(W.Problem("case", case["n1m"], case["n2m"], case["n3m"], TWO_PI, TWO_PI, 1.0, pbc, beta))


def _problems(case):
    return W.config4(seed=case["grids"], count=case["count"], generate=False)


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64).to(_device())


def _field(p, seed):
    """A smooth field of MODES separable modes with a |k|^-2 spectrum that fit
    the boundaries, plus 1e-3 white noise, of zero volume mean."""
    rng = np.random.Generator(np.random.PCG64(seed))
    gen = torch.Generator(device=_device())
    gen.manual_seed(int(rng.integers(1 << 62)))
    kx, ky, kz = rng.integers(0, 13, MODES), rng.integers(0, 13, MODES), rng.integers(0, 7, MODES)
    amp = rng.normal(size=MODES) / (1.0 + kx ** 2 + ky ** 2 + (math.pi * kz) ** 2)
    phase = rng.uniform(0.0, TWO_PI, size=(2, MODES))
    xc, yc, zc = W.centres(p)
    fx = np.cos(kx[:, None] * xc + phase[0][:, None]) if p.pbc[0] else np.cos(kx[:, None] * xc / 2.0)
    fy = np.cos(ky[:, None] * yc + phase[1][:, None]) if p.pbc[1] else np.cos(ky[:, None] * yc / 2.0)
    fz = np.cos(kz[:, None] * (TWO_PI if p.pbc[2] else math.pi) * zc)
    plane = _t(fy)[:, :, None] * _t(fx)[:, None, :]
    f = (_t(amp[:, None] * fz).T @ plane.reshape(MODES, -1)).reshape(p.shape)
    f += 1e-3 * torch.randn(p.shape, dtype=torch.float64, device=f.device, generator=gen)
    w = _t(p.metrics["dx3"][1:p.n3m + 1])
    f -= (f.mean(dim=(1, 2)) * w).sum() / w.sum()
    return f


def _lines(case, seed):
    """Diagonally dominant systems of an implicit diffusion step."""
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed)
    shape = (case["n_row"], case["n_sys"])
    u = lambda: torch.rand(shape, dtype=torch.float64, device=_device(), generator=gen)
    a, c = -(0.2 + u()), -(0.2 + u())
    b = 1.0 - a - c
    d = torch.randn(shape, dtype=torch.float64, device=_device(), generator=gen)
    return a, b, c, d


def prepare(case, seed):
    if case["kind"] == "tdma":
        a, b, c, rhs = _lines(case, seed)
        return {"case": case, "a": a, "b": b, "c": c, "rhs": rhs, "d": torch.empty_like(rhs)}
    if case["kind"] == "batch":
        probs = _problems(case)
        batch = ppf.Batch([dict(n1m=p.n1m, n2m=p.n2m, n3m=p.n3m, L1=p.L1, L2=p.L2, pbc=p.pbc,
                                precision=PREC[case["precision"]], max_sweeps=case["sweeps"]) for p in probs])
        fs = [_field(p, seed * 1000 + k) for k, p in enumerate(probs)]
        Ps = [torch.zeros(p.n3m + 2, p.n2m + 2, p.n1m + 2, dtype=torch.float64, device=_device()) for p in probs]
        m = {k: [_t(p.metrics[k]) for p in probs] for k in ("dmx1", "dmx2", "dmx3", "dx3")}
        return {"case": case, "batch": batch, "fs": fs, "Ps": Ps, "m": m}
    p = _problem(case)
    plan = ppf.Plan(p.n1m, p.n2m, p.n3m, p.L1, p.L2, *p.pbc, precision=PREC[case["precision"]],
                    max_sweeps=case["sweeps"])
    st = {"case": case, "plan": plan, "f": _field(p, seed)}
    st.update({k: _t(p.metrics[k]) for k in ("dmx1", "dmx2", "dmx3", "dx3")})
    if case["kind"] == "grad":
        st["g"] = _field(p, seed + 1)
        for k in ("f", "dx3", "dmx3"):
            st[k].requires_grad_(True)
    else:
        st["P"] = torch.zeros(plan.gshape, dtype=torch.float64, device=_device())
    return st


def run(state):
    kind = state["case"]["kind"]
    if kind == "tdma":
        state["d"].copy_(state["rhs"])   # the solve is in place: this step's right-hand side
        solve = ppf.tdma_cycl_many if state["case"]["cyclic"] else ppf.tdma_many
        solve(state["a"], state["b"], state["c"], state["d"])
        return state["d"]
    if kind == "batch":
        m = state["m"]
        state["batch"].solve(state["fs"], state["Ps"], m["dmx1"], m["dmx2"], m["dmx3"], m["dx3"])
        return state["Ps"]
    if kind == "grad":
        u = PoissonSolve.apply(state["f"], state["dx3"], state["dmx3"], state["plan"], state["dmx1"], state["dmx2"])
        df, ddx3, ddmx3 = torch.autograd.grad(u, (state["f"], state["dx3"], state["dmx3"]), state["g"])
        return {"u": u.detach(), "df": df, "ddx3": ddx3, "ddmx3": ddmx3}
    state["plan"].solve(state["f"], state["P"], state["dmx1"], state["dmx2"], state["dmx3"], state["dx3"])
    return state["P"]


# ---- work -------------------------------------------------------------------

def _solve_work(n1m, n2m, n3m):
    cells = n1m * n2m * n3m
    # transforms there and back (2.5 n log2 n per real line) and the z systems
    return cells * 8 + (n1m + 2) * (n2m + 2) * (n3m + 2) * 8, cells * (5.0 * math.log2(n1m * n2m) + 12.0)


def work(case):
    if case["kind"] == "tdma":
        n = case["n_sys"] * case["n_row"]
        return {"bytes": 5 * 8 * n, "flops": (16 if case["cyclic"] else 9) * n}
    if case["kind"] == "batch":
        w = [_solve_work(p.n1m, p.n2m, p.n3m) for p in _problems(case)]
        return {"bytes": sum(b for b, _ in w), "flops": sum(f for _, f in w)}
    b, f = _solve_work(case["n1m"], case["n2m"], case["n3m"])
    if case["kind"] == "grad":   # f, g read; u, df written
        return {"bytes": 4 * 8 * case["n1m"] * case["n2m"] * case["n3m"], "flops": 2 * f}
    return {"bytes": b, "flops": f}


# ---- the same in plain float64 ------------------------------------------------

def _dct(v, dim, inverse):
    """DCT-II along dim (2 sum x cos), or its inverse, of real or complex data
    by an FFT of the even-odd reordered sequence."""
    v = v.movedim(dim, -1)
    n = v.shape[-1]
    w = torch.polar(torch.ones(n, dtype=torch.float64, device=v.device),
                    -math.pi * torch.arange(n, dtype=torch.float64, device=v.device) / (2 * n))
    if not inverse:
        V = torch.fft.fft(torch.cat((v[..., 0::2], v[..., 1::2].flip(-1)), dim=-1))
        Vm = V.flip(-1).roll(1, dims=-1)
        X = w * V + w.conj() * Vm
        return (X if v.is_complex() else X.real).movedim(-1, dim)
    Xm = torch.cat((torch.zeros_like(v[..., :1]), v[..., 1:].flip(-1)), dim=-1)
    x = torch.fft.ifft(0.5 * w.conj() * (v - 1j * Xm))
    x = x if v.is_complex() else x.real
    h = n // 2
    return torch.stack((x[..., :h], x[..., h:].flip(-1)), dim=-1).flatten(-2).movedim(-1, dim)


def _eig(n, length, periodic, count):
    h = length / n
    if periodic:
        e = [2.0 * (1.0 - math.cos(2.0 * min(m, n - m) * math.pi / n)) / (h * h) for m in range(count)]
    else:
        e = [4.0 * math.sin(0.5 * m * math.pi / n) ** 2 / (h * h) for m in range(count)]
    return _t(np.array(e))


def _poisson(p, f, dx3, dmx3):
    """Interior solution of zero mean.  The z systems are eliminated in the
    subtraction-free form of a diagonally dominant matrix (the pivot is kept
    as ap + q), so the nearly singular low wavenumbers keep full accuracy."""
    nz = p.n3m
    s = torch.fft.rfft(f) if p.pbc[0] else _dct(f, -1, False)
    s = torch.fft.fft(s, dim=1) if p.pbc[1] else _dct(s, 1, False)
    lam = _eig(p.n2m, p.L2, p.pbc[1], s.shape[1])[:, None] + _eig(p.n1m, p.L1, p.pbc[0], s.shape[2])[None, :]
    zero = torch.zeros_like(lam, dtype=torch.bool)
    zero[0, 0] = True
    am = 1.0 / dx3[1:nz + 1] / dmx3[1:nz + 1]
    ap = 1.0 / dx3[1:nz + 1] / dmx3[2:nz + 2]
    one, nil = torch.ones_like(lam), torch.zeros_like(lam)
    cs, gs = [], []
    ratio = g = None
    for k in range(nz):
        q = lam if k == 0 else lam + am[k] * ratio
        piv = q if k == nz - 1 else q + ap[k]
        rhs = -s[k] if k == 0 else -s[k] + am[k] * g
        if k == 0:   # the zero mode is pinned by its first row
            q, piv, rhs = torch.where(zero, one, q), torch.where(zero, one, piv), torch.where(zero, nil, rhs)
        ratio = q / piv
        g = rhs / piv
        c = nil if k == nz - 1 else ap[k] / piv
        if k == 0:
            c = torch.where(zero, nil, c)
        cs.append(c)
        gs.append(g)
    u = gs[-1]
    out = [u]
    for k in range(nz - 2, -1, -1):
        u = gs[k] + cs[k] * u
        out.append(u)
    del cs, gs, s
    s = torch.stack(out[::-1])
    del out
    s = torch.fft.ifft(s, dim=1) if p.pbc[1] else _dct(s, 1, True)
    if not p.pbc[0]:
        s = _dct(s, -1, True)
        s = s.real if s.is_complex() else s
    else:
        s = torch.fft.irfft(s, n=p.n1m)
    return s - s.mean()


def _ghosted(p, u):
    P = torch.zeros(p.n3m + 2, p.n2m + 2, p.n1m + 2, dtype=torch.float64, device=u.device)
    P[1:-1, 1:-1, 1:-1] = u
    for walls in (True, False):
        for axis in range(3):   # x, y, z
            if p.pbc[axis] == walls:
                continue
            Q = P.movedim(2 - axis, 0)
            if walls:
                m = p.metrics[("dmx1", "dmx2", "dmx3")[axis]]
                n = Q.shape[0] - 2
                lo, hi = (m[1] + m[2]) ** 2, (m[n + 1] + m[n]) ** 2
                Q[0] = (lo * Q[1] - m[1] ** 2 * Q[2]) / (lo - m[1] ** 2)
                Q[n + 1] = (hi * Q[n] - m[n + 1] ** 2 * Q[n - 1]) / (hi - m[n + 1] ** 2)
            else:
                Q[0], Q[-1] = Q[-2].clone(), Q[1].clone()
    return P


def _thomas(a, b, c, d):
    """Elimination from the last row upwards, substitution downwards."""
    n = d.shape[0]
    al, ds = [a[-1] / b[-1]], [d[-1] / b[-1]]
    for k in range(n - 2, -1, -1):
        piv = b[k] - c[k] * al[-1]
        ds.append((d[k] - c[k] * ds[-1]) / piv)
        al.append(a[k] / piv)
    x = [ds[-1]]
    for k in range(1, n):
        x.append(ds[n - 1 - k] - al[n - 1 - k] * x[-1])
    return torch.stack(x)


def exact(case, seed):
    if case["kind"] == "tdma":
        a, b, c, d = _lines(case, seed)
        if not case["cyclic"]:
            return _thomas(a, b, c, d)
        # Sherman-Morrison on the corners a[0] (x_0 <- x_{n-1}) and c[-1]
        gam = -b[0]
        bb = b.clone()
        bb[0] -= gam
        bb[-1] -= c[-1] * a[0] / gam
        uu = torch.zeros_like(d)
        uu[0], uu[-1] = gam, c[-1]
        y, q = _thomas(a, bb, c, d), _thomas(a, bb, c, uu)
        r = a[0] / gam
        return y - q * ((y[0] + r * y[-1]) / (1.0 + q[0] + r * q[-1]))
    if case["kind"] == "batch":
        out = []
        for k, p in enumerate(_problems(case)):
            u = _poisson(p, _field(p, seed * 1000 + k), _t(p.metrics["dx3"]), _t(p.metrics["dmx3"]))
            out.append(_ghosted(p, u))
        return out
    p = _problem(case)
    f, dx3, dmx3 = _field(p, seed), _t(p.metrics["dx3"]), _t(p.metrics["dmx3"])
    if case["kind"] == "grad":
        for t in (f, dx3, dmx3):
            t.requires_grad_(True)
        u = _poisson(p, f, dx3, dmx3)
        df, ddx3, ddmx3 = torch.autograd.grad(u, (f, dx3, dmx3), _field(p, seed + 1))
        return {"u": u.detach(), "df": df, "ddx3": ddx3, "ddmx3": ddmx3}
    with torch.no_grad():
        return _ghosted(p, _poisson(p, f, dx3, dmx3))
