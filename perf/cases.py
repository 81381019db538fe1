"""Performance cases of the contact library: what a user's program calls, over the sizes it is used at.

Kinds of case (each through a public entry point of the package):
  apply      Operator.matvec_: one free-space ("fft") or periodic operator
             apply on device tensors, FP32 or FP64 -- the call that outer
             solvers and time loops make for every step
  tangent    TangentialOperator.matvec_: the two-field Cerruti apply
  solve      ContactSolver.solve: one certified contact problem, gap in,
             pressure (and displacement, gap) out, FP64 or FP32 + FP64 polish
  many       aspher_b200.batch.solve_many: a load / surface sweep in one call
  nested     solve_nested: the cascadic driver from a coarse grid up
  gradient   contact_pressure and its backward pass (inverse design)

Surfaces are seeded self-affine height fields (Hurst exponent 0.6-0.9, 0.002
rms, band [4, 64] cycles per domain, less on small grids), the workload of
the repository's benchmark; every case also takes grid sides that are not
powers of two.
"""

import math

import numpy as np
import torch

from aspher_b200 import ContactSolver, Operator, TangentialOperator, contact_pressure, solve_nested
from aspher_b200.batch import solve_many


def listed():
    return [
        # the smallest: an outer loop in Python that applies the operator of a
        # small grid thousands of times (latency, three launches)
        dict(name="apply fft f64 64", kind="apply", backend="fft", n=64, dtype="f64"),
        # a ragged measured grid, periodic, one time step of a plate model
        dict(name="apply periodic f32 1000", kind="apply", backend="periodic", n=1000,
             dtype="f32"),
        # the benchmark's operator apply
        dict(name="apply fft f32 2048", kind="apply", backend="fft", n=2048, dtype="f32"),
        # the largest FP64 level of the precision study
        dict(name="apply fft f64 4096", kind="apply", backend="fft", n=4096, dtype="f64"),
        # friction loops apply the Cerruti block in every iteration
        dict(name="tangent f64 768", kind="tangent", n=768, dtype="f64"),
        # a small certified solve with every field read back (teaching,
        # unit tests, sweeps over a small cell)
        dict(name="solve fft 128", kind="solve", backend="fft", n=128, load=0.005,
             precision="double", precond="fourier", host=True),
        # the reference's default call on a measured grid of any side, no
        # preconditioner named
        dict(name="solve periodic 600", kind="solve", backend="periodic", n=600, load=0.01,
             precision="double", precond="none", host=False),
        # certified FP64 answers from FP32 iterations
        dict(name="solve fft 1024 mixed", kind="solve", backend="fft", n=1024, load=0.01,
             precision="float_then_double", precond="fourier", host=False),
        # an uneven sweep: many small problems of both backends in one call
        dict(name="many uneven 8", kind="many", count=8, lo=256, hi=1024, pow2=True, tol=1e-8),
        # the benchmark's workload: two backends, three loads each, Ns = 2048,
        # at a tolerance of 1e-6
        dict(name="many 6 x 2048", kind="many", count=6, lo=2048, hi=2048, pow2=True, tol=1e-6),
        # the precision study's call
        dict(name="nested fft 2048", kind="nested", backend="fft", coarsest=64, levels=5,
             load=0.002, precision="double"),
        # gradient of a functional of the pressure (forward and backward)
        dict(name="gradient periodic 512", kind="gradient", backend="periodic", n=512, load=0.01),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi):
    """A grid side: a power of two one time in two, else any (odd ones among them)."""
    n = _log_int(rng, lo, hi)
    if rng.random() < 0.5:
        n = min(max(1 << int(round(math.log2(n))), lo), hi)
    return n


def draw(rng):
    kind = rng.choice(["apply", "apply", "apply", "tangent", "solve", "solve", "solve", "many",
                       "nested", "gradient"])
    backend = rng.choice(["fft", "periodic"])
    load = round(math.exp(rng.uniform(math.log(1e-3), math.log(2e-2))), 5)
    if kind == "apply":
        return dict(kind=kind, backend=backend, n=_side(rng, 32, 4096),
                    dtype=rng.choice(["f32", "f64"]))
    if kind == "tangent":
        return dict(kind=kind, n=_side(rng, 32, 2048), dtype=rng.choice(["f32", "f64"]))
    if kind == "solve":
        n = _side(rng, 64, 1024)
        return dict(kind=kind, backend=backend, n=n, load=load,
                    precision=rng.choice(["double", "float_then_double"]),
                    precond=rng.choice(["fourier", "fourier", "none"]), host=n <= 256)
    if kind == "many":
        lo = _log_int(rng, 64, 512)
        return dict(kind=kind, count=rng.randint(3, 10), lo=lo, hi=2 * lo,
                    pow2=rng.random() < 0.5, tol=1e-8)
    if kind == "nested":
        return dict(kind=kind, backend=backend, coarsest=2 * rng.randint(12, 32),
                    levels=rng.randint(2, 4), load=load,
                    precision=rng.choice(["double", "float_then_double"]))
    return dict(kind=kind, backend=backend, n=_side(rng, 64, 512), load=load)


# ---- inputs ------------------------------------------------------------------------


def _gap(n, seed, hurst=0.8, rms=0.002):
    """g0 = -h of a self-affine height field, an FP64 device vector of n * n cells."""
    gen = torch.Generator("cuda").manual_seed(seed)
    k_hi = min(64.0, n / 4.0)
    k_lo = min(4.0, k_hi / 4.0)
    ky = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")
    kx = torch.fft.rfftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")
    k = torch.hypot(ky[:, None], kx[None, :])
    amp = torch.where((k >= k_lo) & (k <= k_hi), k.clamp_min(1e-9) ** (-(1.0 + hurst)),
                      torch.zeros_like(k))
    ph = torch.rand(k.shape, generator=gen, dtype=torch.float64, device="cuda")
    h = torch.fft.irfft2(torch.polar(amp, 2.0 * math.pi * ph), s=(n, n))
    h = h * (rms / h.std(correction=0))
    return (-h).reshape(-1).contiguous()


def _normal(n, seed, dtype=torch.float64):
    gen = torch.Generator("cuda").manual_seed(seed)
    return torch.randn(n, generator=gen, dtype=torch.float64, device="cuda").to(dtype)


def _dtype(case):
    return torch.float64 if case["dtype"] == "f64" else torch.float32


def _many(case, seed):
    """The problems of a batch and the seeds of their surfaces."""
    probs = []
    if case["lo"] == case["hi"]:  # one surface, three loads, both backends
        for backend in ("fft", "periodic"):
            for load in (0.001, 0.005, 0.02)[:max(1, case["count"] // 2)]:
                probs.append((dict(backend=backend, grid_size=case["hi"], p_nominal=load), 0.8,
                              seed))
        return probs
    rng = np.random.default_rng(case["count"] + 1000 * case["lo"])  # the sweep's plan
    for i in range(case["count"]):
        if case["pow2"]:
            sizes = [s for s in (64, 128, 256, 512, 1024) if case["lo"] <= s <= case["hi"]]
            n = int(rng.choice(sizes)) if sizes else case["hi"]
        else:
            n = int(rng.integers(case["lo"], case["hi"] + 1))
        load = float(math.exp(rng.uniform(math.log(1e-3), math.log(2e-2))))
        probs.append((dict(backend="fft" if i % 2 == 0 else "periodic", grid_size=n,
                           p_nominal=load), float(rng.uniform(0.6, 0.9)), seed * 100 + i))
    return probs


def _side_of(case):
    return case["coarsest"] << case["levels"] if case["kind"] == "nested" else case["n"]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "apply":
        x = _normal(case["n"] ** 2, seed, _dtype(case))
        return dict(kind=kind, op=Operator(case["backend"], case["n"]), x=x,
                    y=torch.empty_like(x))
    if kind == "tangent":
        q = _normal(2 * case["n"] ** 2, seed, _dtype(case))
        return dict(kind=kind, op=TangentialOperator(case["n"]), x=q, y=torch.empty_like(q))
    if kind == "solve":
        g = _gap(case["n"], seed)
        return dict(kind=kind, case=case, gap=g.cpu().numpy() if case["host"] else g,
                    solver=ContactSolver(case["n"], backend=case["backend"]))
    if kind == "many":
        todo = _many(case, seed)
        gaps, seen = [], {}
        for p, hurst, s in todo:
            key = (p["grid_size"], hurst, s)
            if key not in seen:
                seen[key] = _gap(p["grid_size"], s, hurst)
            gaps.append(seen[key])
        return dict(kind=kind, case=case, problems=[p for p, _, _ in todo], gaps=gaps)
    if kind == "nested":
        return dict(kind=kind, case=case, gap=_gap(_side_of(case), seed, rms=0.02))
    n = case["n"]
    return dict(kind=kind, case=case, solver=ContactSolver(n, backend=case["backend"]),
                gap=_gap(n, seed), weight=_normal(n * n, seed + 7919))


def run(state):
    kind = state["kind"]
    if kind in ("apply", "tangent"):
        return state["op"].matvec_(state["x"], state["y"])
    case = state["case"]
    if kind == "solve":
        mixed = case["precision"] == "float_then_double"
        r = state["solver"].solve(state["gap"], case["load"], precond=case["precond"],
                                  precision=case["precision"],
                                  float_tol=2e-5 if mixed else None)
        if case["host"]:
            return dict(pressure=r.pressure, displacement=r.displacement, gap=r.gap,
                        approach=r.approach, area=r.contact_area)
        return dict(pressure=r.pressure_device, approach=r.approach, area=r.contact_area)
    if kind == "many":
        rs = solve_many(state["problems"], state["gaps"], tol=case["tol"],
                        polish_tol=0.5 * case["tol"], float_tol=2e-5)
        return [r.pressure_device for r in rs]
    if kind == "nested":
        r = solve_nested(_side_of(case), state["gap"], case["load"], coarsest=case["coarsest"],
                         backend=case["backend"], precision=case["precision"])
        return dict(pressure=r.pressure_device, approach=r.approach, area=r.contact_area)
    gap = state["gap"].detach().requires_grad_(True)
    p = contact_pressure(state["solver"], gap, case["load"], tol=1e-10)
    (p * state["weight"]).sum().backward()
    return dict(pressure=p.detach(), gradient=gap.grad)


# ---- what a pass cannot do without ---------------------------------------------------


def _apply_flops(n, fields=1):
    """Two real 2-D transforms of the (padded: about 2n) grid's data rows and columns."""
    return fields * 2 * 2.5 * n * n * 2 * math.log2(max(2, n * n))


def _iterations(case):
    """About how many CG iterations the solve of such a surface takes."""
    return {"none": 400, "fourier": 150}.get(case.get("precond"), 150)


def work(case):
    kind = case["kind"]
    if kind in ("apply", "tangent"):
        fields = 2 if kind == "tangent" else 1
        b = 8 if case["dtype"] == "f64" else 4
        return {"bytes": 2.0 * fields * b * case["n"] ** 2,
                "flops": _apply_flops(case["n"], fields)}
    if kind == "many":
        sides = [p["grid_size"] for p, _, _ in _many(case, 0)]
        return {"bytes": sum(16.0 * n * n for n in sides),
                "flops": sum(2 * 200 * _apply_flops(n) for n in sides)}
    n = _side_of(case)
    if kind == "solve":
        return {"bytes": (32.0 if case["host"] else 16.0) * n * n,
                "flops": 2 * _iterations(case) * _apply_flops(n)}
    if kind == "nested":
        return {"bytes": 16.0 * n * n, "flops": 2 * 30 * _apply_flops(n)}
    return {"bytes": 32.0 * n * n, "flops": 300 * _apply_flops(n)}


def tolerance(case):
    """About four times what another summation order, or the distance from the
    minimiser at which a certified solve may stop, was seen to change."""
    kind = case["kind"]
    if kind in ("apply", "tangent"):
        return ({"rel": 1e-13, "max": 1e-12} if case["dtype"] == "f64"
                else {"rel": 1e-6, "max": 1e-5})
    if kind == "gradient":
        return {"rel": 1e-7, "max": 1e-5}
    if kind == "nested":
        return {"rel": 2e-6, "max": 2e-4}
    if kind == "many" and case["tol"] > 1e-7:
        return {"rel": 5e-5, "max": 5e-3}
    return {"rel": 5e-7, "max": 5e-5}


# ---- the same in 64 bits, in plain torch -------------------------------------------------


def _cells(f, F, n, near=4):
    """Integrals of f(x, y) over the unit cells at offsets 0..n-1 in each
    direction: F (f = d2F/dxdy) at the corners of the near ones, Gauss points
    in the others (where the corners would cancel)."""
    d = torch.arange(0.0, n, 1.0, dtype=torch.float64, device="cuda")
    out = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    nodes, weights = np.polynomial.legendre.leggauss(6)
    for u, wu in zip(nodes, weights):
        for v, wv in zip(nodes, weights):
            out += float(0.25 * wu * wv) * f(d[None, :] + float(0.5 * u),
                                             d[:, None] + float(0.5 * v))
    e = torch.arange(-0.5, min(n, near), 1.0, dtype=torch.float64, device="cuda")
    v = F(e[None, :], e[:, None])
    m = e.numel() - 1
    out[:m, :m] = v[1:, 1:] - v[:-1, 1:] - v[1:, :-1] + v[:-1, :-1]
    return out


def _love(n):
    return _cells(lambda x, y: 1.0 / torch.hypot(x, y), lambda x, y: _xlog(x, y) + _xlog(y, x), n)


def _xlog(a, b):
    return a * torch.asinh(b / a.abs())


def _spectrum(tab, sx=1.0, sy=1.0):
    """rfft2 of the table embedded in the doubled grid, odd (-1) or even (+1) in each offset."""
    n = tab.shape[0]
    out = torch.zeros(2 * n, 2 * n, dtype=torch.float64, device="cuda")
    out[:n, :n] = tab
    out[n + 1:, :n] = sy * tab[1:].flip(0)
    out[:, n + 1:] = sx * out[:, 1:n].flip(1)
    return torch.fft.rfft2(out)


def _padded(x, n, spec):
    return torch.fft.irfft2(torch.fft.rfft2(x, s=(2 * n, 2 * n)) * spec, s=(2 * n, 2 * n))[:n, :n]


def _operator(backend, n):
    """u = S p on (n, n) FP64 fields: unit domain, unit composite modulus."""
    if backend == "fft":
        spec = _spectrum(_love(n) / (math.pi * n))
        return lambda p: _padded(p, n, spec)
    ky = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")
    kx = torch.fft.rfftfreq(n, 1.0 / n, dtype=torch.float64, device="cuda")
    k = torch.hypot(ky[:, None], kx[None, :])
    sym = torch.where(k > 0, 1.0 / (math.pi * k.clamp_min(0.5)), torch.zeros_like(k))
    return lambda p: torch.fft.irfft2(torch.fft.rfft2(p) * sym, s=(n, n))


def _cerruti(n, nu=0.3):
    """The dense tangential block on stacked fields (unit domain and modulus)."""
    c = 1.0 / (math.pi * n * (1.0 - nu))
    ylog = _cells(lambda x, y: x * x / torch.hypot(x, y) ** 3, lambda x, y: _xlog(y, x), n)
    xy = _cells(lambda x, y: x * y / torch.hypot(x, y) ** 3, lambda x, y: -torch.hypot(x, y), n)
    xx = c * ((1.0 - nu) * _love(n) + nu * ylog)
    sxx, syy, sxy = _spectrum(xx), _spectrum(xx.T.contiguous()), _spectrum(c * nu * xy, -1.0, -1.0)
    return lambda q: torch.stack([_padded(q[0], n, sxx) + _padded(q[1], n, sxy),
                                  _padded(q[0], n, sxy) + _padded(q[1], n, syy)])


def _solution(backend, n, gap, load, most=4000, tol=1e-12):
    """Minimiser of p.Sp/2 + p.g0 over p >= 0, mean p = load: projected CG far
    past the cases' tolerances, then its displacement."""
    S = _operator(backend, n)
    g0 = gap.reshape(n, n)
    g0 = g0 - g0.mean()
    p = torch.full_like(g0, load)
    total = load * n * n
    t = torch.zeros_like(p)
    gp, G_old, delta = torch.zeros_like(p), 1.0, 0.0
    scale = float(g0.max() - g0.min())
    for it in range(most):
        on = p > 0
        v = S(p) + g0
        g = v - v[on].mean()
        gc = torch.where(on, g, torch.zeros_like(g))
        if it % 10 == 9 and float((p * (g - g.min())).sum()) <= tol * total * scale:
            break
        G = float((gc * gc).sum())
        beta = delta * max(0.0, float((gc * (g - gp)).sum())) / G_old
        t = torch.where(on, gc + beta * t, torch.zeros_like(t))
        G_old, gp = G, g
        r = S(t)
        r = r - r[on].mean()
        rt = float((r * t).sum())
        if not rt > 0.0 or G == 0.0:
            break
        tau = float((gc * t).sum()) / rt
        new = torch.where(on, (p - tau * t).clamp_min(0.0), p)
        miss = (new == 0) & (g < 0)
        new = torch.where(miss, -tau * g, new)
        delta = 0.0 if bool(((new > 0) != on).any()) else 1.0
        p = new * (total / float(new.sum()))
    return p, S


def _adjoint(S, on, w):
    """lam with S lam - mu = w on the contact set, sum lam = 0, 0 elsewhere (CG)."""
    def project(v):
        v = torch.where(on, v, torch.zeros_like(v))
        return torch.where(on, v - v[on].mean(), v)

    x = torch.zeros_like(w)
    r = project(w)
    d, rr = r, float((r * r).sum())
    stop = 1e-26 * rr
    for _ in range(4000):
        if rr <= stop:
            break
        Sd = project(S(d))
        a = rr / float((d * Sd).sum())
        x, r = x + a * d, r - a * Sd
        new = float((r * r).sum())
        d, rr = r + (new / rr) * d, new
    return x


def exact(case, seed):
    kind = case["kind"]
    if kind == "apply":
        n = case["n"]
        x = _normal(n * n, seed, _dtype(case)).double()
        return _operator(case["backend"], n)(x.reshape(n, n)).reshape(-1)
    if kind == "tangent":
        n = case["n"]
        q = _normal(2 * n * n, seed, _dtype(case)).double()
        return _cerruti(n)(q.reshape(2, n, n)).reshape(-1)
    if kind == "solve":
        n = case["n"]
        p, S = _solution(case["backend"], n, _gap(n, seed), case["load"])
        if case["host"]:
            return dict(pressure=p.cpu().numpy(), displacement=S(p).cpu().numpy(), gap=None,
                        approach=None, area=None)
        return dict(pressure=p.reshape(-1), approach=None, area=None)
    if kind == "many" and case["hi"] <= 1024:
        out = []
        for prob, hurst, s in _many(case, seed):
            n = prob["grid_size"]
            out.append(_solution(prob["backend"], n, _gap(n, s, hurst),
                                 prob["p_nominal"], 1500)[0].reshape(-1))
        return out
    if kind == "nested":
        n = _side_of(case)
        p = _solution(case["backend"], n, _gap(n, seed, rms=0.02), case["load"], 1500)[0]
        return dict(pressure=p.reshape(-1), approach=None, area=None)
    if kind == "gradient":
        n = case["n"]
        p, S = _solution(case["backend"], n, _gap(n, seed), case["load"], 8000, 1e-14)
        lam = _adjoint(S, p > 0, _normal(n * n, seed + 7919).reshape(n, n))
        return dict(pressure=p.reshape(-1), gradient=-lam.reshape(-1))
    return None  # six large solves take too long this way
