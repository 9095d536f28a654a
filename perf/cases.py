"""Timed cases: what a design program has this framework do, through its public entry points.

One step of a periodic topology optimization is: filter and project the design (``PaperOuter`` or
``ResidentOuter``), hand the density to the operator and build its diagonal scaling, solve the macro
strain loads to a certified residual, form the element energies and the homogenized tensor, and
update the design by the optimality criteria. The cases are those calls on their own, certified
homogenizations of one design, and a batch of designs of uneven grids.

Grids follow the repository's tests, benchmark and serving range: even 5-smooth edges from 8 to 108
for everything that holds a solver context, any edge for the filters. Designs are thresholded
periodic Gaussian noise with SIMP stiffness, as the benchmark's. Element weak-material ratios are the
study's 1e-4, 1e-6 and 1e-9, each with the exponents that certify there.

A solve to the default relative residual of 1e-8 fixes the homogenized tensor to far more digits than
the displacements (its error is quadratic in theirs), and what the displacements hold beyond that
residual depends on the order of summation, as the iteration counts do. Those solves therefore return
the tensor, which is what a homogenization is called for; the solves to a tight residual, as a
sensitivity check runs them, return the displacements and the element energies too.
"""
import math
import random

import numpy as np
import torch

import __graft_entry__

pgj = __graft_entry__.load_package()

GRIDS = (8, 10, 12, 16, 18, 20, 24, 30, 32, 36, 40, 48, 50, 54, 60, 64, 72, 80, 90, 96, 100, 108)
MEDIUM = pgj.PAPER_MEDIUM
F64 = torch.float64


def listed():
    return [
        # a new design of the smallest grid of the design driver enters the solver: density copy,
        # diagonal scaling, right-hand sides (launch latency)
        dict(name="setup_n16", kind="setup", n=16, loads=6, precision="fp64", alpha=0.5, emin=1e-4),
        # the operator surface on its own at the benchmark grid: K(a) u and M_alpha^-1 r, six loads
        dict(name="apply_n64", kind="apply", n=64, loads=6, precision="fp64", emin=1e-6),
        dict(name="precondition_n64", kind="precondition", n=64, loads=6, alpha=0.5, emin=1e-6),
        # element energies of six loads and the homogenized tensor, a grid off the powers of two
        dict(name="responses_n54", kind="responses", n=54, loads=6, emin=1e-6),
        # one design update of either study at its usual grid: filter, projection, OC bisection
        dict(name="paper_update_n64", kind="paper", n=64, rmin=3.0, volume=0.3, emin=1e-9),
        dict(name="study1_update_n32", kind="study1", n=32, beta=4.0, volume=0.3),
        # a sensitivity check: small grid, tight residual, displacements and energies read back
        dict(name="sensitivity_n16", kind="sensitivity", n=16, loads=6, precision="fp64", alpha=0.5, emin=1e-3),
        # certified homogenizations of one design: the FP64 drop-in at the studies' two grids, the
        # mixed-precision solver at the benchmark grid and at the largest grid of the serving range
        dict(name="solve_fp64_n32", kind="solve", n=32, loads=6, precision="fp64", alpha=0.5, emin=1e-4),
        dict(name="solve_fp64_n64", kind="solve", n=64, loads=6, precision="fp64", alpha=0.5625, emin=1e-4),
        dict(name="solve_mixed_n64", kind="solve", n=64, loads=6, precision="mixed", alpha=0.5, emin=1e-6),
        dict(name="solve_mixed_n96", kind="solve", n=96, loads=6, precision="mixed", alpha=0.5625, emin=1e-4),
        # independent designs of uneven grids in flight together, densities on the host
        dict(name="batch_mixed_uneven", kind="batch", grids="24,32,48,64,24,32,48,64", precision="mixed",
             alpha=0.5, emin=1e-4),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _grid(rng, lo, hi):
    """A grid edge of the set, spread over the logarithm of the range."""
    at = _log_uniform(rng, lo, hi)
    return min((g for g in GRIDS if lo <= g <= hi), key=lambda g: abs(math.log(g / at)))


def _contrast(rng, choices=(1e-4, 1e-6, 1e-9)):
    """(emin, alpha): the exponent lies around the one calibrated for the weak-material ratio."""
    emin = rng.choice(choices)
    lo, hi = {1e-3: (0.3, 0.7), 1e-4: (0.45, 0.7), 1e-6: (0.5, 0.75), 1e-9: (0.78, 0.85)}[emin]
    return emin, round(rng.uniform(lo, hi), 4)


def draw(rng):
    kind = rng.choice(("setup", "apply", "precondition", "responses", "paper", "study1", "sensitivity",
                       "solve", "solve", "solve", "solve", "batch"))
    precision = rng.choice(("fp64", "mixed"))
    loads = rng.choice((1, 2, 3, 6, 6))
    if kind == "setup":
        emin, alpha = _contrast(rng)
        return dict(kind=kind, n=_grid(rng, 8, 108), loads=loads, precision=precision, alpha=alpha, emin=emin)
    if kind == "apply":
        return dict(kind=kind, n=_grid(rng, 8, 108), loads=loads, precision=precision, emin=_contrast(rng)[0])
    if kind == "precondition":
        emin, alpha = _contrast(rng)
        return dict(kind=kind, n=_grid(rng, 8, 108), loads=loads, alpha=alpha, emin=emin)
    if kind == "responses":
        return dict(kind=kind, n=_grid(rng, 8, 108), loads=6, emin=_contrast(rng)[0])
    if kind == "paper":
        return dict(kind=kind, n=int(round(_log_uniform(rng, 9, 97))), rmin=round(rng.uniform(1.2, 3.5), 3),
                    volume=round(rng.uniform(0.2, 0.5), 4), emin=_contrast(rng)[0])
    if kind == "study1":
        return dict(kind=kind, n=int(round(_log_uniform(rng, 9, 97))), beta=rng.choice((1.0, 2.0, 4.0, 8.0)),
                    volume=round(rng.uniform(0.25, 0.4), 4))
    if kind == "sensitivity":
        emin, alpha = _contrast(rng, (1e-3, 1e-4))
        return dict(kind=kind, n=_grid(rng, 8, 40), loads=6, precision=precision, alpha=alpha, emin=emin)
    if kind == "solve":
        n = _grid(rng, 10, 108)
        emin, alpha = _contrast(rng, (1e-4,) if n > 64 else (1e-4, 1e-6) if n > 32 else (1e-4, 1e-6, 1e-9))
        if n > 80:
            precision = "mixed"
        return dict(kind=kind, n=n, loads=6, precision=precision, alpha=alpha, emin=emin)
    grids = [_grid(rng, 12, 64) for _ in range(rng.randint(3, 8))]
    emin, alpha = _contrast(rng, (1e-4,))
    return dict(kind="batch", grids=",".join(map(str, grids)), precision=precision, alpha=alpha, emin=emin)


# ------------------------------------------------------------------------------------------- inputs
def _generator(seed, *more):
    g = torch.Generator(device="cuda")
    g.manual_seed(random.Random(repr((int(seed),) + more)).getrandbits(48))
    return g


def _density(n, seed, vf=0.35, tag=0):
    """Physical density in (0, 1): periodic Gaussian noise of n / 16 cells behind a smooth threshold."""
    noise = torch.randn((n, n, n), generator=_generator(seed, n, tag), device="cuda", dtype=F64)
    k = torch.fft.fftfreq(n, device="cuda", dtype=F64) * (2 * math.pi)
    g = torch.exp(-0.5 * (n / 16.0) ** 2 * k * k)
    f = torch.fft.ifftn(torch.fft.fftn(noise) * g[:, None, None] * g[None, :, None] * g[None, None, :]).real
    q = f.reshape(-1).kthvalue(max(1, int(round((1.0 - vf) * n ** 3)))).values
    return torch.sigmoid((f - q) / (0.1 * f.std(correction=0)))


def _design(n, seed, emin, tag=0):
    """Stiffness multiplier of a design: SIMP with exponent 3."""
    return (emin + _density(n, seed, tag=tag) ** 3 * (1.0 - emin)).contiguous()


def _fields(n, loads, seed, dtype=F64):
    """Smooth displacement-like vectors with a rough part, (loads, 3 n^3)."""
    g = _generator(seed, n, "u")
    v = torch.randn((loads, n, n, n, 3), generator=g, device="cuda", dtype=F64)
    smooth = sum(torch.roll(v, s, d) for d in (1, 2, 3) for s in (-1, 1))
    return ((smooth + 0.1 * v) / n).to(dtype).reshape(loads, -1).contiguous()


def _macros(loads):
    return np.eye(6)[6 - loads:] if loads <= 3 else np.eye(6)[:loads]


def prepare(case, seed):
    kind, n = case["kind"], case.get("n")
    s = dict(case=dict(case))
    if kind in ("paper", "study1"):
        x = _density(n, seed, vf=case["volume"])
        energy = _density(n, seed, tag=1) + 0.05
        if kind == "paper":
            s["outer"] = pgj.PaperOuter(n, case["volume"], rmin=case["rmin"], beta=4.0, eta=0.5, emin=case["emin"])
            s["energy"] = -energy  # local objective of a stiffness maximisation
        else:
            s["outer"] = pgj.ResidentOuter(n, volume=case["volume"])
            s["energy"] = energy
        s["x"] = x.clamp(0.01, 0.99).contiguous()
        return s
    if kind == "batch":
        s["batch"] = pgj.Batch(slots=2, designs=4, precision=case["precision"])
        s["requests"] = []
        for i, g in enumerate(map(int, case["grids"].split(","))):
            s["batch"].warm(g)
            a = _design(g, seed, case["emin"], tag=i).cpu().pin_memory()
            s["requests"].append(pgj.Request(a, case["alpha"], tag=i))
        return s
    op = pgj.Operator(n, case["loads"], *MEDIUM, precision=case.get("precision", "fp64"))
    s["op"], s["a"] = op, _design(n, seed, case["emin"])
    if kind in ("apply", "precondition", "responses"):
        op.set_material(s["a"])
        s["u"] = _fields(n, case["loads"], seed,
                         torch.float32 if kind == "apply" and case["precision"] == "mixed" else F64)
        if kind == "precondition":
            op.set_alpha(case["alpha"])
    elif kind in ("solve", "sensitivity"):
        s["u"] = torch.zeros((6, 3 * n ** 3), device="cuda", dtype=F64)
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "paper":
        o = s["outer"]
        o.set_initial(s["x"])
        o.evaluate()
        o.step(s["energy"])
        return dict(ph=o.ph, dp=o.dp, a=o.a, new=o.new, change=o.change, steps=o.steps)
    if kind == "study1":
        o = s["outer"]
        o.set_initial(s["x"])
        o.evaluate(case["beta"])
        o.step(s["energy"])
        return dict(ph=o.ph, dp=o.dp, a=o.a, new=o.new, change=o.change)
    if kind == "batch":
        results = s["batch"].run(s["requests"])
        return [r.C for r in sorted(results, key=lambda r: r.tag)]
    op = s["op"]
    if kind == "setup":
        op.set_material(s["a"])
        op.set_alpha(case["alpha"])
        return dict(scale=op.scale, f=op.compute_rhs(_macros(case["loads"])))
    if kind == "apply":
        return op.apply(s["u"])
    if kind == "precondition":
        return op.apply_precond(s["u"])
    if kind == "responses":
        return dict(e=op.energies(s["u"], np.eye(6)), C=op.effective_tensor(s["u"]))
    op.set_material(s["a"])
    op.set_alpha(case["alpha"])
    u = s["u"].zero_()
    if kind == "sensitivity":
        op.solve(np.eye(6), 1e-11, u)
        return dict(u=u, e=op.energies(u, np.eye(6)), C=op.effective_tensor(u))
    op.solve(np.eye(6), 1e-8, u)
    return op.effective_tensor(u)


# ---------------------------------------------------------------------------------------- accounting
def _iterations(n, emin):
    """Rough PCG iteration count of a certified solve (measured on the benchmark's designs)."""
    return {1e-3: 260, 1e-4: 330, 1e-6: 560, 1e-9: 800}[emin] * (n / 32.0) ** 0.6


def work(case):
    kind = case["kind"]
    if kind == "batch":
        grids = map(int, case["grids"].split(","))
        parts = [work(dict(kind="solve", n=g, loads=6, precision=case["precision"], emin=case["emin"])) for g in grids]
        return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))
    n = case["n"]
    N = float(n) ** 3
    L = case.get("loads", 6)
    V = 24.0 * N  # one FP64 vector
    fft = 3 * 3 * 2.5 * N * math.log2(n)  # real transforms of three components, one direction
    if kind == "setup":  # density in, scale and right-hand sides out
        return dict(bytes=8 * N + V + L * V + 8 * N, flops=L * 60 * N + 30 * N)
    if kind == "apply":
        half = 0.5 if case["precision"] == "mixed" else 1.0
        return dict(bytes=2 * L * V * half + 8 * N, flops=L * 300 * N)
    if kind == "precondition":  # r in, z out, scale
        return dict(bytes=2 * L * V + V, flops=L * (2 * fft + 60 * N))
    if kind == "responses":  # displacements read by each of the two calls, energies out
        return dict(bytes=2 * L * V + L * 8 * N + 16 * N, flops=L * 600 * N + 21 * 42 * N)
    if kind == "paper":  # fields in and out once; about 45 bisections of the cone filter
        taps = 4.19 * case["rmin"] ** 3
        return dict(bytes=8 * 8 * N, flops=47 * 2 * taps * N)
    if kind == "study1":
        return dict(bytes=8 * 8 * N, flops=47 * 3 * 4 * (2 * int(3.6 * n / 32 + 0.5) + 1) * N)
    if kind == "sensitivity":
        its = 1.4 * _iterations(n, case["emin"])
    else:
        its = _iterations(n, case["emin"])
    s = 0.5 if case["precision"] == "mixed" else 1.0
    # an iteration reads and writes x, r, p, q and the half spectrum (the direction once more for the
    # operator); grids whose vectors fit the caches need only touch memory for density and solution
    per = L * 15 * V * s if 9 * L * V * s > 126e6 else 0.0
    return dict(bytes=its * per + 2 * L * V + 8 * N, flops=its * L * (2 * fft + 400 * N))


# ------------------------------------------------------------------------------ 64-bit plain results
OFFSETS = [(b & 1, (b >> 1) & 1, (b >> 2) & 1) for b in range(8)]  # (x, y, z) of local node b


def _element(n):
    """24 x 24 Q1 stiffness of a voxel of edge 1 / n, 2 x 2 x 2 Gauss points, E = 1 multiplier."""
    lam, mu = MEDIUM
    c = np.zeros((6, 6))
    c[:3, :3] = lam
    c[range(3), range(3)] += 2 * mu
    c[range(3, 6), range(3, 6)] = mu
    ke = np.zeros((24, 24))
    for q in range(8):
        p = [0.5 + (0.5 if (q >> d) & 1 else -0.5) / math.sqrt(3.0) for d in range(3)]
        B = np.zeros((6, 24))
        for b, o in enumerate(OFFSETS):
            w = [p[d] if o[d] else 1 - p[d] for d in range(3)]
            dx, dy, dz = ((2 * o[d] - 1) * n * w[(d + 1) % 3] * w[(d + 2) % 3] for d in range(3))
            B[:, 3 * b:3 * b + 3] = [[dx, 0, 0], [0, dy, 0], [0, 0, dz], [0, dz, dy], [dz, 0, dx], [dy, dx, 0]]
        ke += B.T @ c @ B
    return torch.tensor(ke / n ** 3 / 8, device="cuda", dtype=F64)


def _gather(u, n):
    """(L, 3N) -> (L, 24, N): the element's nodal values."""
    v = u.view(-1, n, n, n, 3).permute(0, 4, 1, 2, 3)
    return torch.cat([torch.roll(v, (-z, -y, -x), (2, 3, 4)) for x, y, z in OFFSETS], 1).reshape(v.shape[0], 24, -1)


def _scatter(f, n):
    f = f.view(f.shape[0], 24, n, n, n)
    q = sum(torch.roll(f[:, 3 * b:3 * b + 3], (z, y, x), (2, 3, 4)) for b, (x, y, z) in enumerate(OFFSETS))
    return q.permute(0, 2, 3, 4, 1).reshape(f.shape[0], -1)


def _K(a, u, ke):
    n = a.shape[0]
    return _scatter(torch.matmul(ke, _gather(u, n)) * a.reshape(1, 1, -1), n)


def _affine(n, macros):
    """(L, 24, 1) nodal values of the macro strains' linear fields on an element at the origin."""
    m = torch.as_tensor(np.asarray(macros), device="cuda", dtype=F64)
    xx, yy, zz, yz, xz, xy = m.unbind(1)
    E = torch.stack([xx, xy / 2, xz / 2, xy / 2, yy, yz / 2, xz / 2, yz / 2, zz], 1).view(-1, 3, 3)
    o = torch.tensor(OFFSETS, device="cuda", dtype=F64) / n
    return torch.einsum("lcd,bd->lbc", E, o).reshape(-1, 24, 1)


def _rhs(a, macros, ke):
    n = a.shape[0]
    return -_scatter(torch.matmul(ke, _affine(n, macros)) * a.reshape(1, 1, -1), n)


def _scale(a, alpha, ke):
    n = a.shape[0]
    d = _scatter(torch.diagonal(ke).reshape(1, 24, 1) * a.reshape(1, 1, -1), n)
    log = d.log()
    return torch.exp(-0.5 * alpha * (log - log.mean()))


def _project(u):
    v = u.view(u.shape[0], -1, 3)
    return (v - v.mean(1, keepdim=True)).reshape(u.shape)


def _green(n, ke):
    """Inverse Fourier symbol of the homogeneous operator, (n, n, n/2+1, 3, 3), zero at the origin."""
    e = torch.zeros((3, n, n, n, 3), device="cuda", dtype=F64)
    for c in range(3):
        e[c, 0, 0, 0, c] = 1.0
    q = _K(torch.ones((n, n, n), device="cuda", dtype=F64), e.reshape(3, -1), ke).view(3, n, n, n, 3)
    s = torch.fft.rfftn(q, dim=(1, 2, 3)).permute(1, 2, 3, 4, 0)
    s[0, 0, 0] = torch.eye(3, device="cuda", dtype=F64)
    g = torch.linalg.inv(s)
    g[0, 0, 0] = 0
    return g


def _precondition(r, s, green, n):
    v = torch.fft.rfftn((s * _project(r)).view(-1, n, n, n, 3), dim=(1, 2, 3))
    w = torch.fft.irfftn(torch.einsum("zyxij,lzyxj->lzyxi", green, v), s=(n, n, n), dim=(1, 2, 3))
    return _project(s * w.reshape(r.shape))


def _solution(a, alpha, ke, rtol):
    """Plain preconditioned conjugate gradients, restarted once on the true residual."""
    n = a.shape[0]
    f, s, green = _rhs(a, np.eye(6), ke), _scale(a, alpha, ke), _green(n, ke)
    dot = lambda x, y: (x * y).sum(1, keepdim=True)  # noqa: E731
    target = rtol * f.norm(dim=1, keepdim=True).clamp_min(1e-300)
    u = torch.zeros_like(f)
    for _ in range(2):
        r = f - _K(a, u, ke)
        z = _precondition(r, s, green, n)
        p, rz = z, dot(r, z)
        for it in range(6000):
            q = _K(a, p, ke)
            step = rz / dot(p, q).clamp_min(1e-300)
            u, r = u + step * p, r - step * q
            if it % 20 == 19 and bool((r.norm(dim=1, keepdim=True) <= target).all()):
                break
            z = _precondition(r, s, green, n)
            new = dot(r, z)
            p, rz = z + new / rz.clamp_min(1e-300) * p, new
        u = _project(u)
    return u


def _energies(u, ke, macros):
    n = round((u.shape[1] / 3) ** (1 / 3))
    v = _gather(u, n) + _affine(n, macros)
    return (v * torch.matmul(ke, v)).sum(1) * n ** 3


def _tensor(a, u, ke):
    n = a.shape[0]
    v = _gather(u, n) + _affine(n, np.eye(6))
    return torch.einsum("ikn,jkn->ij", v, torch.matmul(ke, v) * a.reshape(1, 1, -1))


def _cone(x, rmin):
    n, r, y = x.shape[0], math.ceil(rmin) - 1, torch.zeros_like(x)
    for dz in range(-r, r + 1):
        for dy in range(-r, r + 1):
            for dx in range(-r, r + 1):
                w = rmin - math.sqrt(dx * dx + dy * dy + dz * dz)
                if w > 0 and max(abs(dx), abs(dy), abs(dz)) < n:
                    to = tuple(slice(max(0, -d), n - max(0, d)) for d in (dz, dy, dx))
                    fr = tuple(slice(max(0, d), n - max(0, -d)) for d in (dz, dy, dx))
                    y[to] += w * x[fr]
    return y


def _paper(case, x, energy):
    rmin, beta, eta, emin, move, exponent, floor = case["rmin"], 4.0, 0.5, case["emin"], 0.1, 0.3, 0.001
    hs, N = _cone(torch.ones_like(x), rmin), x.numel()
    den = math.tanh(beta * eta) + math.tanh(beta * (1 - eta))

    def physical(x):
        q = torch.tanh(beta * (_cone(x, rmin) / hs - eta))
        return (math.tanh(beta * eta) + q) / den, beta * (1 - q * q) / den

    ph, dp = physical(x)
    g = _cone(dp * (3 * (1 - emin) * ph * ph) * energy / hs, rmin)
    ratio = -(g / N) / _cone(dp / hs, rmin)
    lo, hi, steps = 0.0, 1e9, 0
    while steps < 180 and (hi - lo) / (hi + lo) > 1e-4 and hi > 1e-40:
        mid = 0.5 * (lo + hi)
        v = x * (ratio / mid).clamp_min(1e-10) ** exponent
        new = torch.maximum(torch.maximum(torch.minimum(torch.minimum(x + move, v), torch.ones_like(x)), x - move),
                            torch.full_like(x, floor))
        lo, hi = (mid, hi) if float(physical(new)[0].mean()) > case["volume"] else (lo, mid)
        steps += 1
    return dict(ph=ph, dp=dp, a=emin + (1 - emin) * ph ** 3, new=new, change=(new - x).abs().max().reshape(1),
                steps=steps)


def _study1(case, x, energy):
    n, beta, move = x.shape[0], case["beta"], 0.1
    sigma = 0.9 * n / 32
    radius = int(4 * sigma + 0.5)
    w = torch.exp(-0.5 * (torch.arange(-radius, radius + 1, device="cuda", dtype=F64) / sigma) ** 2)
    w = (w / w.sum()).tolist()

    def gauss(x):
        for axis in range(3):
            x = sum(w[k + radius] * torch.roll(x, k, axis) for k in range(-radius, radius + 1))
        return x

    def physical(x):
        q = torch.tanh(beta * (gauss(x) - 0.5))
        half = math.tanh(0.5 * beta)
        return (half + q) / (2 * half), beta * (1 - q * q) / (2 * half)

    ph, dp = physical(x)
    g, dv = gauss(dp * 3 * (1 - 1e-4) * ph * ph * energy), gauss(dp)
    ratio = g.clamp_min(1e-30) / dv.clamp_min(1e-30)
    lo, hi = 0.0, float(ratio.max()) * 1e4
    for _ in range(45):
        mid = 0.5 * (lo + hi)
        new = torch.minimum(torch.maximum(x * (ratio / max(mid, 1e-30)).sqrt(), (x - move).clamp_min(0)),
                            (x + move).clamp_max(1))
        lo, hi = (mid, hi) if float(physical(new)[0].mean()) > case["volume"] else (lo, mid)
    return dict(ph=ph, dp=dp, a=1e-4 + (1 - 1e-4) * ph ** 3, new=new, change=(new - x).abs().max().reshape(1))


def exact(case, seed):
    kind, n = case["kind"], case.get("n")
    if kind == "batch":
        grids = [int(g) for g in case["grids"].split(",")]
        if sum(g ** 3.6 for g in grids) > 6 * 64 ** 3.6:
            return None
        out = []
        for i, g in enumerate(grids):
            ke, a = _element(g), _design(g, seed, case["emin"], tag=i)
            out.append(_tensor(a, _solution(a, case["alpha"], ke, 1e-9), ke))
        return out
    if kind in ("paper", "study1"):
        x, energy = _density(n, seed, vf=case["volume"]).clamp(0.01, 0.99), _density(n, seed, tag=1) + 0.05
        return _paper(case, x, -energy) if kind == "paper" else _study1(case, x, energy)
    ke, a = _element(n), _design(n, seed, case["emin"])
    if kind == "setup":
        return dict(scale=_scale(a, case["alpha"], ke).reshape(1, -1), f=_rhs(a, _macros(case["loads"]), ke))
    if kind in ("apply", "precondition", "responses"):
        u = _fields(n, case["loads"], seed, torch.float32 if case.get("precision") == "mixed" else F64).to(F64)
        if kind == "apply":
            return torch.cat([_K(a, v[None], ke) for v in u])
        if kind == "precondition":
            return _precondition(u, _scale(a, case["alpha"], ke), _green(n, ke), n)
        e = torch.cat([_energies(u[i:i + 1], ke, np.eye(6)[i:i + 1]) for i in range(6)])
        return dict(e=e, C=_tensor(a, u, ke))
    if kind == "solve":
        return None if n > 96 else _tensor(a, _solution(a, case["alpha"], ke, 1e-9), ke)
    u = _solution(a, case["alpha"], ke, 1e-14)
    return dict(u=u, e=_energies(u, ke, np.eye(6)), C=_tensor(a, u, ke))
