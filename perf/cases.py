"""The workloads that this framework's speed is measured on, through its public
entry points: whole runs from host arrays (longitudinal_evolve), bunches kept
on the device (ResidentBunch), batches (Batch, sweep.run_batched) and
parameter scans (scan_parameter).

A case is a dict of plain values; prepare() makes what a program has in hand
before the call, run() is one pass through the calls, work() counts what the
pass cannot do without, and exact() is the same pass in plain float64 torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from haissinskijulia_b200 import sweep
from haissinskijulia_b200.api import (Batch, Context, Particles, ResidentBunch,
                                      create_simulation_buffers, default_context,
                                      longitudinal_evolve)
from haissinskijulia_b200.rings import benchmark_ring, reference_ring
from haissinskijulia_b200.sensitivity import (AlphaCompactionTransform, BunchLengthFoM,
                                              EmittanceFoM, EnergySpreadFoM, VoltageTransform,
                                              scan_parameter)

# ----------------------------------------------------------------------------- the cases


def listed():
    return [
        # The smallest run worth a call: a bunch of the served requests' least
        # size on the reference's rule for its bins (one per 100 particles).
        dict(name="evolve_1e4", kind="evolve", n=10_000, nbins=128, turns=100),
        # The reference's own benchmark: its ring and wake, 1e5 particles, from
        # host arrays and back.
        dict(name="evolve_1e5", kind="evolve", n=100_000, nbins=1024, turns=100),
        # The plain method on the benchmark ring, 4096 bins, on the device.
        dict(name="resident_1e5", kind="resident", n=100_000, nbins=4096, turns=100, wake=True,
             fast=False, eta=True, log_every=0),
        # A ragged count and a bin count that is no power of two (the scans take
        # n/10 bins), with the turn log and its line density.
        dict(name="resident_1e6_ragged", kind="resident", n=999_983, nbins=10_000, turns=100,
             wake=True, fast=False, eta=True, log_every=10),
        # A production bunch between the small runs and the one at scale.
        dict(name="resident_1e7", kind="resident", n=10_000_000, nbins=4096, turns=40, wake=True,
             fast=False, eta=True, log_every=0),
        # The plain method at scale: 1e8 particles, 16384 bins, the log's
        # moments and line density.
        dict(name="resident_1e8", kind="resident", n=100_000_000, nbins=16384, turns=25,
             wake=True, fast=False, eta=True, log_every=25),
        # Tracking without collective effects and with a constant slip factor.
        dict(name="resident_no_wake", kind="resident", n=20_000_001, nbins=0, turns=40,
             wake=False, fast=False, eta=False, log_every=0),
        # The opt-in single-precision excitation normals on the finest grid.
        dict(name="resident_fast", kind="resident", n=5_000_003, nbins=16384, turns=50, wake=True,
             fast=True, eta=True, log_every=0),
        # The ragged sweep: 256 bunches of 1e4 to 2e6 particles in one batch.
        dict(name="sweep_256", kind="batch", points=256, n_lo=10_000, n_hi=2_000_000, nbins=4096,
             turns=48, points_seed=2024),
        # The intensity scan: 32 bunches of 1e6 particles, 8192 bins.
        dict(name="intensity_32", kind="batch", points=32, n_lo=1_000_000, n_hi=1_000_000,
             nbins=8192, turns=64, points_seed=7),
        # Served solves: requests of mixed sizes, bins and turns admitted and
        # retired while others run.
        dict(name="served_40", kind="served", points=40, n_lo=10_000, n_hi=400_000, turns_lo=50,
             turns_hi=300, slots=16, points_seed=11),
        # A parameter scan with its derivative samples: many short runs.
        dict(name="scan_voltage", kind="scan", n=20_000, points=6, samples=8,
             transform="voltage", fom="emittance"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["evolve", "resident", "resident", "resident", "batch", "served", "scan"])
    if kind == "evolve":
        return dict(kind=kind, n=_log_int(rng, 1e4, 1e6), nbins=_log_int(rng, 64, 4096),
                    turns=rng.randint(50, 100))
    if kind == "resident":
        n = _log_int(rng, 2e4, 5e7)
        wake = rng.random() < 0.85
        return dict(kind=kind, n=n, nbins=_log_int(rng, 256, 16384) if wake else 0,
                    turns=max(10, min(100, int(1e9 / n))), wake=wake, fast=rng.random() < 0.2,
                    eta=rng.random() < 0.8, log_every=rng.choice([0, 0, 10]))
    if kind == "batch":
        lo = _log_int(rng, 1e4, 2e5)
        points = _log_int(rng, 8, 256)
        return dict(kind=kind, points=points, n_lo=lo,
                    n_hi=_log_int(rng, lo, max(lo + 1, min(2e6, 4e7 / points))),
                    nbins=_log_int(rng, 1024, 8192), turns=rng.randint(32, 64),
                    points_seed=rng.randint(1, 10**6))
    if kind == "served":
        return dict(kind=kind, points=rng.randint(16, 48), n_lo=10_000,
                    n_hi=_log_int(rng, 5e4, 4e5), turns_lo=50, turns_hi=rng.randint(100, 300),
                    slots=rng.choice([8, 16, 32]), points_seed=rng.randint(1, 10**6))
    return dict(kind=kind, n=10 * _log_int(rng, 640, 4000), points=rng.randint(3, 8),
                samples=rng.randint(2, 8), transform=rng.choice(["voltage", "alpha"]),
                fom=rng.choice(["emittance", "length", "spread"]))


def _points(case):
    """The bunches of a batch or of a served stream: one row each of particles,
    voltage, population, bins, turns, as the sweeps draw them."""
    rng = np.random.default_rng(case["points_seed"])
    out = []
    for _ in range(case["points"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        v = float(rng.uniform(3e6, 7e6))
        pop = float(math.exp(rng.uniform(math.log(1e9), math.log(1e11))))
        if case["kind"] == "served":
            nbins = int(rng.choice([2048, 4096, 8192]))
            turns = int(rng.integers(case["turns_lo"], case["turns_hi"] + 1))
        else:
            nbins, turns = case["nbins"], case["turns"]
        out.append((n, v, pop, nbins, turns))
    return out


def _scan_values(case):
    lo, hi = (4e6, 6e6) if case["transform"] == "voltage" else (2.5e-4, 5e-4)
    return [float(v) for v in np.linspace(lo, hi, case["points"])]


def work(case):
    """Bytes: the particles in and out once, or once per turn where they do not
    fit the 126 MB second-level cache (every turn needs the wake of the whole
    bunch).  Flops: about 60 per particle and turn, and per bin and turn the
    handful that a wake potential and a kick-table entry take."""
    if case["kind"] in ("evolve", "resident"):
        rows = [(case["n"], case["nbins"], case["turns"])]
    elif case["kind"] in ("batch", "served"):
        rows = [(n, nbins, turns) for n, _, _, nbins, turns in _points(case)]
    else:
        base, short = case["points"], 2 * case["samples"] * case["points"]
        rows = [(case["n"], case["n"] // 10, 100)] * base + [(case["n"], case["n"] // 10, 10)] * short
    held = 16 * sum(r[0] for r in rows) <= 126e6 or case["kind"] in ("served", "scan")
    nbytes = sum(32 * n * (1 if held else t) for n, _, t in rows)
    flops = sum(t * (60 * n + 20 * b) for n, b, t in rows)
    return {"bytes": nbytes, "flops": flops}


# ----------------------------------------------------------------------------- prepare, run

_fast_context = None


def _context(fast=False):
    global _fast_context
    if not fast:
        return default_context()
    if _fast_context is None:
        _fast_context = Context(0)
        _fast_context.set_pass_layout(23)     # the library's layout, single-precision normals
    return _fast_context


def _gaussian(n, seed, sigma_z, sigma_E):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    z = torch.randn(n, dtype=torch.float64, device="cuda", generator=g) * sigma_z
    dE = torch.randn(n, dtype=torch.float64, device="cuda", generator=g) * sigma_E
    return z, dE


def _host_gaussian(n, seed, sigma_z, sigma_E):
    rng = np.random.default_rng(seed)
    return rng.normal(0.0, sigma_z, n), rng.normal(0.0, sigma_E, n)


def _resident_ring(case):
    cfg = benchmark_ring(n_turns=case["turns"], nbins=max(case["nbins"], 1),
                         use_wakefield=case["wake"])
    cfg.params.update_eta = case["eta"]
    return cfg


def prepare(case, seed):
    kind = case["kind"]
    if kind == "evolve":
        cfg = reference_ring(n_turns=case["turns"])
        z, dE = _host_gaussian(case["n"], seed, cfg.sigma_z, cfg.sigma_E)
        return dict(kind=kind, particles=Particles(z, dE), params=cfg.params, seed=seed,
                    buffers=create_simulation_buffers(case["n"], case["nbins"],
                                                      ctx=_context()))
    if kind == "resident":
        cfg = _resident_ring(case)
        z, dE = _gaussian(case["n"], seed, cfg.sigma_z, cfg.sigma_E)
        torch.cuda.synchronize()
        b = ResidentBunch(_context(case["fast"]), z.data_ptr(), dE.data_ptr(), case["n"],
                          cfg.params, case["nbins"], wake=cfg.wake, seed=seed)
        if case["log_every"]:
            b.set_log(case["log_every"], capacity=8, density=case["wake"])
        return dict(kind=kind, bunch=b, z=z, dE=dE, turns=case["turns"], log=case["log_every"],
                    z_out=torch.empty_like(z), dE_out=torch.empty_like(dE))
    if kind == "batch":
        pts = _points(case)
        rings = [benchmark_ring(n_turns=t, nbins=b, population=pop, voltage=v)
                 for _, v, pop, b, t in pts]
        total = sum(p[0] for p in pts)
        z, dE = _gaussian(total, seed, rings[0].sigma_z, rings[0].sigma_E)
        torch.cuda.synchronize()
        first = np.concatenate([[0], np.cumsum([p[0] for p in pts])])
        bt = Batch(_context(), sum(p[0] + 4 for p in pts), len(pts), case["nbins"])
        return dict(kind=kind, batch=bt, z=z, dE=dE, z_out=torch.empty_like(z),
                    dE_out=torch.empty_like(dE), turns=case["turns"],
                    z_ptr=[z.data_ptr() + 8 * int(f) for f in first[:-1]],
                    dE_ptr=[dE.data_ptr() + 8 * int(f) for f in first[:-1]], first=first,
                    n=[p[0] for p in pts], params=[r.params for r in rings],
                    wakes=[r.wake for r in rings], nbins=[p[3] for p in pts],
                    seeds=[1000 * seed + i for i in range(len(pts))])
    if kind == "served":
        pts = [sweep.Point(n, v, pop, b, t, 1000 * seed + i)
               for i, (n, v, pop, b, t) in enumerate(_points(case))]
        return dict(kind=kind, points=pts, slots=case["slots"])
    cfg = reference_ring(n_turns=100)
    z, dE = _host_gaussian(case["n"], seed, cfg.sigma_z, cfg.sigma_E)
    return dict(kind=kind, particles=Particles(z, dE), params=cfg.params, seed=1000 * seed,
                samples=case["samples"], values=_scan_values(case),
                transform={"voltage": VoltageTransform(),
                           "alpha": AlphaCompactionTransform()}[case["transform"]],
                fom={"emittance": EmittanceFoM(), "length": BunchLengthFoM(),
                     "spread": EnergySpreadFoM()}[case["fom"]])


def run(s):
    kind = s["kind"]
    if kind == "evolve":
        sE, sz, E0 = longitudinal_evolve(s["particles"], s["params"], s["buffers"],
                                         seed=s["seed"])
        c = s["particles"].coordinates
        return dict(z=c.z, dE=c.dE, sigma_E=sE, sigma_z=sz, E0=E0)
    if kind == "resident":
        b = s["bunch"]
        b.advance(s["turns"])
        r = b.observe(s["z_out"].data_ptr(), s["dE_out"].data_ptr())
        out = dict(z=s["z_out"], dE=s["dE_out"], sigma_E=r.sigma_E, sigma_z=r.sigma_z, E0=r.E0)
        if s["log"]:
            out["log"] = b.read_log(max_records=8)
        return out
    if kind == "batch":
        bt = s["batch"]
        ids, err = bt.add_many(s["z_ptr"], s["dE_ptr"], s["n"], s["params"], s["nbins"],
                               s["seeds"], [s["turns"]] * len(s["n"]), wakes=s["wakes"])
        if err is not None:
            raise err
        bt.advance(s["turns"])
        res = []
        for i, bid in enumerate(ids):
            at = 8 * int(s["first"][i])
            res.append(bt.take_device(bid, s["z_out"].data_ptr() + at,
                                      s["dE_out"].data_ptr() + at))
        return dict(z=s["z_out"], dE=s["dE_out"], sigma_E=np.array([r.sigma_E for r in res]),
                    sigma_z=np.array([r.sigma_z for r in res]),
                    E0=np.array([r.E0 for r in res]))
    if kind == "served":
        sv = sweep.run_batched(_context(), s["points"], max_bunches=s["slots"], copy_out=True)
        return dict(z=np.concatenate([x.z for x in sv]), dE=np.concatenate([x.dE for x in sv]),
                    sigma_E=np.array([x.result.sigma_E for x in sv]),
                    sigma_z=np.array([x.result.sigma_z for x in sv]),
                    E0=np.array([x.result.E0 for x in sv]))
    _, fom, _, _, runs = scan_parameter(s["transform"], s["fom"], s["values"], s["particles"],
                                        s["params"], n_samples=s["samples"], ctx=_context(),
                                        seed=s["seed"], return_runs=True)
    # the gradients are differences of the runs' figures of merit, nearly equal ones
    return dict(fom=fom, runs=np.array([r.fom for r in runs]))


# ----------------------------------------------------------------------------- exact
#
# The turn in float64 torch from the same inputs: RF kick, excitation with the
# Philox-4x32-10 normals of (seed, particle, turn), damping, drift, histogram,
# wake potential by FFT, interpolated kick, E0 update.  Several bunches with
# the same bin count run side by side as segments of one array.

_C = 299792458.0
_LAYERS = 2048
_zig = None


def _ziggurat():
    """(X_i, D_i, f_i, r) of the 2048-layer ziggurat, solved in long double."""
    global _zig
    if _zig is not None:
        return _zig
    L = np.longdouble
    half = L(0.5)

    def mills(r):
        # the tail's area over its density: 1/(r + 1/(r + 2/(r + 3/(r + ...))))
        t = r
        for k in range(400, 0, -1):
            t = r + L(k) / t
        return L(1) / t

    def layers(r, keep=None):
        fr = np.exp(-half * r * r)
        v = r * fr + fr * mills(r)
        x, fx = r, fr
        for i in range(1, _LAYERS - 1):
            fx = fx + v / x
            if fx >= 1:
                return L(1)
            x = np.sqrt(L(-2) * np.log(fx))
            if keep is not None:
                keep[i + 1] = x
        if keep is not None:
            keep[0], keep[1] = v / fr, r
        return fx + v / x - L(1)

    lo, hi = L(4), L(4.5)
    for _ in range(70):
        mid = half * (lo + hi)
        if layers(mid) > 0:
            lo = mid
        else:
            hi = mid
    X = np.zeros(_LAYERS + 1, dtype=L)
    layers(hi, X)
    K = np.ceil(np.ldexp(X[1:] / X[:-1], 52))
    D = (L(1) + np.ldexp(K, -52)).astype(np.float64)
    f = np.exp(-half * X * X).astype(np.float64)
    dev = [torch.from_numpy(a).cuda() for a in (X[:-1].astype(np.float64), D, f)]
    _zig = (*dev, float(X[1]))
    return _zig


def _philox(pair, seed, turn, tag=0):
    """The four words of Philox-4x32-10; pair, seed and turn as int64 tensors
    or ints, tag the bits set in the counter's last word."""
    m = 0xFFFFFFFF
    c0, c1 = pair & m, pair >> 32
    c2 = torch.full_like(c0, turn & m)
    c3 = torch.full_like(c0, turn >> 32) | tag
    k0, k1 = seed & m, (seed >> 32) & m
    for _ in range(10):
        # a 32 x 32-bit product wraps in int64; its halves are masked out
        p0 = c0 * 0xD2511F53
        p1 = c2 * 0xCD9E8D57
        c0, c1, c2, c3 = (((p1 >> 32) & m) ^ c1 ^ k0, p1 & m, ((p0 >> 32) & m) ^ c3 ^ k1, p0 & m)
        k0 = (k0 + 0x9E3779B9) & m
        k1 = (k1 + 0xBB67AE85) & m
    return c0, c1, c2, c3


def _normals_of(pair, seed, turn, h, hi, lo):
    """Normals of the draws (hi, lo) of half h of the pairs."""
    X, D, f, r = _ziggurat()

    def parts(hi, lo):
        return hi >> 21, ((hi >> 20) & 1) == 1, (((hi & 0xFFFFF) << 32) | lo).double() * 2.0**-52

    i, neg, u = parts(hi, lo)
    x = u * X[i]
    at = torch.nonzero(1.0 + u >= D[i]).reshape(-1)
    if at.numel():
        xs, ns = x[at], neg[at]
        left = torch.arange(at.numel(), device=at.device)
        il, ul = i[at], u[at]
        sd = (lambda k: seed[at][k]) if torch.is_tensor(seed) else (lambda k: seed)
        pl = pair[at]
        for a in range(1, 60):
            if not left.numel():
                break
            w0, w1, w2, w3 = _philox(pl[left], sd(left), turn, (2 * a - 1 + h) << 24)
            tail = il[left] == 0
            u1 = ((((w1 & 0xFFFFF) << 32) | w0).double() + 0.5) * 2.0**-52
            u2 = ((((w3 & 0xFFFFF) << 32) | w2).double() + 0.5) * 2.0**-52
            ta, tb = -torch.log(u1) / r, -torch.log(u2)
            xw = ul[left] * X[il[left]]
            fi, fi1 = f[il[left]], f[il[left] + 1]
            y = fi + (u1 - 0.5 * 2.0**-52) * (fi1 - fi)
            ok = torch.where(tail, tb + tb > ta * ta, y < torch.exp(-0.5 * xw * xw))
            xn = torch.where(tail, r + ta, xw)
            again = ~tail & ~ok
            i2, n2, d2 = parts(w3, w2)
            xn = torch.where(again, d2 * X[i2], xn)
            ok = ok | (again & (1.0 + d2 < D[i2]))
            il[left] = torch.where(again, i2, il[left])
            ul[left] = torch.where(again, d2, ul[left])
            ns[left] = torch.where(again, n2, ns[left])
            xs[left] = xn
            left = left[~ok]
        x[at], neg[at] = xs, ns
    return torch.where(neg, -x, x)


def _pair_normals(pair, seed, turn):
    w0, w1, w2, w3 = _philox(pair, seed, turn)
    return (_normals_of(pair, seed, turn, 0, w1, w0), _normals_of(pair, seed, turn, 1, w3, w2))


def _std(v):
    """The reference's single-pass spread, about the mean's square."""
    n = v.numel()
    m = float(v.mean())
    d = v - m
    return math.sqrt(max(0.0, (float((d * d).sum()) - float(d.sum()) ** 2 / n) / (n - 1)))


def _track(z, dE, sizes, params, wakes, nbins, seeds, turns, first_turn=1, log_every=0):
    """`turns` turns of the bunches z, dE concatenates (changed in place);
    (σ_E, σ_z, E0) of each and the log records of the first."""
    dev = z.device
    ns = len(sizes)
    p0 = params[0]
    cut = np.concatenate([[0], np.cumsum(sizes)])
    spans = [slice(int(cut[k]), int(cut[k + 1])) for k in range(ns)]
    many = ns > 1
    seg = torch.repeat_interleave(torch.arange(ns, device=dev), torch.tensor(sizes, device=dev)) \
        if many else None

    def vec(vals):
        return torch.tensor(vals, dtype=torch.float64, device=dev)[seg] if many else vals[0]

    if p0.use_excitation:
        pair = torch.cat([torch.arange((n + 1) // 2, device=dev) for n in sizes])
        if many:
            half = torch.tensor([(n + 1) // 2 for n in sizes], device=dev)
            sd = torch.repeat_interleave(torch.tensor(seeds, device=dev), half)
        else:
            sd = int(seeds[0])
    sz0 = [_std(z[k]) for k in spans]
    sE0 = [_std(dE[k]) for k in spans]
    E0 = [p.E0 for p in params]
    B, wake = nbins, bool(p0.use_wakefield)
    records = []
    if wake:
        P = 1
        while P < 2 * B:
            P *= 2
        w = [max(m.half_width_sigmas * s, 0.0) for m, s in zip(wakes, sz0)]
        k2 = torch.arange(B, device=dev, dtype=torch.float64) * 2 + (1 - B)
        cent = torch.stack([k2 * (x / B) for x in w])
        Wf, lam = [], []
        for m, c in zip(wakes, cent):
            W = m.wake_factor * torch.exp(c / m.ctau) * (
                torch.cos(m.wake_sqrt * c) + m.sin_coef * torch.sin(m.wake_sqrt * c))
            Wf.append(torch.fft.rfft(torch.where(c > 0, torch.zeros_like(W), W), P))
            lam.append(torch.exp(-0.5 * (c / m.delta_std) ** 2)
                       / (math.sqrt(2 * math.pi) * m.delta_std))
        Wf, lam = torch.stack(Wf), torch.stack(lam)
        inv = [B / (2 * x) for x in w]
        w_i, inv_i = vec(w), vec(inv)
        c1 = vec([float(c[0]) for c in cent])
        cB = vec([float(c[-1]) for c in cent])
        invc = vec([(B - 1) / float(c[-1] - c[0]) if B > 1 else 0.0 for c in cent])
    for turn in range(first_turn, first_turn + turns):
        g0 = [e / p.mass for e, p in zip(E0, params)]
        b0 = [math.sqrt(1 - 1 / g ** 2) for g in g0]
        k = [p.freq_rf * 2 * math.pi / (b * _C) for p, b in zip(params, b0)]
        start = dE.clone() if p0.update_E0 else None
        phi = vec([p.phi_s for p in params])
        dE += vec([p.voltage for p in params]) * (
            torch.sin(phi - z * vec(k)) - vec([math.sin(p.phi_s) for p in params]))
        dU = [4 * 8.85e-5 * (e / 1e9) ** 3 / p.radius for e, p in zip(E0, params)]
        if p0.use_excitation:
            amp = [math.sqrt(1 - (1 - u) ** 2) * s for u, s in zip(dU, sE0)]
            r0, r1 = _pair_normals(pair, sd, turn)
            r = torch.stack([r0, r1], dim=1).reshape(-1)
            if many:
                keep = [n for n in sizes]
                at = np.concatenate([[0], np.cumsum([(n + 1) // 2 * 2 for n in sizes])])
                r = torch.cat([r[int(at[q]):int(at[q]) + n] for q, n in enumerate(keep)])
            dE += vec(amp) * r[: z.numel()]
        if p0.SR_damping:
            dE *= vec([1 - u for u in dU])
        h = [2 * math.pi * p.harmonic / (b * b * e * q)
             for p, b, e, q in zip(params, b0, E0, k)]
        if p0.update_eta:
            gam = vec(g0) + dE / vec([p.mass for p in params])
            z -= vec(h) * (vec([p.alpha_c for p in params]) - 1 / (gam * gam)) * dE
        else:
            z -= vec([q * (p.alpha_c - 1 / g ** 2) for q, p, g in zip(h, params, g0)]) * dE
        if wake:
            b = torch.floor((z + w_i) * inv_i).long().clamp_(0, B - 1)
            idx = (b + seg * B if many else b)[(z >= -w_i) & (z <= w_i)]
            cnt = torch.bincount(idx, minlength=ns * B).reshape(ns, B)
            cur = []
            for q, (p, m) in enumerate(zip(params, wakes)):
                sz = _std(z[spans[q]])
                pf = m.population if m.population > 0 else \
                    1e11 / 10.0 ** min(10, len(str(sizes[q])) - 1) * sizes[q]
                cur.append(pf / E0[q] / (2 * math.pi * p.radius) * sz
                           / ((p.alpha_c - 1 / g0[q] ** 2) * sE0[q] ** 2))
            dens = lam * cnt.double() / cnt.sum(dim=1, keepdim=True)
            pot = torch.fft.irfft(torch.fft.rfft(dens, P) * Wf, P)[:, :B]
            pot = (pot * torch.tensor(cur, dtype=torch.float64, device=dev)[:, None]).reshape(-1)
            u = (torch.minimum(torch.maximum(z, c1), cB) if many else z.clamp(c1, cB)) - c1
            u = u * invc
            fl = torch.floor(u).clamp_(0, max(B - 2, 0))
            at = fl.long() + (seg * B if many else 0)
            u -= fl
            dE -= pot[at] * (1 - u) + pot[at + 1] * u
        if p0.update_E0:
            mean = [float((dE[q] - start[q]).sum()) / n for q, n in zip(spans, sizes)]
            E0 = [e + m for e, m in zip(E0, mean)]
            dE -= vec(mean)
        if log_every and turn % log_every == 0:
            rec = [float(turn), E0[0], _std(z), _std(dE), float(z.mean()), float(dE.mean())]
            rec += [cur[0], float(cnt.sum())] + cnt[0].tolist() if wake else [0.0, 0.0]
            records.append(rec)
    return ([_std(dE[q]) for q in spans], [_std(z[q]) for q in spans], E0, records)


def exact(case, seed):
    kind = case["kind"]
    if kind == "evolve":
        cfg = reference_ring(n_turns=case["turns"])
        z, dE = (torch.from_numpy(a).cuda()
                 for a in _host_gaussian(case["n"], seed, cfg.sigma_z, cfg.sigma_E))
        sE, sz, E0, _ = _track(z, dE, [case["n"]], [cfg.params], [cfg.wake], case["nbins"],
                               [seed], case["turns"])
        return dict(z=z.cpu().numpy(), dE=dE.cpu().numpy(), sigma_E=sE[0], sigma_z=sz[0],
                    E0=E0[0])
    if kind == "resident":
        if case["fast"]:
            return None                       # single-precision normals by design
        cfg = _resident_ring(case)
        z, dE = _gaussian(case["n"], seed, cfg.sigma_z, cfg.sigma_E)
        sE, sz, E0, rec = _track(z, dE, [case["n"]], [cfg.params], [cfg.wake], case["nbins"],
                                 [seed], case["turns"], log_every=case["log_every"])
        out = dict(z=z, dE=dE, sigma_E=sE[0], sigma_z=sz[0], E0=E0[0])
        if case["log_every"]:
            out["log"] = np.array(rec[-8:])
        return out
    if kind == "batch":
        pts = _points(case)
        rings = [benchmark_ring(n_turns=t, nbins=b, population=pop, voltage=v)
                 for _, v, pop, b, t in pts]
        z, dE = _gaussian(sum(p[0] for p in pts), seed, rings[0].sigma_z, rings[0].sigma_E)
        sE, sz, E0, _ = _track(z, dE, [p[0] for p in pts], [r.params for r in rings],
                               [r.wake for r in rings], case["nbins"],
                               [1000 * seed + i for i in range(len(pts))], case["turns"])
        return dict(z=z, dE=dE, sigma_E=np.array(sE), sigma_z=np.array(sz), E0=np.array(E0))
    if kind == "served":
        zs, es, res = [], [], []
        for i, (n, v, pop, b, t) in enumerate(_points(case)):
            sd = 1000 * seed + i
            cfg = benchmark_ring(n_turns=t, nbins=b, population=pop, voltage=v)
            # particle i starts from the two normals of pair i at turn 0, under
            # the initial bunch's own stream of the seed
            tag = (sd ^ 0x6A09E667F3BCC909) & 0xFFFFFFFFFFFFFFFF
            r0, r1 = _pair_normals(torch.arange(n, device="cuda"), tag, 0)
            z, dE = cfg.sigma_z * r0, cfg.sigma_E * r1
            sE, sz, E0, _ = _track(z, dE, [n], [cfg.params], [cfg.wake], b, [sd], t)
            zs.append(z.cpu().numpy())
            es.append(dE.cpu().numpy())
            res.append((sE[0], sz[0], E0[0]))
        res = np.array(res)
        return dict(z=np.concatenate(zs), dE=np.concatenate(es), sigma_E=res[:, 0],
                    sigma_z=res[:, 1], E0=res[:, 2])
    return _exact_scan(case, seed)


def _exact_scan(case, seed):
    cfg = reference_ring(n_turns=100)
    z0, e0 = (torch.from_numpy(a).cuda()
              for a in _host_gaussian(case["n"], seed, cfg.sigma_z, cfg.sigma_E))
    field = {"voltage": "voltage", "alpha": "alpha_c"}[case["transform"]]
    n = case["n"]

    def foms(values, turns, seeds, update_E0):
        ps = [cfg.params.replace(n_turns=turns, update_E0=update_E0, **{field: v})
              for v in values]
        k = len(values)
        z, e = z0.repeat(k), e0.repeat(k)
        sE, sz, _, _ = _track(z, e, [n] * k, ps, [cfg.wake] * k, n // 10, seeds, turns)
        if case["fom"] == "length":
            return sz
        if case["fom"] == "spread":
            return sE
        out = []
        for q in range(k):
            dz = z[q * n:(q + 1) * n] - z[q * n:(q + 1) * n].mean()
            de = e[q * n:(q + 1) * n] - e[q * n:(q + 1) * n].mean()
            r = float((dz * de).sum()) / math.sqrt(float((dz * dz).sum()) * float((de * de).sum()))
            out.append(sz[q] * sE[q] * math.sqrt(1 - r * r))
        return out

    vals = _scan_values(case)
    m = case["samples"]
    base = foms(vals, 100, [1000 * seed] * len(vals), True)
    runs = []
    for v, b in zip(vals, base):
        lo, hi = v - 0.01 * v, v + 0.01 * v
        sd = [1000 * seed + 1 + q for q in range(m)]
        f = foms([hi] * m + [lo] * m, 10, sd + sd, False)
        runs += [b] + [x for q in range(m) for x in (f[q], f[m + q])]
    return dict(fom=np.array(base), runs=np.array(runs))
