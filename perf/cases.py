"""The calls this package is measured on, from the smallest to the largest, over its public entry points.

What a program does with the package falls into six kinds, and each case is one call of one of them:

  accel      one acceleration evaluation of a system (msystem::accel), the state read back
  steps      a run of fixed RK12 steps of one system (msystem::integrate), the state read back
  ensemble   many independent point-mass systems of uneven size and duration in one call
  particles  massless test particles against a few perturbers, FP64 or mixed precision
  serve      small-body requests with adaptive steps against a B-spline ephemeris, submitted together
  fit        the least-squares B-spline fit that builds such an ephemeris from samples

Sizes come from the repository's own workloads: 33 bodies (config1), 48 and 504 bodies with every force term
(small_full, config2), ensembles of 8-300 bodies, 9 perturbers with J2-J4 on the star, the ringed planet with
its moons, 419 perturbers in the served ephemeris. Where a system carries more than point masses it is written
by `ephemeris_b200.synth` and read by the loader, as a user's files are; point-mass systems are drawn here.

Positions, velocities, frames and angular momenta are held as double-double pairs. The outputs here are their
sums: the value a program reads, the low word alone is rounding.
"""
import math
import os
import re
import tempfile

import numpy as np
import torch

from ephemeris_b200 import (Batch, Context, Models, MSystem, NPLANES, PLANES, Particles, Server, bspline_fit_batch,
                            set_log_level, synth)

DAY, AU, GM_SUN, C = synth.DAY, synth.AU, synth.GM_SUN, 299792458.0
DT = 0.05 * DAY          # the fixed step of the system and ensemble workloads
CHANNELS = 10            # position, velocity, Newtonian acceleration / c^2, potential / c^2

# ---------------------------------------------------------------------------------------------- cases


def listed():
    return [
        # one evaluation of a star, planets and moons: the smallest call a program makes (a loader, a monitor)
        {"name": "accel_33", "kind": "accel", "full": False, "bodies": 33},
        # config1: point masses and 1PN, a cadence of 20 steps between two outputs
        {"name": "steps_33_point", "kind": "steps", "full": False, "bodies": 33, "steps": 20},
        # a planetary system with every force term: time-lagged tides, harmonics, a ring
        {"name": "steps_48_full", "kind": "steps", "full": True, "bodies": 48, "steps": 10},
        # config2, the headline system, half an output cadence
        {"name": "steps_504_full", "kind": "steps", "full": True, "bodies": 504, "steps": 10},
        # config2 with twice the asteroids: more bodies than one shared-memory tile holds
        {"name": "steps_1001_full", "kind": "steps", "full": True, "bodies": 1001, "steps": 4},
        # an ensemble in plain FP64, uneven sizes and durations
        {"name": "ensemble_200", "kind": "ensemble", "members": 200, "n_min": 8, "n_max": 300, "k_min": 5, "k_max": 60,
         "mixed": False},
        # the same in mixed precision, larger, the form of the ensemble workload
        {"name": "ensemble_512_mixed", "kind": "ensemble", "members": 512, "n_min": 8, "n_max": 300, "k_min": 3,
         "k_max": 50, "mixed": True},
        # the particle workload: the star with J2-J4, eight planets, FP64
        {"name": "particles_1m", "kind": "particles", "ringed": False, "particles": 1000000, "steps": 10, "mixed": False},
        # a ragged cloud about the ringed planet, every field a particle can feel, mixed precision
        {"name": "particles_ring_mixed", "kind": "particles", "ringed": True, "particles": 60001, "steps": 12, "mixed": True},
        # one small request: its latency is what a caller waits for
        {"name": "serve_one", "kind": "serve", "requests": 1, "p_min": 5, "p_max": 5, "days": 360.0},
        # a burst of requests of mixed size and duration, which is how a server runs at capacity
        {"name": "serve_24", "kind": "serve", "requests": 24, "p_min": 1, "p_max": 4096, "days": 360.0},
        # an ephemeris fitted from a generator's samples
        {"name": "fit_419", "kind": "fit", "series": 419, "intervals": 365, "degree": 3},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["accel", "steps", "steps", "steps", "ensemble", "ensemble", "particles", "particles", "particles",
                       "serve", "serve", "fit"])
    if kind in ("accel", "steps"):
        full = rng.random() < 0.6
        c = {"kind": kind, "full": full, "bodies": _log(rng, 24, 1100) if full else _log(rng, 2, 1100)}
        if kind == "steps":
            c["steps"] = _log(rng, 1, 30 if c["bodies"] < 600 else 8)
        return c
    if kind == "ensemble":
        top = _log(rng, 24, 300)
        k = _log(rng, 4, 50)
        return {"kind": kind, "members": _log(rng, 2, 512), "n_min": rng.randint(2, 12), "n_max": top,
                "k_min": rng.randint(1, k), "k_max": k, "mixed": rng.random() < 0.5}
    if kind == "particles":
        ringed = rng.random() < 0.35
        return {"kind": kind, "ringed": ringed, "particles": _log(rng, 60, 80000 if ringed else 1000000),
                "steps": rng.randint(1, 10), "mixed": rng.random() < 0.5}
    if kind == "serve":
        p = _log(rng, 1, 4096)
        return {"kind": kind, "requests": _log(rng, 1, 24), "p_min": rng.randint(1, p), "p_max": p,
                "days": round(math.exp(rng.uniform(math.log(30.0), math.log(360.0))), 1)}
    return {"kind": "fit", "series": _log(rng, 1, 419), "intervals": _log(rng, 40, 365), "degree": rng.choice([2, 3, 3, 3, 5])}


# ---------------------------------------------------------------------------------------------- inputs


def _kepler(rng, mu, a, e, inc):
    """States of Kepler orbits of semi-major axes a (arrays [n]) about a mass mu: position, velocity [3][n]."""
    n = len(a)
    node, argp, m = (rng.uniform(0, 2 * math.pi, n) for _ in range(3))
    ecc = m.copy()
    for _ in range(12):
        ecc = ecc - (ecc - e * np.sin(ecc) - m) / (1 - e * np.cos(ecc))
    return _orbit(mu, a, e, inc, node, argp, ecc)


def _orbit(mu, a, e, inc, node, argp, ecc):
    """The state at eccentric anomaly ecc (numpy arrays or torch tensors of one shape)."""
    lib = torch if isinstance(ecc, torch.Tensor) else np
    ce, se = lib.cos(ecc), lib.sin(ecc)
    b = lib.sqrt(1 - e * e)
    rate = lib.sqrt(mu / a ** 3) / (1 - e * ce)
    x, y, vx, vy = a * (ce - e), a * b * se, -a * rate * se, a * b * rate * ce
    co, so, cw, sw, ci, si = lib.cos(node), lib.sin(node), lib.cos(argp), lib.sin(argp), lib.cos(inc), lib.sin(inc)
    p = (co * cw - so * sw * ci, so * cw + co * sw * ci, sw * si)
    q = (-co * sw - so * cw * ci, -so * sw + co * cw * ci, cw * si)
    return lib.stack([x * p[k] + y * q[k] for k in range(3)]), lib.stack([vx * p[k] + vy * q[k] for k in range(3)])


def _point_system(rng, n):
    """Star, planets and moons as point masses, the config1 recipe at any size: gm [n], radius, r, v [3][n].
    Planets keep apart by at least 3 % in semi-major axis; each moon has its own orbit radius about its planet."""
    n_planets = min(max(1, -(-n // 4)), n - 1)
    n_moons = n - 1 - n_planets
    u = (np.arange(n_planets) + rng.uniform(0.1, 0.9, n_planets)) / n_planets
    a = 0.4 * AU * np.exp(u * math.log(30.0 / 0.4))
    gp = GM_SUN * np.exp(rng.uniform(math.log(1e-9), math.log(1e-3 if n <= 64 else 1e-6), n_planets))
    e = rng.uniform(0, 0.1, n_planets) / (1 if n <= 64 else 10)
    rp, vp = _kepler(rng, GM_SUN + gp, a, e, rng.uniform(0, 3 * synth.DEG, n_planets))
    host = np.arange(n_moons) % n_planets
    order = np.arange(n_moons) // n_planets
    per = max(1, -(-n_moons // n_planets))
    gm = gp[host] * np.exp(rng.uniform(math.log(1e-8), math.log(1e-4), n_moons))
    radius_p = (3 * gp / synth.G / (4 * math.pi * 2000.0)) ** (1 / 3)
    am = radius_p[host] * (10.0 + 50.0 * (order + rng.uniform(0.1, 0.9, n_moons)) / per)
    rm, vm = _kepler(rng, gp[host] + gm, am, rng.uniform(0, 0.02, n_moons), rng.uniform(0, 3 * synth.DEG, n_moons))
    g = np.concatenate([[GM_SUN], gp, gm])
    r = np.concatenate([np.zeros((3, 1)), rp, rp[:, host] + rm], 1)
    v = np.concatenate([np.zeros((3, 1)), vp, vp[:, host] + vm], 1)
    r -= (r * g).sum(1, keepdims=True) / g.sum()
    v -= (v * g).sum(1, keepdims=True) / g.sum()
    radius = (3 * g / synth.G / (4 * math.pi * 2000.0)) ** (1 / 3)
    radius[0] = 6.96e8
    return g, radius, r, v


def _newton_1pn(g, r, v):
    """Potential, Newtonian and post-Newtonian acceleration of point masses (EIH with the accelerations on its
    right-hand side Newtonian): r, v [3][n] (numpy, or torch on any device), in their own precision."""
    lib = torch if isinstance(r, torch.Tensor) else np
    n = r.shape[1]
    d = r[:, None, :] - r[:, :, None]                # d[:, i, j] = r_j - r_i
    q = (d * d).sum(0)
    q = q + (lib.eye(n, dtype=q.dtype, device=q.device) if lib is torch else np.eye(n, dtype=q.dtype))
    inv = 1 / lib.sqrt(q)
    w = g[None, :] * inv
    if lib is torch:
        w.fill_diagonal_(0)
    else:
        np.fill_diagonal(w, 0)
    w3 = w * inv * inv
    phi = -w.sum(1)
    na = (w3 * d).sum(2)
    c2 = C * C
    beta = v / C
    b2 = (beta * beta).sum(0)
    p, a = phi / c2, na / c2
    rb = (d * beta[:, None, :]).sum(0)
    bb = (beta[:, :, None] * beta[:, None, :]).sum(0)
    da = (d * a[:, None, :]).sum(0)
    delta = 4 * p[:, None] + p[None, :] + b2[:, None] + 2 * b2[None, :] - 4 * bb + (da - 3 * (rb * inv) ** 2) / 2
    b = beta[:, None, :] - beta[:, :, None]
    ga = (3.5 * w * a[:, None, :] + w3 * delta * d + w3 * (rb - 4 * (d * b).sum(0)) * b).sum(2)
    return phi, na, ga


def _point_planes(g, radius, r, v):
    """The plane array of a point-mass system, with the acceleration of its start state filled in."""
    n = len(g)
    pl = np.zeros((NPLANES, n))
    pl[PLANES["R_HI"]:PLANES["R_HI"] + 3] = r
    pl[PLANES["V_HI"]:PLANES["V_HI"] + 3] = v
    for k in range(3):
        pl[PLANES["S_HI"] + 4 * k] = 1
    pl[PLANES["GM"]] = pl[PLANES["GM0"]] = g
    pl[PLANES["RADIUS"]] = radius
    pl[PLANES["R2"]] = radius * radius
    pl[PLANES["INERTIA"]] = 0.4
    pl[PLANES["A"]] = 0.6
    pl[PLANES["TIDE_DELAY_FACTOR"]] = 1
    for k in range(3):
        pl[PLANES["GI"] + 4 * k] = 0.4 * radius * radius
    pl[PLANES["GP_INDEX"]] = pl[PLANES["RING_INDEX"]] = -1
    on = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (g, r, v)]
    phi, na, ga = (x.cpu().numpy() for x in _newton_1pn(*on))
    pl[PLANES["PHI"]] = phi
    pl[PLANES["NACCEL"]:PLANES["NACCEL"] + 3] = na
    pl[PLANES["GACCEL"]:PLANES["GACCEL"] + 3] = ga
    pl[PLANES["BETA"]:PLANES["BETA"] + 3] = v / C
    pl[PLANES["BETA2"]] = ((v / C) ** 2).sum(0)
    return pl


def _load(system):
    """A system with more than point masses, through its files and the loader."""
    set_log_level(50)
    with tempfile.TemporaryDirectory() as d:
        ms = MSystem(0)
        if not ms.load(synth.write_system(system, d)):
            raise RuntimeError("the system did not load")
    return ms


def _full_system(n, seed):
    """Every force term: small_full up to config2's own size, from there config2 with more asteroids."""
    return synth.make_small_full(seed, n) if n < 300 else synth.make_config2(seed, n_asteroids=n - 162)


def _cloud(seed, n, mu, a_range, e_max, i_max, r0, v0):
    """Test particles on Kepler orbits, [12][n] (position hi, lo, velocity hi, lo) in pinned host memory."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    u = torch.rand(6, n, generator=gen, device="cuda", dtype=torch.float64)
    a = a_range[0] + (a_range[1] - a_range[0]) * u[0]
    e, inc, node, argp, m = e_max * u[1], i_max * u[2], 2 * math.pi * u[3], 2 * math.pi * u[4], 2 * math.pi * u[5]
    ecc = m.clone()
    for _ in range(12):
        ecc = ecc - (ecc - e * torch.sin(ecc) - m) / (1 - e * torch.cos(ecc))
    r, v = _orbit(torch.tensor(mu, dtype=torch.float64, device="cuda"), a, e, inc, node, argp, ecc)
    out = torch.zeros(12, n, dtype=torch.float64, pin_memory=True)
    out[0:3] = r.cpu() + torch.tensor(r0, dtype=torch.float64)[:, None]
    out[6:9] = v.cpu() + torch.tensor(v0, dtype=torch.float64)[:, None]
    return out


def _tracks(seed, bodies, intervals):
    """Samples [body][2 intervals + 1][channel], half a day apart, of a star and planets and small bodies on
    Kepler orbits about it, and their GM: what a generator records of an integration."""
    rng = np.random.default_rng(seed)
    gm = np.concatenate([[GM_SUN], GM_SUN * np.exp(rng.uniform(math.log(1e-9), math.log(1e-3), min(8, bodies))),
                         GM_SUN * np.exp(rng.uniform(math.log(1e-16), math.log(1e-10), max(0, bodies - 9)))])[:bodies]
    a = np.concatenate([[1.0], np.sort(np.exp(rng.uniform(math.log(0.4), math.log(30.0), 8))), rng.uniform(2.1, 3.3, max(0, bodies - 9))])[:bodies] * AU
    e, inc = rng.uniform(0, 0.1, bodies), rng.uniform(0, 10 * synth.DEG, bodies)
    node, argp, m0 = (rng.uniform(0, 2 * math.pi, bodies) for _ in range(3))
    dev = lambda x: torch.from_numpy(np.asarray(x)).cuda()[:, None]  # noqa: E731
    t = torch.arange(2 * intervals + 1, dtype=torch.float64, device="cuda")[None, :] * (DAY / 2)
    a, e, inc, node, argp, m0, g = (dev(x) for x in (a, e, inc, node, argp, m0, gm))
    m = m0 + torch.sqrt(GM_SUN / a ** 3) * t
    e, inc, node, argp, a = (x.expand_as(m) for x in (e, inc, node, argp, a))
    ecc = m.clone()
    for _ in range(12):
        ecc = ecc - (ecc - e * torch.sin(ecc) - m) / (1 - e * torch.cos(ecc))
    r, v = _orbit(torch.tensor(GM_SUN, dtype=torch.float64, device="cuda"), a, e, inc, node, argp, ecc)
    r[:, 0] = 0
    v[:, 0] = 0
    share = (g / g.sum())[None]
    r, v = r - (share * r).sum(1, keepdim=True), v - (share * v).sum(1, keepdim=True)
    out = torch.empty(bodies, t.shape[1], CHANNELS, dtype=torch.float64, device="cuda")
    out[:, :, 0:3], out[:, :, 3:6] = r.permute(1, 2, 0), v.permute(1, 2, 0)
    for lo in range(0, t.shape[1], 64):                     # Newtonian field of the bodies on one another
        x = r[:, :, lo:lo + 64]
        d = x[:, None] - x[:, :, None]
        q = (d * d).sum(0)
        q[range(bodies), range(bodies)] = math.inf
        w = g[None, :] / torch.sqrt(q)
        out[:, lo:lo + 64, 6:9] = ((w / q)[None] * d).sum(2).nan_to_num(0.0).permute(1, 2, 0) / (C * C)
        out[:, lo:lo + 64, 9] = -w.sum(1) / (C * C)
    return gm, out.cpu().numpy()


def _requests(case, seed, star):
    """Sizes, durations and the orbits' shapes are the case's own; where on its orbit a particle is, and how the
    orbit lies, comes from the seed."""
    own, rng = np.random.default_rng(case["requests"]), np.random.default_rng(seed + 1)
    for q in range(case["requests"]):
        n = int(round(math.exp(own.uniform(math.log(case["p_min"]), math.log(case["p_max"])))))
        a, e = own.uniform(0.5, 50.0, n) * AU, own.uniform(0, 0.6, n)
        r, v = _kepler(rng, GM_SUN, a, e, rng.uniform(0, 20 * synth.DEG, n))
        z = np.zeros((3, n))
        days = case["days"] * math.exp(-own.uniform(0, math.log(4.0))) if case["requests"] > 1 else case["days"]
        yield np.concatenate([r + star[0:3, None], z, v + star[3:6, None], z]), days * DAY


def _sizes(case):
    """Bodies and steps of an ensemble's members: the case's own, whatever the seed."""
    rng = np.random.default_rng(case["members"])
    n = np.round(np.exp(rng.uniform(math.log(case["n_min"]), math.log(case["n_max"]), case["members"]))).astype(int)
    return n, rng.integers(case["k_min"], case["k_max"] + 1, case["members"])


def _served_intervals(case):
    return int(math.ceil(case["days"])) + 2


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("accel", "steps"):
        if case["full"]:
            system = _load(_full_system(case["bodies"], seed))
            return {"kind": kind, "system": system, "steps": case.get("steps")}
        ctx = Context(0)
        ctx.upload(_point_planes(*_point_system(np.random.default_rng(seed), case["bodies"])))
        return {"kind": kind, "system": ctx, "steps": case.get("steps"), "t": (0.0, 0.0)}
    if kind == "ensemble":
        n, k = _sizes(case)
        rng = np.random.default_rng(seed)
        b = Batch(0)
        b.set_precision(case["mixed"])
        b.upload([_point_planes(*_point_system(rng, int(m))) for m in n])
        return {"kind": kind, "batch": b, "steps": k, "t": None}
    if kind == "particles":
        sysm = synth.make_ringed_subsystem(seed) if case["ringed"] else synth.make_config5(seed, 1)[0]
        ms = _load(sysm)
        host = sysm.bodies[0]
        if case["ringed"]:
            x = _cloud(seed, case["particles"], host.GM, (2.6 * host.R_km * 1e3, 12 * host.R_km * 1e3), 0.1, 30 * synth.DEG, host.r, host.v)
        else:
            x = _cloud(seed, case["particles"], GM_SUN, (1.5 * AU, 50 * AU), 0.3, 20 * synth.DEG, host.r, host.v)
        p = Particles(0)
        p.set_precision(case["mixed"])
        p.upload(ms.planes(), ms.models(), x.numpy())
        pert = torch.empty(NPLANES, ms.size(), dtype=torch.float64, pin_memory=True)
        return {"kind": kind, "set": p, "dt": ms.delta_t, "steps": case["steps"], "t": (0.0, 0.0), "pert": pert, "part": x}
    n = case["intervals"] if kind == "fit" else _served_intervals(case)
    gm, samples = _tracks(seed, case["series"] if kind == "fit" else 419, n)
    if kind == "fit":
        return {"kind": kind, "samples": samples, "n": n, "degree": case["degree"]}
    return {"kind": kind, "server": Server(bspline_fit_batch(samples, n, 3), gm, DAY), "requests": list(_requests(case, seed, samples[0, 0]))}


# ---------------------------------------------------------------------------------------------- one pass


def _state(pl):
    """The fields of a plane array, double-double pairs as their sums."""
    f = lambda name, w: pl[PLANES[name]:PLANES[name] + w]  # noqa: E731
    out = {k.lower(): f(k + "_HI", w) + f(k + "_LO", w) for k, w in (("R", 3), ("V", 3), ("GL", 3), ("S", 9))}
    for k, w in (("W", 3), ("GM", 1), ("EXJ2", 1), ("PHI", 1), ("BETA", 3), ("BETA2", 1), ("NACCEL", 3), ("DACCEL", 3),
                 ("GACCEL", 3), ("DTORQUE", 3), ("GI", 9), ("C_POTENTIAL", 9), ("MIN_DISTANCE", 1), ("MAX_INFLUENCE", 1)):
        out[k.lower()] = f(k, w)
    return out


def run(state):
    kind = state["kind"]
    if kind in ("accel", "steps"):
        s = state["system"]
        if isinstance(s, MSystem):
            s.accel(1) if kind == "accel" else s.integrate(DT, state["steps"], 1)
            return _state(s.planes())
        if kind == "accel":
            s.accel()
        else:
            state["t"] = s.integrate(DT, state["steps"], state["t"])
        return _state(s.download())
    if kind == "ensemble":
        b = state["batch"]
        state["t"] = b.integrate(DT, state["steps"], state["t"])
        return _state(np.concatenate(b.download(), axis=1))
    if kind == "particles":
        p = state["set"]
        state["t"] = p.integrate(state["dt"], state["steps"], state["t"])
        x = state["part"]
        p.download(state["pert"].numpy(), x.numpy())
        return {"perturbers": _state(state["pert"]), "r": x[0:3] + x[3:6], "v": x[6:9] + x[9:12]}
    if kind == "fit":
        return bspline_fit_batch(state["samples"], state["n"], state["degree"])
    srv = state["server"]
    ids = [srv.submit(x, 0.0, t, tol=1e-13, h0=DAY) for x, t in state["requests"]]
    done = [srv.result(i)[0] for i in ids]
    return [np.concatenate([x[0:3] + x[3:6], x[6:9] + x[9:12]]) for x in done]


# ---------------------------------------------------------------------------------------------- work


def work(case):
    """Bytes: the state in and out once. Operations: the pair and field terms of every stage evaluation and the
    stage combination, counted as the benchmark counts them (Newtonian 20, 1PN 80, deformation 90, spin 80,
    lagged tide 120, harmonics 250 / 80 zonal, ring disk 60 per pair; 3900 per body and step)."""
    kind = case["kind"]
    if kind in ("accel", "steps"):
        n, steps = case["bodies"], case.get("steps", 0)
        pairs = n * (n - 1)
        stage = 100 * pairs
        if case["full"]:
            tidal = 86 if n >= 300 else 9 + max(max(n - 9, 8) * 77 // 495, 6)
            heavy = min(n, tidal + (21 if n >= 300 else 1))
            stage += 180 * (pairs - (n - heavy) * (n - heavy - 1)) + 120 * tidal * (n - 1) + 9 * 250 * n + 2 * 60 * n
        return {"bytes": 2 * 8 * NPLANES * n, "flops": stage if kind == "accel" else steps * (25 * stage + 3900 * n)}
    if kind == "ensemble":
        lo, hi, k = math.log(case["n_min"]), math.log(case["n_max"]), (case["k_min"] + case["k_max"]) / 2
        span = max(hi - lo, 1e-9)                           # means of n and n^2 over a log-uniform draw
        n1, n2 = (math.exp(hi) - math.exp(lo)) / span, (math.exp(2 * hi) - math.exp(2 * lo)) / (2 * span)
        m = case["members"]
        return {"bytes": 2 * 8 * NPLANES * m * n1, "flops": m * k * (25 * 100 * (n2 - n1) + 3900 * n1)}
    if kind == "particles":
        stage = 5 * (100 + 85) + 250 + 2 * 60 if case["ringed"] else 9 * 100 + 80
        n = case["particles"]
        return {"bytes": 2 * 8 * 12 * n, "flops": n * case["steps"] * (25 * stage + 3900)}
    if kind == "serve":
        lo, hi = math.log(case["p_min"]), math.log(case["p_max"])
        n = case["requests"] * (case["p_max"] if hi == lo else (case["p_max"] - case["p_min"]) / (hi - lo))
        attempts = case["days"] * (0.54 if case["requests"] > 1 else 1.0) / 20.0
        return {"bytes": 2 * 8 * 12 * n + 8 * CHANNELS * 419 * (_served_intervals(case) + 3),
                "flops": n * attempts * 3 * (25 * 419 * 100 + 3900)}
    n, d, ch = case["intervals"], case["degree"], case["series"] * CHANNELS
    return {"bytes": 8 * ch * (3 * n + d + 1), "flops": ch * (20 * (2 * n + 1) * (d + 1) + 40 * d * (n + d))}


# ---------------------------------------------------------------------------------------------- in 64 bits


def _rk12():
    """Rows 1..25 of the Feagin table (row 25 the weights) and the nodes, in extended precision."""
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "include", "eph_rk12_table.h")
    with open(path) as f:
        bits = np.array([int(x, 16) for x in re.findall(r"0x([0-9a-f]{16})ull", f.read())], dtype=np.uint64)
    c = bits.view(np.float64).astype(np.longdouble).reshape(-1, 2).sum(1)
    rows = [c[k * (k - 1) // 2:k * (k + 1) // 2] for k in range(1, 26)]
    return rows, [r.sum() for r in rows]


def _rk12_step(rows, dt, r0, v0, f0, accel):
    """One step of the method from (r0, v0) with f0 there; accel(k, r, v) is the acceleration at node k."""
    vs, fs = [v0], [f0]
    for k, row in enumerate(rows, 1):
        use = [j for j in range(k) if row[j] != 0]
        as_is = (lambda x: x) if isinstance(r0, np.ndarray) else float
        r = r0 + as_is(dt) * sum(as_is(row[j]) * vs[j] for j in use)
        v = v0 + as_is(dt) * sum(as_is(row[j]) * fs[j] for j in use)
        f = accel(k, r, v)
        if k < 25:
            vs.append(v)
            fs.append(f)
    return r, v, f


def _zonal(x, gm, radius, js):
    """Acceleration at x [3][n] of a body at the origin whose axis is z, from its zonal terms J_n."""
    s2 = (x * x).sum(0)
    r = s2 ** 0.5
    s = x[2] / r
    legendre = {2: ((3 * s * s - 1) / 2, 3 * s), 3: ((5 * s ** 3 - 3 * s) / 2, (15 * s * s - 3) / 2),
                4: ((35 * s ** 4 - 30 * s * s + 3) / 8, (35 * s ** 3 - 15 * s) / 2)}
    out = 0 * x
    for n, j in js.items():
        p, dp = legendre[n]
        w = -gm * j * (radius / r) ** n / s2
        out[:] += w * (-(n + 1) * p - s * dp) * (x / r)
        out[2] += w * dp
    return out


def _exact_point(g, r, v, steps):
    """Point masses with 1PN in extended precision over `steps` steps (None: one evaluation)."""
    g, r, v = (np.asarray(x, np.longdouble) for x in (g, r, v))
    phi, na, ga = _newton_1pn(g, r, v)
    if steps:
        rows, _ = _rk12()
        for _ in range(steps):
            r, v, f = _rk12_step(rows, np.longdouble(DT), r, v, na + ga, lambda k, x, y: sum(_newton_1pn(g, x, y)[1:]))
            phi, na, ga = _newton_1pn(g, r, v)
    as_doubles = lambda x: np.asarray(x, np.float64)  # noqa: E731
    return {"r": as_doubles(r), "v": as_doubles(v), "phi": as_doubles(phi)[None], "naccel": as_doubles(na),
            "gaccel": as_doubles(ga), "beta": as_doubles(v / C)}


def _exact_particles(case, seed):
    """Particles against the star (J2-J4 about its fixed axis) and the planets; the perturbers in extended
    precision, the particles in 64 bits."""
    sysm = synth.make_config5(seed, 1)[0]
    star = sysm.bodies[0]
    js = {2: star.j2, **{n: c for n, _, c, _ in sysm.geopotentials["S0"][2]}}
    g = np.array([b.GM for b in sysm.bodies], np.longdouble)
    rad = np.longdouble(star.R_km) * 1000
    rows, nodes = _rk12()
    dt = sysm.delta_t

    def field(r, v):
        phi, na, ga = _newton_1pn(g, r, v)
        pull = np.zeros_like(r)
        pull[:, 1:] = _zonal(r[:, 1:] - r[:, :1], g[0], rad, js)
        pull[:, 0] = -(g[1:] / g[0] * pull[:, 1:]).sum(1)
        return phi / (C * C), na, na + ga + pull

    def particle(rp, vp, phi, na, x, y):
        at = lambda q: torch.tensor(np.asarray(q, np.float64), device=x.device)  # noqa: E731
        beta = y / C
        b2 = (beta * beta).sum(0)
        total, newton, pot, terms = torch.zeros_like(x), torch.zeros_like(x), 0 * b2, []
        for j in range(len(g)):
            d = at(rp[:, j])[:, None] - x
            inv = (d * d).sum(0) ** -0.5
            w = float(g[j]) * inv
            newton += w * inv * inv * d
            pot -= w
            terms.append((d, inv, w))
        for j, (d, inv, w) in enumerate(terms):
            w3 = w * inv * inv
            bj, aj = at(vp[:, j] / C)[:, None], at(na[:, j] / (C * C))[:, None]
            rb = (d * bj).sum(0)
            delta = 4 * pot / (C * C) + float(phi[j]) + b2 + 2 * (bj * bj).sum(0) - 4 * (beta * bj).sum(0) + \
                ((d * aj).sum(0) - 3 * (rb * inv) ** 2) / 2
            b = bj - beta
            total += 3.5 * w * aj + w3 * delta * d + w3 * (rb - 4 * (d * b).sum(0)) * b
        return newton + (total + _zonal(-terms[0][0], float(g[0]), float(rad), js))

    r = np.array([b.r for b in sysm.bodies], np.longdouble).T
    v = np.array([b.v for b in sysm.bodies], np.longdouble).T
    x0 = _cloud(seed, case["particles"], GM_SUN, (1.5 * AU, 50 * AU), 0.3, 20 * synth.DEG, star.r, star.v).cuda()
    x, y = x0[0:3], x0[6:9]
    phi, na, f = field(r, v)
    a = particle(r, v, phi, na, x, y)
    for _ in range(case["steps"]):
        seen = []

        def perturbers(k, rk, vk):
            p, n, fk = field(rk, vk)
            seen.append((rk, vk, p, n))
            return fk

        r, v, f = _rk12_step(rows, np.longdouble(dt), r, v, f, perturbers)
        x, y, a = _rk12_step(rows, dt, x, y, a, lambda k, xk, yk: particle(*seen[k - 1], xk, yk))
    return {"r": x.cpu(), "v": y.cpu()}


def _exact_request(case, seed):
    """One request with steps of a fifth of the shortest orbit's radian, far below the tolerance of the call."""
    n = _served_intervals(case)
    gm, samples = _tracks(seed, 419, n)
    coef = _exact_fit(samples, n, 3)
    x, end = next(_requests(case, seed, samples[0, 0]))
    rows, nodes = _rk12()

    def field(t):
        i = min(max(int(math.floor(t / DAY)), 0), n - 1)
        u = t / DAY - i
        b = np.array([(1 - u) ** 3, 3 * u ** 3 - 6 * u * u + 4, -3 * u ** 3 + 3 * u * u + 3 * u + 1, u ** 3]) / 6
        return np.tensordot(coef[:, i:i + 4], b, ((1,), (0,)))

    def accel(t, r, v):
        e = field(t)
        d = e[:, 0:3].T[:, None, :] - r[:, :, None]
        inv = (d * d).sum(0) ** -0.5
        w = gm[None, :] * inv
        w3 = w * inv * inv
        newton, pot = (w3 * d).sum(2), -w.sum(1)
        bj, aj, bi = (e[:, 3:6].T / C)[:, None, :], e[:, 6:9].T[:, None, :], (v / C)[:, :, None]
        rb = (d * bj).sum(0)
        delta = 4 * pot[:, None] / (C * C) + e[None, :, 9] + (bi * bi).sum(0) + 2 * (bj * bj).sum(0) - 4 * (bi * bj).sum(0) + \
            ((d * aj).sum(0) - 3 * (rb * inv) ** 2) / 2
        b = bj - bi
        return newton + (3.5 * w * aj + w3 * delta * d + w3 * (rb - 4 * (d * b).sum(0)) * b).sum(2)

    r, v = x[0:3] + x[3:6], x[6:9] + x[9:12]
    steps = int(math.ceil(end / (2 * DAY)))
    h = end / steps
    f = accel(0.0, r, v)
    rows = [np.asarray(q, np.float64) for q in rows]
    for s in range(steps):
        r, v, f = _rk12_step(rows, h, r, v, f, lambda k, a, b: accel(h * (s + float(nodes[k - 1])), a, b))
    return [np.concatenate([r, v])]


def _exact_fit(samples, n, degree):
    """The least-squares problem itself, by its normal equations in 64 bits with one refinement."""
    series, count, ch = samples.shape
    m = n + degree
    x = np.arange(count) * (n / (count - 1))
    b = np.zeros((count, m))
    for i in range(m):
        b[:, i] = _bspline(degree, x - i)
    y = samples.transpose(1, 0, 2).reshape(count, -1)
    bt, yt = torch.from_numpy(b).cuda(), torch.from_numpy(np.ascontiguousarray(y)).cuda()
    chol = torch.linalg.cholesky(bt.T @ bt)
    c = torch.cholesky_solve(bt.T @ yt, chol)
    for _ in range(2):
        c = c + torch.cholesky_solve(bt.T @ (yt - bt @ c), chol)
    return c.cpu().numpy().reshape(m, series, ch).transpose(1, 0, 2)


def _bspline(d, x):
    """Uniform B-spline of degree d on [-d, 1), the last knot interval's right end included (x = 1 reads 0)."""
    if d == 0:
        return ((x >= 0) & (x < 1)).astype(np.float64)
    return ((x + d) * _bspline(d - 1, x + 1) + (1 - x) * _bspline(d - 1, x)) / d


def exact(case, seed):
    """None where the force model has no plain form outside the package (tides with their spin iteration,
    tesseral harmonics, rings) or where it would take too long (adaptive requests by the dozen, many members)."""
    kind = case["kind"]
    empty = {k: None for k in ("r", "v", "gl", "s", "w", "gm", "exj2", "phi", "beta", "beta2", "naccel", "daccel", "gaccel",
                               "dtorque", "gi", "c_potential", "min_distance", "max_influence")}
    if kind in ("accel", "steps") and not case["full"]:
        n, steps = case["bodies"], case.get("steps")
        if (steps or 1) * n * n > 1500000:
            return None
        g, _, r, v = _point_system(np.random.default_rng(seed), n)
        return {**empty, **_exact_point(g, r, v, steps)}
    if kind == "ensemble":
        n, k = _sizes(case)
        rng = np.random.default_rng(seed)
        if sum(int(a) * int(b) ** 2 for a, b in zip(k, n)) > 1500000:
            return None
        every = []
        for m, s in zip(n, k):
            g, _, r, v = _point_system(rng, int(m))
            every.append(_exact_point(g, r, v, int(s)))
        return {**empty, **{q: np.concatenate([e[q] for e in every], axis=1) for q in every[0]}}
    if kind == "particles" and not case["ringed"]:
        return {"perturbers": empty, **_exact_particles(case, seed)}
    if kind == "serve" and case["requests"] == 1 and case["p_max"] <= 16:
        return _exact_request(case, seed)
    if kind == "fit":
        n, d = case["intervals"], case["degree"]
        return _exact_fit(_tracks(seed, case["series"], n)[1], n, d)
    return None
