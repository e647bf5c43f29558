"""Requests at the sizes where the request kernel's work split changes: one particle to more than a block, every number
of lanes per particle, perturber counts around the chunks of the spline evaluation, spline degrees with and without
a specialised form, softened perturbers, one and two sets of perturber records. The reference integrates the same
splines in numpy with fixed RK12 steps far below the request's; a request holds every step to 1e-13 of the distance from
body 0, its result after some 20 steps to 5e-11."""
import math
import os
import re

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DAY, AU, GM_SUN, C = 86400.0, 1.495978707e11, 1.32712440018e20, 299792458.0
DAYS = 24


def _tracks(m, soft):
    """Samples [m][4 DAYS + 1][10] of a star at rest and bodies on circular orbits, their GM and softening."""
    rng = np.random.default_rng(m)
    gm = np.concatenate([[GM_SUN], GM_SUN * 10 ** rng.uniform(-9, -4, m - 1)])
    a = np.concatenate([[1.0], np.linspace(0.7, 30, m)[1:]]) * AU
    ph, inc = rng.uniform(0, 2 * math.pi, m), rng.uniform(0, 0.1, m)
    t = np.arange(4 * DAYS + 1) * DAY / 4
    w = np.sqrt(GM_SUN / a ** 3)
    th = w[:, None] * t + ph[:, None]
    ci, si = np.cos(inc)[:, None], np.sin(inc)[:, None]
    r = np.stack([np.cos(th), np.sin(th) * ci, np.sin(th) * si], -1) * a[:, None, None]
    v = np.stack([-np.sin(th), np.cos(th) * ci, np.cos(th) * si], -1) * (a * w)[:, None, None]
    r[0] = 0
    v[0] = 0
    out = np.zeros((m, len(t), 10))
    out[..., 0:3], out[..., 3:6] = r, v
    for k in range(m):
        d = r - r[k]
        q = (d * d).sum(-1)
        q[k] = np.inf
        out[k, :, 6:9] = (gm[:, None, None] * d * q[..., None] ** -1.5).sum(0) / C ** 2
        out[k, :, 9] = -(gm[:, None] * q ** -0.5).sum(0) / C ** 2
    return out, gm, (np.where(np.arange(m) % 3 == 0, (0.02 * AU) ** 2, 0.0) if soft else None)


def _basis(d, x):
    if d == 0:
        return 1.0 if 0 <= x < 1 else 0.0
    return ((x + d) * _basis(d - 1, x + 1) + (1 - x) * _basis(d - 1, x)) / d


def _table():
    with open(os.path.join(os.path.dirname(__file__), "..", "include", "eph_rk12_table.h")) as f:
        bits = np.array([int(x, 16) for x in re.findall(r"0x([0-9a-f]{16})ull", f.read())], dtype=np.uint64)
    c = bits.view(np.float64).reshape(-1, 2).sum(1)
    return [c[k * (k - 1) // 2:k * (k + 1) // 2] for k in range(1, 26)]


def _reference(coefs, d, gm, sr2, x, t0, t1):
    n = coefs.shape[1] - d
    sr2 = np.zeros(len(gm)) if sr2 is None else sr2

    def accel(t, r, v):
        i = min(max(int(math.floor(t / DAY)), 0), n - 1)
        e = np.tensordot(coefs[:, i:i + d + 1], np.array([_basis(d, t / DAY - i - k) for k in range(d + 1)]), ((1,), (0,)))
        dr = e[:, 0:3].T[:, None, :] - r[:, :, None]
        inv = np.maximum((dr * dr).sum(0), sr2) ** -0.5
        w = gm * inv
        w3 = w * inv * inv
        newton, pot = (w3 * dr).sum(2), -w.sum(1)
        bj, aj, bi = (e[:, 3:6].T / C)[:, None, :], e[:, 6:9].T[:, None, :], (v / C)[:, :, None]
        rb = (dr * bj).sum(0)
        delta = 4 * pot[:, None] / C ** 2 + e[None, :, 9] + (bi * bi).sum(0) + 2 * (bj * bj).sum(0) - 4 * (bi * bj).sum(0) + \
            ((dr * aj).sum(0) - 3 * (rb * inv) ** 2) / 2
        b = bj - bi
        return newton + (3.5 * w * aj + w3 * delta * dr + w3 * (rb - 4 * (dr * b).sum(0)) * b).sum(2)

    rows = _table()
    steps = 2 * int(math.ceil(abs(t1 - t0) / DAY))
    h = (t1 - t0) / steps
    r, v = x[0:3].copy(), x[3:6].copy()
    f = accel(t0, r, v)
    for s in range(steps):
        t = t0 + s * h
        vs, fs = [v], [f]
        for row in rows:
            rk = r + h * sum(a * q for a, q in zip(row, vs) if a)
            vk = v + h * sum(a * q for a, q in zip(row, fs) if a)
            fk = accel(t + h * row.sum(), rk, vk)
            vs.append(vk)
            fs.append(fk)
        r, v, f = rk, vk, fk
    return r


@pytest.mark.parametrize("m,p,degree,soft", [
    (1, 1, 3, False), (5, 7, 3, True), (17, 8, 3, False), (18, 9, 3, False), (19, 300, 3, True), (37, 2500, 3, False),
    (6, 5000, 3, False), (7, 5000, 3, True), (12, 20000, 3, False), (31, 40001, 3, False),
    (19, 40, 1, False), (19, 40, 2, True), (13, 40, 5, False), (13, 40, 8, False), (1000, 33, 3, False), (1000, 5000, 3, True),
])
def test_requests(m, p, degree, soft):
    from ephemeris_b200 import Server, bspline_fit_batch, synth
    samples, gm, sr2 = _tracks(m, soft)
    coefs = bspline_fit_batch(samples, DAYS, degree)
    rng = np.random.default_rng(p)
    parts = synth.kepler_cloud(rng, GM_SUN, rng.uniform(2.0, 9.0, p) * AU, rng.uniform(0, 0.3, p), rng.uniform(0, 0.3, p),
                               np.zeros(3), np.zeros(3))
    srv = Server(coefs, gm, DAY, 0.0, degree, sr2)
    t0, t1 = (0.5 * DAY, (DAYS - 0.5) * DAY) if p % 2 else ((DAYS - 0.5) * DAY, 0.5 * DAY)   # both directions
    rid = srv.submit(parts, t0, t1, tol=1e-13, h0=DAY)
    lanes, per, blocks = srv.shape(rid)
    assert lanes * per <= 256 and per * blocks >= p
    out, acc, _ = srv.result(rid)
    srv.close()
    assert acc >= p and np.isfinite(out).all()
    some = np.unique(np.concatenate([np.arange(min(p, per + 1)), [p - 1], rng.integers(0, p, 12)]))[:40]
    some = np.unique(np.concatenate([some, [p - 1]]))
    want = _reference(coefs, degree, gm, sr2, parts[:, some], t0, t1)
    off = np.linalg.norm(out[0:3, some] + out[3:6, some] - want, axis=0) / np.linalg.norm(want, axis=0)
    assert off.max() <= 5e-11, off.max()
