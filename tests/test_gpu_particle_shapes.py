"""The particle kernel where its work split changes: one particle to just over a block, one to 32 perturbers, calls
cut into several rounds (perturbers of a round beside the particles of the one before), geopotentials that are zonal,
fit the expanded tables or exceed them, softened hosts. The reference is the single-system kernel on the perturbers plus
the particles as bodies of GM = 1e-20 m^3/s^2 (its own parity with the oracle is tested elsewhere); tolerances as in
tests/test_gpu_particles.py."""
import numpy as np
import pytest

from tests.test_gpu_particles import _check, _combined, _gpu

pytestmark = pytest.mark.gpu


def _reference(pl, md, calls):
    from ephemeris_b200 import Context
    c = Context(0)
    c.upload(pl, md)
    t = (0.0, 0.0)
    for dt, k in calls:
        t = c.integrate(dt, k, t)
    out = c.download()
    c.close()
    return out, t


def _points(n):
    from ephemeris_b200 import synth
    sysm = synth.make_config1(1001)
    sysm.bodies = sysm.bodies[:n]
    return sysm


def _cloud(sysm, n, seed, a=(1.5, 50.0)):
    from ephemeris_b200 import synth
    rng = np.random.default_rng(seed)
    star = sysm.bodies[0]
    return synth.kepler_cloud(rng, star.GM, rng.uniform(*a, n) * synth.AU, rng.uniform(0, 0.3, n),
                              rng.uniform(0, 20 * synth.DEG, n), star.r, star.v)


@pytest.mark.parametrize("n_pert,n_part,calls", [
    (1, 1, [(4320.0, 1)]), (2, 255, [(4320.0, 3)]), (9, 256, [(4320.0, 17)]), (32, 257, [(4320.0, 35)]),
    (9, 600, [(4320.0, -9), (2160.0, 16), (4320.0, 1)]),
])
def test_sizes_and_rounds(tmp_path, n_pert, n_part, calls):
    sysm = _points(n_pert)
    pl, md, _, n = _combined(tmp_path, sysm, _cloud(sysm, n_part, 7), "points")
    ref, t1 = _reference(pl, md, calls)
    out, t = _gpu(pl, md, n, calls)
    _check(out, ref, n)
    assert t == pytest.approx(t1, rel=1e-15)


@pytest.mark.parametrize("model", [(2, 0), (8, 0), (6, 4), (8, 8), (3, 3)])
@pytest.mark.parametrize("soft", [False, True])
def test_fields(tmp_path, model, soft):
    """Geopotentials of every form on the ringed planet, and with a second model on its first moon; the planet softened."""
    from ephemeris_b200 import synth
    nz, nt = model
    rng = np.random.default_rng(40)
    sysm = synth.make_ringed_subsystem(ring_ratio=0.05)
    host = sysm.bodies[0]
    terms = [(n, 0, rng.normal(0, 1e-4) / n, 0.0) for n in range(3, nz + 1)]
    terms += [(n, m, rng.normal(0, 1e-6) / n, rng.normal(0, 1e-6) / n) for n in range(3, nt + 1) for m in range(1, n + 1)]
    if terms:
        sysm.geopotentials[host.sid] = (nz, nt, terms)
    else:
        sysm.geopotentials = {}
        host.gp_factor = 0.0
    a = rng.uniform(3.0, 12.0, 130) * host.R_km * 1e3
    parts = synth.kepler_cloud(rng, host.GM, a, rng.uniform(0, 0.1, 130), rng.uniform(0, 30 * synth.DEG, 130), host.r, host.v)
    pl, md, dt, n = _combined(tmp_path, sysm, parts, "ringed")
    if soft:
        pl[54, 0] = (3.5 * host.R_km * 1e3) ** 2
        from ephemeris_b200 import Context
        c = Context(0)
        c.upload(pl, md)
        c.accel()
        pl = c.download()
        c.close()
    ref, _ = _reference(pl, md, [(dt, 10)])
    out, _ = _gpu(pl, md, n, [(dt, 10)])
    _check(out, ref, n)
