"""The ensemble kernel at the sizes where its split of the work changes: units that fill a CTA's threads or just do not,
odd remainders, systems on one CTA and shared by clusters of 2 to 16, systems whose stage store leaves shared
memory, and the largest ones. Tolerances as in tests/test_gpu_batch.py; the single-system kernel is the reference
for the large sizes (its own parity with the oracle is tested elsewhere)."""
import os

import numpy as np
import pytest

from tests.parity import accel_error, position_error, rel_err

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 7, 31, 32, 33, 47, 63, 95, 96, 97, 127, 129, 191, 257, 400, 511, 738, 739, 768]


def _system(n, seed=11):
    from ephemeris_b200 import Context, PLANES, synth
    import ephemeris_b200 as eph
    sysm = synth.make_ensemble_member(seed * 1000 + n, max(n, 2))
    bodies = sysm.bodies[:n]
    pl = np.zeros((eph.NPLANES, n))
    for i, b in enumerate(bodies):
        pl[PLANES["R_HI"]:PLANES["R_HI"] + 3, i] = b.r
        pl[PLANES["V_HI"]:PLANES["V_HI"] + 3, i] = b.v
        pl[PLANES["GM"], i] = pl[PLANES["GM0"], i] = b.GM
        pl[PLANES["RADIUS"], i] = b.R_km * 1e3
    for k in range(3):
        pl[PLANES["S_HI"] + 4 * k] = 1
    pl[PLANES["R2"]] = pl[PLANES["RADIUS"]] ** 2
    pl[PLANES["A"]] = 0.6
    pl[PLANES["TIDE_DELAY_FACTOR"]] = 1
    pl[PLANES["GP_INDEX"]] = pl[PLANES["RING_INDEX"]] = -1
    c = Context(0)
    c.upload(pl)
    c.accel()
    out = c.download()
    c.close()
    return out


def _run(pl, steps, coop_min, mixed=False, extra=0):
    from ephemeris_b200 import Batch
    b = Batch(0)
    b.set_precision(mixed)
    b.set_coop_min(coop_min)
    b.upload([pl] * (1 + extra))
    assert b.info()[0] == 1 + extra
    b.integrate(600.0, steps)
    out = b.download()
    b.close()
    return out


@pytest.mark.parametrize("n", SIZES)
def test_sizes_against_the_single_system_path(n):
    from ephemeris_b200 import Context
    pl = _system(n)
    c = Context(0)
    c.upload(pl)
    c.integrate(600.0, 3)
    ref = c.download()
    c.close()
    out = _run(pl, 3, 0)[0]
    assert np.isfinite(out[0:12]).all()
    if n > 1:
        assert position_error(out, ref) <= 1e-12
        assert accel_error(out, ref) <= 1e-14
    for p in (100, 101):
        assert rel_err(out[p], ref[p]) <= 1e-15 or (n == 1 and np.array_equal(out[p], ref[p]))


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [33, 64, 97, 300, 768])
def test_sharing_a_system_changes_no_result(n, mixed):
    """One system alone (as many CTAs as help), never shared beyond what its memory needs, and among enough copies
    that every one runs on the fewest CTAs: bit-identical states."""
    pl = _system(n)
    alone = _run(pl, 2, 0, mixed)[0]
    assert np.array_equal(alone, _run(pl, 2, 1 << 30, mixed)[0])
    assert all(np.array_equal(alone, o) for o in _run(pl, 2, 0, mixed, extra=150))


def test_separations_over_the_whole_range():
    """phi = -GM / r of two bodies 1e-3 m to 1e17 m apart: the separation is exact, r^2, 1/r, the product with GM and
    the scalings by 1/c^2 and c^2 round once each, so the relative error is at most 6e-16."""
    import ephemeris_b200 as eph
    from ephemeris_b200 import Batch, PLANES
    rng = np.random.default_rng(5)
    d = 10.0 ** rng.uniform(-3, 17, 400)
    pls = []
    for x in d:
        pl = np.zeros((eph.NPLANES, 2))
        pl[0, 1] = x
        for k in range(3):
            pl[PLANES["S_HI"] + 4 * k] = 1
        pl[PLANES["GM"]] = pl[PLANES["GM0"]] = 1.0
        pl[PLANES["GP_INDEX"]] = pl[PLANES["RING_INDEX"]] = -1
        pls.append(pl)
    b = Batch(0)
    b.upload(pls)
    b.integrate(1e-30, 1)
    phi = np.array([o[PLANES["PHI"]] for o in b.download()])
    b.close()
    want = -1 / d.astype(np.longdouble)[:, None]
    assert float(np.max(np.abs(phi / want - 1))) <= 6e-16


@pytest.mark.parametrize("bad", ["nan", "coincident", "far"])
def test_degenerate_bodies_as_in_the_single_system_path(bad):
    """A NaN coordinate, two bodies in one place (no softening) and a body at 1e200 m: the same fields are finite, NaN
    or infinite as in the single-system kernel."""
    from ephemeris_b200 import Context
    pl = _system(40)
    if bad == "nan":
        pl[1, 17] = np.nan
    elif bad == "coincident":
        pl[0:12, 17] = pl[0:12, 18]
        pl[54, [17, 18]] = 0
        pl[67:79, 17] = pl[67:79, 18]
    else:
        pl[0, 17] = 1e200
    c = Context(0)
    c.upload(pl)
    c.integrate(600.0, 2)
    ref = c.download()
    c.close()
    for coop in (0, 1 << 30):
        out = _run(pl, 2, coop)[0]
        for p in list(range(3)) + list(range(6, 9)) + [65, 66] + list(range(67, 70)) + list(range(76, 79)) + [100, 101]:
            assert np.array_equal(np.isnan(out[p]), np.isnan(ref[p])), (bad, p)
            assert np.array_equal(np.isinf(out[p]), np.isinf(ref[p])), (bad, p)
