"""The pair sweeps' 1/sqrt(m) through eph_deform: a body of GM = 1 and 1099 without mass, all in one place, the softening
sR2 of each a number of its own, so that its potential is -1/sqrt(sR2), with no other rounding. The binomial series drops
5 e^3/16 of the result, |e| <= 2^-19: at most 0.02 units in the last place beyond the half of the last rounding."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ulps(got, m):
    """|got - 1/sqrt(m)| in units in the last place of the result, in integers."""
    mant, ex = math.frexp(m)
    if ex % 2:
        mant, ex = 2 * mant, ex - 1
    want = math.isqrt((1 << 354) // int(mant * 2 ** 54))            # 2^150 / sqrt(mant)
    have = int(math.ldexp(got, ex // 2) * 2 ** 60) << 90
    return abs(have - want) / 2.0 ** (want.bit_length() - 53)


@pytest.mark.parametrize("lo,hi", [(-0.1, 2.1), (-60, 140), (-900, 900)])
def test_within_the_series_bound(lo, hi):
    import ephemeris_b200 as eph
    from ephemeris_b200 import Context, PLANES as P
    n = 1100
    m = np.exp2(np.random.default_rng(int(hi)).uniform(lo, hi, n))
    m[0] = 0
    pl = np.zeros((eph.NPLANES, n))
    pl[P["SR2"]] = m
    pl[P["GM0"]] = pl[P["R2"]] = pl[P["RADIUS"]] = pl[P["TIDE_DELAY_FACTOR"]] = 1
    pl[P["GM"], 0] = 1
    pl[P["A"]] = 0.6
    for k in range(3):
        pl[P["S_HI"] + 4 * k] = 1
    pl[P["GP_INDEX"]] = pl[P["RING_INDEX"]] = -1
    c = Context(0)
    c.upload(pl)
    c.deform()
    phi = c.download()[P["PHI"]]
    c.close()
    assert max(_ulps(-p, x) for p, x in zip(phi[1:], m[1:])) <= 0.52
