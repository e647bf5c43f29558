"""eph_accel of point-like systems: up to 300 bodies on the point-mass kernel (one cluster), which has to leave what the
step kernel leaves (reached by asking for a launch shape). Exactly equal fields and tolerances as in
tests/test_gpu_point_route.py."""
import numpy as np
import pytest

from tests.test_gpu_batch_shapes import _system
from tests.test_gpu_point_route import _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 33, 128, 257, 300, 301])
@pytest.mark.parametrize("exj2", [0.0, 1e-4])
def test_accel_leaves_what_the_step_kernel_leaves(n, exj2):
    from ephemeris_b200 import PLANES as P, Context
    pl = _system(n, seed=31)
    pl[P["EXJ2"]] = exj2                # not zero: the step kernel's harmonics see it
    pl[P["GI"]:P["GI"] + 9] = 7.0
    pl[P["MIN_DISTANCE"], 0], pl[P["MAX_INFLUENCE"], 1] = 1e3, 1e9   # maxima that are loaded go on
    out = []
    for shape in (False, True):
        c = Context(0)
        c.upload(pl)
        if shape:
            c.set_launch(0, 8)
        got = []
        c.accel()
        got.append(c.download())
        c.integrate(600.0, 1)
        c.accel()
        got.append(c.download())
        c.close()
        out.append(got)
    for a, b in zip(*out):
        _same(a, b, n)
    assert out[0][0][P["MIN_DISTANCE"], 0] == 1e3 and out[0][0][P["MAX_INFLUENCE"], 1] == 1e9
