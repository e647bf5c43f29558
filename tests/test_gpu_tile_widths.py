"""Full-physics systems around the widths at which the step kernel stages the bodies differently: one tile up to 576, pass
A whole at twice the stride up to 1152, chunks beyond. One acceleration evaluation and one RK12 step against the oracle,
tolerances as in tests/test_gpu_paths.py."""
import os

import numpy as np
import pytest

from tests.parity import accel_error, position_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,step", [(576, False), (577, True), (1151, False), (1152, True), (1153, False), (1184, False)])
def test_tile_widths(tmp_path, oracle, n, step):
    from ephemeris_b200 import Context, Models, MSystem, synth
    from oracle.pyoracle import Models as OModels
    sysm = synth.make_config2(2002, n_asteroids=n - 162)
    ms = MSystem(0)
    assert ms.load(synth.write_system(sysm, os.path.join(str(tmp_path), "big")))
    pl, md, dt = ms.planes(), ms.models(), ms.delta_t
    ms.close()
    assert pl.shape[1] == n
    om = OModels(md.gp_nz, md.gp_nt, md.gp_coef, md.ring_ndisk, md.ring_param, md.ring_disk)
    c = Context(0)
    c.upload(pl, md)
    c.accel()
    out = c.download()
    ref = oracle.accel(pl, om)
    assert accel_error(out, ref) <= 1e-14
    assert np.allclose(out[36:39], ref[36:39], rtol=1e-13, atol=0)      # the angular-velocity fixed point
    if step:
        c.upload(pl, md)
        c.integrate(dt, 1)
        assert position_error(c.download(), oracle.integrate(pl, om, dt, 1)[0]) <= 1e-12
    c.close()


def test_nan_sticks_in_the_maxima(oracle):
    """One body without a position: the maxima of every body are NaN, those of a pair the comparisons must not pass over."""
    from ephemeris_b200 import PLANES, Context
    from oracle.pyoracle import Models
    from tests.test_gpu_batch_shapes import _system
    pl = _system(40, seed=3)
    rows = [PLANES["MIN_DISTANCE"], PLANES["MAX_INFLUENCE"]]
    for bad in (None, 33):
        p = pl.copy()
        if bad is not None:
            p[PLANES["R_HI"], bad] = np.nan
        c = Context(0)
        c.upload(p)
        c.accel()
        out = c.download()[rows]
        c.close()
        ref = oracle.accel(p, Models.empty())[rows]
        assert np.array_equal(np.isnan(out), np.isnan(ref))
        assert np.isnan(out).all() == (bad is not None)
        assert np.allclose(out, ref, rtol=1e-13, atol=0, equal_nan=True)
