"""Systems of point-like bodies through eph_integrate / eph_rk12: up to 300 bodies they run on the point-mass kernel
(one cluster), which has to leave what the step kernel leaves. The step kernel is reached by asking for a launch
shape. Fields that such bodies do not change come out exactly equal, the others within the parity tolerances of
tests/test_gpu_parity.py."""
import numpy as np
import pytest

from tests.parity import accel_error, position_error, rel_err
from tests.test_gpu_batch_shapes import _system

pytestmark = pytest.mark.gpu


def _go(pl, calls, step_kernel, device_copy=False):
    from ephemeris_b200 import Context
    c = Context(0)
    c.upload(pl)
    if step_kernel:
        c.set_launch(0, 8)
    if device_copy:
        c.upload_device(c.device_planes_ptr())
    t = (0.0, 0.0)
    for kind, dt, k in calls:
        if kind == "rk12":
            c.rk12(dt, k, t)
        else:
            t = c.integrate(dt, k, t)
    out = c.download()
    c.close()
    return out, t


def _same(a, b, n):
    from ephemeris_b200 import PLANES as P
    for name, w in (("GL_HI", 3), ("GL_LO", 3), ("S_HI", 9), ("S_LO", 9), ("W", 3), ("GM", 1), ("EXJ2", 1), ("DACCEL", 3),
                    ("DTORQUE", 3), ("GI", 9), ("C_POTENTIAL", 9)):
        assert np.array_equal(a[P[name]:P[name] + w], b[P[name]:P[name] + w]), name
    if n > 1:
        assert position_error(a, b) <= 1e-12
        assert accel_error(a, b) <= 1e-14
    for p in (P["PHI"], P["BETA2"], P["MIN_DISTANCE"], P["MAX_INFLUENCE"]):
        fin = np.isfinite(b[p])
        assert np.array_equal(np.isfinite(a[p]), fin)
        if not b[p][fin].any():             # a body alone: exact zeros, no relative error
            assert np.array_equal(a[p][fin], b[p][fin])
        else:
            assert rel_err(a[p][fin], b[p][fin]) <= (2e-15 if p < 100 else 1e-15)


@pytest.mark.parametrize("n", [1, 2, 5, 33, 64, 130, 256, 300, 301])
def test_leaves_what_the_step_kernel_leaves(n):
    pl = _system(n, seed=21)
    pl[40] = 1e-4                       # EXJ2, C_POTENTIAL and GI as another program may have left them
    pl[82:100] = 7.0
    calls = [("integrate", 600.0, 3), ("integrate", -300.0, 2), ("rk12", 600.0, 2), ("rk12", 500.0, 1)]
    for k in (1, 2, 4):
        a, ta = _go(pl, calls[:k], False)
        b, tb = _go(pl, calls[:k], True)
        assert ta == tb
        _same(a, b, n)


def test_odd_bodies_stay_on_the_step_kernel():
    """No mass, no radius, a mass rate, a moment of inertia of zero, planes handed over on the device: bit for bit the
    step kernel's results."""
    base = _system(40, seed=22)
    for plane, value in ((39, 0.0), (41, 0.0), (53, 0.0), (52, 0.0), (42, 1e3)):
        pl = base.copy()
        pl[plane, 7] = value
        a, _ = _go(pl, [("integrate", 600.0, 2)], False)
        b, _ = _go(pl, [("integrate", 600.0, 2)], True)
        assert np.array_equal(a, b, equal_nan=True), plane
    a, _ = _go(base, [("integrate", 600.0, 2)], False, device_copy=True)
    b, _ = _go(base, [("integrate", 600.0, 2)], True)
    assert np.array_equal(a, b)


def test_two_calls_are_one():
    pl = _system(97, seed=23)
    assert np.array_equal(_go(pl, [("integrate", 600.0, 5)], False)[0][0:100],
                          _go(pl, [("integrate", 600.0, 2), ("integrate", 600.0, 3)], False)[0][0:100])


@pytest.mark.parametrize("then", ["nothing", "upload", "costs", "autotune", "larger", "accel"])
def test_planes_the_caller_holds_stay_on_the_step_kernel(then):
    """The caller may write to planes whose address it has, until a larger system is uploaded: whatever else is called
    in between, a spin written there turns the frames (the step kernel's results, bit for bit)."""
    import torch
    from ephemeris_b200 import Context, PLANES as P
    pl = _system(40, seed=24)
    spun = pl.copy()
    spun[P["W"] + 2, 5] = 1e-4
    spun[P["GL_HI"] + 2, 5] = 1e-4 * spun[P["GI"] + 8, 5]

    def through(c):                                     # writes `spun` to the context's planes, as its owner may
        ptr = c.device_planes_ptr() if then == "larger" else held
        src = Context(0)
        src.upload(spun)
        torch.cuda.synchronize()
        _copy(ptr, src.device_planes_ptr(), spun.nbytes)
        src.close()

    c = Context(0)
    c.upload(_system(30, seed=24) if then == "larger" else pl)
    held = c.device_planes_ptr()
    if then in ("upload", "larger"):
        c.upload(pl)
    elif then == "costs":
        c.set_body_costs(None)
    elif then == "autotune":
        c.autotune(600.0, 1, 1, False)
        c.set_launch(0, 0)
    elif then == "accel":
        c.accel()
    through(c)
    c.integrate(600.0, 2)
    out = c.download()
    c.close()
    r = Context(0)
    r.upload(pl)
    r.set_launch(0, 8)
    held = r.device_planes_ptr()
    through(r)
    r.integrate(600.0, 2)
    ref = r.download()
    r.close()
    assert not np.array_equal(ref[P["S_HI"]:P["S_HI"] + 9, 5], pl[P["S_HI"]:P["S_HI"] + 9, 5])
    assert np.array_equal(out, ref)


def _copy(dst, src, nbytes):
    from cuda.bindings import runtime
    err, = runtime.cudaMemcpy(dst, src, nbytes, runtime.cudaMemcpyKind.cudaMemcpyDeviceToDevice)
    assert int(err) == 0
    err, = runtime.cudaDeviceSynchronize()
    assert int(err) == 0


@pytest.mark.parametrize("n", [41, 77, 143, 200])
def test_tuned_shapes_are_kept_apart(n):
    """A system with a mass rate stays on the step kernel, and a shape tuned for it is one of that kernel: a later system
    of the same size that may run on the point-mass kernel is tuned by itself and stays there."""
    from ephemeris_b200 import Context, PLANES as P
    pl = _system(n, seed=25)
    barred = pl.copy()
    barred[P["DGM"], 1] = 1e-3
    c = Context(0)
    c.upload(barred)
    c.autotune(600.0, 2, 2, True)
    c.close()
    c = Context(0)
    c.upload(pl)
    c.autotune(600.0, 2, 2, True)
    c.integrate(600.0, 2)
    out = c.download()
    c.close()
    assert np.array_equal(out, _go(pl, [("integrate", 600.0, 2)], False)[0])
    assert not np.array_equal(out, _go(pl, [("integrate", 600.0, 2)], True)[0])
