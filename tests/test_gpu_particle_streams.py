"""A particle set beside other work of the process: the perturbers' maxima (min_distance, max_influence) of a call are
those of that call alone, whatever is queued on the default stream when it is made."""
import numpy as np
import pytest

from tests.test_gpu_particle_shapes import _cloud, _points
from tests.test_gpu_particles import _combined

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("own_stream", [True, False])
def test_maxima_with_work_pending_on_the_default_stream(tmp_path, own_stream):
    import torch
    from ephemeris_b200 import Particles
    sysm = _points(9)
    cloud = _cloud(sysm, 300, 7)
    pl, md, _, n = _combined(tmp_path, sysm, cloud, "points")
    got = []
    for pending in (False, True):
        p = Particles(0)
        stream = torch.cuda.Stream()
        if not own_stream:
            p.set_stream(stream.cuda_stream)
        p.upload(np.ascontiguousarray(pl[:, :n]), md, np.ascontiguousarray(pl[0:12, n:]))
        t = p.integrate(4320.0, 9)          # leaves the inverted distances and the records' buffers in place
        torch.cuda.synchronize()
        if pending:
            torch.cuda._sleep(100_000_000)  # some 50 ms on the default stream
        p.integrate(4320.0, 9, t)
        torch.cuda.synchronize()
        got.append(p.download()[0])
        p.close()
    assert np.isfinite(got[0]).all()
    assert np.array_equal(got[0], got[1])


def test_a_call_that_fails_leaves_the_time_and_the_set(tmp_path):
    """A call on a stream that is being captured cannot wait for its work: it reports an error, the caller's time stays
    that of the particles (none of whose steps ran), and the set goes on afterwards as if the call had not been made."""
    import ctypes
    import torch
    from ephemeris_b200 import Particles
    sysm = _points(5)
    pl, md, _, n = _combined(tmp_path, sysm, _cloud(sysm, 100, 8), "points")
    got = []
    for broken in (False, True):
        p = Particles(0)
        p.upload(np.ascontiguousarray(pl[:, :n]), md, np.ascontiguousarray(pl[0:12, n:]))
        t = p.integrate(4320.0, 17)
        if broken:
            hi, lo = ctypes.c_double(t[0]), ctypes.c_double(t[1])
            stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
            with torch.cuda.stream(stream):
                graph.capture_begin(capture_error_mode="relaxed")
                p.set_stream(stream.cuda_stream)
                rc = p.lib.eph_particles_integrate(p.h, 4320.0, 17, ctypes.byref(hi), ctypes.byref(lo))
                p.set_stream(None)
                with pytest.raises(RuntimeError):
                    graph.capture_end()                  # the wait has ended the capture
            assert rc != 0 and (hi.value, lo.value) == tuple(t)
        t = p.integrate(4320.0, 17, t)
        got.append((*p.download(), t))
        p.close()
    assert got[0][2] == got[1][2]
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])


def test_an_error_that_was_reported_fails_no_later_call(tmp_path):
    """After a call that reported an error, every entry point that launches a kernel on the default stream or a stream of
    its own runs as before."""
    import torch
    from ephemeris_b200 import Context, EphError, Server, bspline_fit_batch
    sysm = _points(5)
    pl, md, _, n = _combined(tmp_path, sysm, _cloud(sysm, 10, 9), "points")
    pl = np.ascontiguousarray(pl[:, :n])
    c = Context(0)
    c.upload(pl, md)

    def broken():
        stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.stream(stream):
            graph.capture_begin(capture_error_mode="relaxed")
            c.set_stream(stream.cuda_stream)
            with pytest.raises(EphError):
                c.integrate(4320.0, 1)
            c.set_stream(None)
            with pytest.raises(RuntimeError):
                graph.capture_end()

    broken()
    samples, _ = c.record_samples(4320.0, 20, 1)
    c.close()
    c = Context(0)
    c.upload(pl, md)
    assert np.array_equal(samples, c.record_samples(4320.0, 20, 1)[0])
    broken()
    coefs = bspline_fit_batch(np.ascontiguousarray(samples.transpose(1, 0, 2)), 10, 3)
    assert np.isfinite(coefs).all()
    srv = Server(coefs, pl[39], 8640.0)
    broken()
    assert np.isfinite(srv.eval(8640.0)).all()
    broken()
    state = np.concatenate([pl[0:12, 1:2] + np.array([[1e10], [0], [0]] + [[0]] * 9)])
    out, accepted, _ = srv.result(srv.submit(state, 0.0, 8640.0, tol=1e-12, h0=8640.0))
    assert accepted >= 1 and np.isfinite(out).all()
    srv.close()
    c.close()
