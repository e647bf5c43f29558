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
