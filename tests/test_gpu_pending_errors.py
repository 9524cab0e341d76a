"""A call that fails on the host leaves no error behind in the CUDA runtime for the next call to
answer for: handles initialise, step and answer as if nothing had happened."""
import ctypes as C

import numpy as np
import pytest
import torch

from graphyt_gb300 import scenes
from tests.helpers import rel_l2

pytestmark = pytest.mark.gpu


def _no_such_device():
    """A gy_create that fails on the host: there is no such device."""
    from graphyt_gb300 import _lib
    g = _lib.GridDesc()
    g.L[:] = [1.0, 1.0, 1.0]
    g.cellsize, g.psep = 0.125, 0.0625
    h = C.c_void_p()
    assert _lib.load().gy_create(C.byref(g), 9999, C.byref(h)) != 0


def test_a_failed_call_leaves_no_error_behind(gpu_lib):
    from graphyt_gb300 import _lib, graphyt
    _no_such_device()
    s = graphyt.from_scene(scenes.two_blocks())
    s.iterate_GPU_steps(2)
    s.close()
    _no_such_device()
    prm = torch.ones(int(gpu_lib.gy_mlp_param_count()), device="cuda")
    X, Y = torch.zeros(5, 16, device="cuda"), torch.full((5, 7), np.nan, device="cuda")
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(gpu_lib.gy_mlp_forward(p(prm), p(X), 5, p(Y), None, stream))
    assert torch.isfinite(Y).all()


def test_getters_are_not_refused_for_another_handles_error(gpu_lib):
    from graphyt_gb300 import graphyt
    s = graphyt.from_scene(scenes.two_blocks())
    s.iterate_GPU_steps(2)
    want = s._get_particles("pos"), s._get_particles_int("material")
    _no_such_device()
    got = s._get_particles("pos"), s._get_particles_int("material")
    for a, b in zip(got, want):
        assert np.array_equal(a, b)
    s.close()


@pytest.mark.parametrize("use_graph", [1, 0])
def test_a_step_is_not_refused_for_another_handles_error(gpu_lib, use_graph):
    """A step refused after its launch would leave the device one scalar slot and one sort ahead of
    the host; the later steps, past all 32 slots of the ring, are those of an undisturbed handle
    (tolerance: the order of the node sums, as in the repeat-run test)."""
    from graphyt_gb300 import graphyt
    out = []
    for disturbed in (True, False):
        s = graphyt.from_scene(scenes.two_blocks(), options=dict(use_graph=use_graph))
        dt = s.dt
        for k in range(40):
            if disturbed and k in (0, 1, 5, 17):
                _no_such_device()
            if k == 20:  # new scalars reach the step they are set for
                s.setDt(0.5 * dt)
            s.iterate_GPU(k * dt, k)
        out.append({f: s._get_particles(f) for f in ("pos", "vel", "stress", "density")})
        s.close()
    for f in out[0]:
        assert rel_l2(out[0][f], out[1][f]) <= 2e-6, f
