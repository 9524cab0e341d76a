"""What is not a number stays visible: a value that has gone bad is passed on, not turned into an
ordinary one, whichever kernel takes it."""
import numpy as np
import pytest

from graphyt_gb300 import scenes

pytestmark = pytest.mark.gpu

STATE_HEADER = 88  # bytes before a saved state's first field, the offset along x of every slot


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_a_nan_offset_reaches_the_nodes(gpu_lib, tmp_path, axis):
    """A particle whose offset is NaN makes its stencil's nodes, and so its neighbours, NaN: the warp
    P2G (p2g_lanes 3) spreads it to the particles that the column kernel (9), with the weights as
    they are defined, does."""
    from graphyt_gb300 import graphyt
    sc = scenes.tiny_block(model=1, n_side=6)
    path = str(tmp_path / "s")
    bad = []
    for lanes in (9, 3):
        s = graphyt.from_scene(sc, options=dict(p2g_lanes=lanes))
        s.iterate_GPU(0.0, 0)
        s.save(path)
        state = np.fromfile(path, np.uint8)
        state[STATE_HEADER:].view(np.float32)[axis * sc.n + sc.n // 2] = np.nan
        state.tofile(path)
        s.load(path)
        assert np.isnan(s._get_particles("pos")[:, axis]).sum() == 1
        s.iterate_GPU(s.dt, 1)
        bad.append(np.isnan(s._get_particles("vel")).any(axis=1))
        s.close()
    assert bad[0].sum() > 1
    # the slots of the two handles hold the particles in the same order: one particle was hit
    assert np.array_equal(bad[0], bad[1])
