"""The getters' rows, put together on the device, against the fields of a saved state of the same
moment: the same FP32 values as doubles, in insertion order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# slab fields (slot order in a saved state, after its 88-byte header)
OX, VX, S0, E0, RHO, MASS, KEY, INFO, PID, EQPS, EP0, DMG, SMAX, NX, COUNT = (0, 3, 6, 12, 18, 19, 20, 21, 22, 23, 24, 30,
                                                                              31, 32, 35)


def _scene(name):
    from graphyt_gb300 import scenes
    if name == "damage":
        return scenes.damage_block()
    if name == "two bodies":
        return scenes.two_blocks(rigid_second=True)
    if name == "2D":
        return scenes.block_2d()
    if name == "warm":
        return scenes.thermal_block(n_side=6)
    return scenes.tiny_block(n_side=1)


@pytest.mark.parametrize("name", ["one", "damage", "two bodies", "2D", "warm"])
@pytest.mark.parametrize("steps", [0, 1, 4])
def test_getters_equal_the_saved_state(gpu_lib, tmp_path, name, steps):
    from graphyt_gb300 import graphyt
    sc = _scene(name)
    s = graphyt.from_scene(sc)
    s.iterate_GPU_steps(steps)
    s.save(str(tmp_path / "s"))
    raw = np.fromfile(str(tmp_path / "s"), np.uint8)[88:88 + 4 * COUNT * sc.n]
    f = np.frombuffer(raw.tobytes(), np.float32).reshape(COUNT, sc.n)
    at = np.empty(sc.n, np.int64)  # slot of each particle
    at[f[PID].view(np.int32)] = np.arange(sc.n)
    has_dp = name == "damage"
    for field, first, w, on in [("vel", VX, 3, True), ("stress", S0, 6, True), ("strain", E0, 6, True),
                                ("pstrain", EP0, 6, has_dp), ("eqps", EQPS, 1, has_dp), ("damage", DMG, 1, has_dp),
                                ("smax", SMAX, 1, has_dp), ("mass", MASS, 1, True), ("density", RHO, 1, True)]:
        want = f[first:first + w, at].T.astype(np.float64) if on else np.zeros((sc.n, w))
        assert np.array_equal(s._get_particles(field).reshape(sc.n, w), want), field
    assert np.array_equal(s._get_particles("pos0"), sc.pos)
    assert np.array_equal(s._get_particles("pos"), sc.pos + s._get_particles("disp"))
    if steps == 0:
        assert not np.any(s._get_particles("disp"))
    vol = s._get_particles("volume")
    first_vol = sc.psep ** (3 if sc.is3D else 2)
    want = f[MASS, at].astype(np.float64) / f[RHO, at].astype(np.float64)
    assert np.allclose(vol, want if steps else first_vol, rtol=1e-15, atol=0)
    assert np.array_equal(s._get_particles_int("device_slot"), at)
    assert np.array_equal(s._get_particles_int("material"), sc.mat)
    assert np.array_equal(s._get_particles_int("object"), sc.obj)
    if name == "warm" and steps == 0:
        assert np.array_equal(s._get_particles("temp"), sc.temp.astype(np.float32))
    # the rows use memory that the next step writes: a step after reading equals one without
    b = graphyt.from_scene(sc)
    b.iterate_GPU_steps(steps)
    for q in (s, b):
        q.iterate_GPU(steps * q.dt, steps)
    for field in ("vel", "stress", "density"):
        x, y = s._get_particles(field), b._get_particles(field)
        assert np.linalg.norm(x - y) <= 2e-6 * max(np.linalg.norm(y), 1e-30)  # the order of P2G's atomics
    s.close()
    b.close()
