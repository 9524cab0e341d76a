"""The step's block merge sort against a sort from scratch of the same keys: two handles hold the
same state, one continues with the merge and the other sorts from scratch, and after one step
every particle sits in the same slot (the sort's permutation, bit for bit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fast_block(n_side, speed, seed=4, jitter=0.3):
    """A block crossing the grid and spreading: many particles change cell and block per step."""
    from graphyt_gb300 import scenes
    sc = scenes.tiny_block(model=1, n_side=n_side, cellsize=0.0625, L=(2.0, 2.0, 2.0), gravity=(0.0, 0.0, 0.0))
    rng = np.random.default_rng(seed)
    sc.pos = sc.pos + jitter * sc.psep * rng.uniform(-1, 1, sc.pos.shape)
    sc.vel = speed * (1.0 + 0.5 * rng.standard_normal(sc.vel.shape))
    sc.materials[0].update(bulkMod=1.0, shearMod=0.5)  # soft: the particles fly, they do not interact
    return sc


def _piled(n):
    """n particles in one cell: a block of many chunks whose particles all share a key."""
    from graphyt_gb300 import scenes
    sc = _fast_block(4, 0.0)
    rng = np.random.default_rng(7)
    pos = 0.5 + 0.0625 * (0.3 + 0.4 * rng.random((n, 3)))
    zero = np.zeros(n, np.int32)
    out = scenes.Scene("piled", sc.L, sc.cellsize, sc.psep, pos, zero, zero.copy(), sc.materials, CFL=0.3,
                       vel=rng.standard_normal((n, 3)))
    return scenes._finish(out, None)


def _scene(name):
    """A scene and its time step: up to a third of a cell per step where it is fast."""
    from graphyt_gb300 import scenes
    if name in ("slow", "fast", "one", "piled"):
        sc = {"slow": lambda: _fast_block(11, 0.05), "fast": lambda: _fast_block(16, 1.0),
              "one": lambda: _fast_block(1, 1.0), "piled": lambda: _piled(3001)}[name]()
        sc.dt = 0.2 * sc.cellsize
        return sc
    return scenes.two_blocks() if name == "two bodies" else scenes.disk_impact_2d()


@pytest.mark.parametrize("name", ["slow", "fast", "one", "piled", "two bodies", "2D"])
def test_block_merge_gives_the_stable_sort(gpu_lib, tmp_path, name):
    from graphyt_gb300 import graphyt
    sc = _scene(name)
    a = graphyt.from_scene(sc)
    b = graphyt.from_scene(sc, options=dict(full_sort=1))
    moved = 0
    for k in range(0, 24, 3):
        a.iterate_GPU_steps(3, step0=k, t0=k * a.dt)
        a.save(str(tmp_path / "s"))
        b.load(str(tmp_path / "s"))
        before = a._get_particles_int("device_slot")
        if k == 12:  # the merge serves the next sort, whatever cadence follows
            a.set_options(sort_every=3)
        for s in (a, b):
            s.iterate_GPU((k + 3) * a.dt, k + 3)
        slots = a._get_particles_int("device_slot")
        assert np.array_equal(slots, b._get_particles_int("device_slot")), k
        assert np.array_equal(np.sort(slots), np.arange(sc.n))
        moved += int(np.sum(slots != before))
        if k == 12:
            a.set_options(sort_every=1)
    assert moved > 0 or name not in ("fast", "piled")
    a.Synchronise()
    a.close()
    b.close()


def test_block_merge_counts_survive_a_sort_from_scratch(gpu_lib, tmp_path):
    """Sorting from scratch between merged steps (full_sort on for a while, a state loaded) leaves
    no stale counts behind: the slots stay those of a handle that sorts from scratch throughout."""
    from graphyt_gb300 import graphyt
    sc = _scene("fast")
    a = graphyt.from_scene(sc)
    a.iterate_GPU_steps(4)
    a.set_options(full_sort=1)
    a.iterate_GPU_steps(2, step0=4)
    a.set_options(full_sort=0)
    a.iterate_GPU_steps(3, step0=6)
    a.save(str(tmp_path / "s"))
    b = graphyt.from_scene(sc, options=dict(full_sort=1))
    b.load(str(tmp_path / "s"))
    for s in (a, b):
        s.iterate_GPU(9 * a.dt, 9)
    assert np.array_equal(a._get_particles_int("device_slot"), b._get_particles_int("device_slot"))
    a.load(str(tmp_path / "s"))
    a.iterate_GPU(9 * a.dt, 9)
    assert np.array_equal(a._get_particles_int("device_slot"), b._get_particles_int("device_slot"))
    a.close()
    b.close()


@pytest.mark.parametrize("n_side", [20, 47])
def test_particle_update_does_not_depend_on_how_many_segments_there_may_be(gpu_lib, n_side):
    """The same block in a small grid and in one of so many cell blocks that the particle update
    loads ahead: segments of one chunk (8,000 particles) and of several, with remainders (103,823).
    The node sums add in another order from run to run: with up to 64 terms of 6e-8 a step's node
    velocity is good to 4e-6 of the fastest particle's, three steps' to 1.2e-5; a strain increment
    has the gradient 2 v / h times dt = 0.2 h, and the stress at most 3 K = 3 times the strain."""
    from graphyt_gb300 import graphyt
    out = []
    for L in (2.25, 8.0 if n_side == 20 else 4.0):
        sc = _fast_block(n_side, 0.5)
        sc.L = [L, L, L]
        sc.dt = 0.2 * sc.cellsize
        s = graphyt.from_scene(sc)
        s.iterate_GPU_steps(3)
        out.append([s._get_particles(f) for f in ("pos", "vel", "stress")])
        s.close()
    vmax = np.abs(sc.vel).max()
    for a, b, tol in zip(*out, (2e-5 * sc.dt, 2e-5, 3 * 2e-5)):
        assert np.isfinite(a).all() and np.ptp(a) > 0
        assert np.abs(a - b).max() <= tol * vmax


@pytest.mark.parametrize("n_side, bodies", [(80, 1), (80, 2), (160, 1)])
def test_large_problems_take_longer_segments(gpu_lib, n_side, bodies):
    """512,000 particles of one body, whose blocks' remainders of up to a warp go with the last
    piece, and of two bodies apart, whose particle update takes whole blocks; 4.1 million, whose P2G
    takes whole blocks.  Against full_sort, which cuts no pieces; tolerances as above."""
    from graphyt_gb300 import graphyt
    out = []
    for options in (None, dict(full_sort=1)):
        sc = _fast_block(n_side, 0.5)
        sc.L = [6.0, 6.0, 6.0] if n_side == 160 else [4.0, 4.0, 4.0]
        sc.dt = 0.2 * sc.cellsize
        if n_side == 160:
            sc.vel[np.arange(sc.n) % 200 > 0] = 0.0  # (few, for the surface takes them one by one)
        if bodies == 2:
            far = sc.pos[:, 0] > sc.pos[:, 0].mean()
            sc.obj[far] = 1
            sc.pos[far, 0] += 0.75
        s = graphyt.from_scene(sc, options=options)
        s.iterate_GPU_steps(3)
        out.append([s._get_particles(f) for f in ("pos", "vel", "stress")])
        s.close()
    vmax = np.abs(sc.vel).max()
    for a, b, tol in zip(*out, (2e-5 * sc.dt, 2e-5, 3 * 2e-5)):
        assert np.isfinite(a).all() and np.ptp(a) > 0
        assert np.abs(a - b).max() <= tol * vmax
