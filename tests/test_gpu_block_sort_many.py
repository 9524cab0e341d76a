"""The block merge sort where more movers enter a block in one step than are ranked one against
another: they are sorted by slot, in a time that grows with their number and not with its square."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = 0.0625


def _converging(n, background):
    """Two piles of n particles, a cell block apart, flying into the block between them from lower and
    from higher slots, and particles at rest in it and around."""
    from graphyt_gb300 import scenes
    rng = np.random.default_rng(n)
    pile = 0.02 * H * (rng.random((2 * n, 3)) - 0.5) + 0.53
    pile[n:, 0] += 1.2512 - 0.53  # both reach their block boundary in the 19th step
    side = round(background ** (1 / 3))
    grid = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3) * (1.2 / max(side, 1)) + 0.35
    if background > 100000:  # beside the path: as heavy as that the particles at rest would stop the piles
        grid = (grid - 0.35) * (1.0 / 1.2) + [0.35, 0.75, 0.35]
    vel = np.zeros((2 * n + len(grid), 3))
    vel[:n, 0], vel[n:2 * n, 0] = 1.0, -1.0
    pos = np.concatenate([pile, grid])
    zero = np.zeros(len(pos), np.int32)
    base = scenes.tiny_block(model=1, n_side=4, cellsize=H)
    base.materials[0].update(bulkMod=1.0, shearMod=0.5)
    sc = scenes._finish(scenes.Scene("converging", [2.0] * 3, H, H / 2, pos, zero, zero.copy(), base.materials, CFL=0.3,
                                     vel=vel), None)
    sc.dt = 0.2 * H
    return sc


def _entering(x0, x1):
    """The most particles that enter one of the cell blocks along x."""
    b0, b1 = (np.floor((x / H - 0.25) / 4).astype(int) for x in (x0, x1))
    return np.bincount(b1[b0 != b1], minlength=1).max()


# slots of two (three), three and five digits; just below and above the limit of 256 entering
@pytest.mark.parametrize("n, background", [(128, 1000), (129, 1000), (700, 0), (3000, 27000), (400, 300763)])
def test_many_movers_into_a_block_keep_the_stable_order(gpu_lib, tmp_path, n, background):
    from graphyt_gb300 import graphyt
    sc = _converging(n, background)
    a = graphyt.from_scene(sc)
    b = graphyt.from_scene(sc, options=dict(full_sort=1))
    a.iterate_GPU_steps(15)
    most = 0
    for k in range(15, 24):  # a merges what the step before moved, b sorts the same state from scratch
        a.save(str(tmp_path / "s"))
        b.load(str(tmp_path / "s"))
        before = a._get_particles("pos")[:, 0]
        for s in (a, b):
            s.iterate_GPU(k * sc.dt, k)
        slots = a._get_particles_int("device_slot")
        assert np.array_equal(np.sort(slots), np.arange(sc.n)), k
        assert np.array_equal(slots, b._get_particles_int("device_slot")), k
        if k < 23:
            most = max(most, _entering(before, a._get_particles("pos")[:, 0]))
    assert most >= 2 * n
    a.close()
    b.close()


def test_a_pile_crossing_a_block_boundary_takes_no_longer_than_its_size(gpu_lib):
    """64,000 particles entering a block in one step: 1.3 ms, and 470 ms by ranks.  The worst of 60
    steps, waited for one by one, with room for a busy host."""
    from graphyt_gb300 import graphyt
    sc = _converging(32000, 1000)
    s = graphyt.from_scene(sc)
    worst = []
    for _ in range(2):
        s.iterate_GPU_steps(3)
        s.Synchronise()
        times = []
        for k in range(3, 40):
            t = time.perf_counter()
            s.iterate_GPU(k * sc.dt, k)
            s.Synchronise()
            times.append(time.perf_counter() - t)
        worst.append(max(times))
        s.close()
        s = graphyt.from_scene(sc)
    s.close()
    assert min(worst) < 0.05


@pytest.mark.parametrize("L", [(5.25, 5.25, 4.75), (10.25, 10.25, 10.25)])
def test_the_cluster_scan_gives_the_stable_sort(gpu_lib, tmp_path, L):
    """Grids of 8,379 and 68,921 cell blocks, just above and well above what one CTA scans, no multiple
    of four or eight: particles all over them, so that every CTA of the cluster has blocks with movers
    in and out, land slot for slot where a sort from scratch puts them."""
    from graphyt_gb300 import graphyt, scenes
    rng = np.random.default_rng(11)
    n = 60000
    pos = 0.2 + rng.random((n, 3)) * (np.array(L) - 0.5)
    vel = rng.uniform(-1.5, 1.5, (n, 3))
    zero = np.zeros(n, np.int32)
    base = scenes.tiny_block(model=1, n_side=4, cellsize=H)
    base.materials[0].update(bulkMod=1.0, shearMod=0.5)
    sc = scenes._finish(scenes.Scene("spread", list(L), H, H / 2, pos, zero, zero.copy(), base.materials, CFL=0.3, vel=vel),
                        None)
    sc.dt = 0.2 * H
    a = graphyt.from_scene(sc)
    b = graphyt.from_scene(sc, options=dict(full_sort=1))
    a.iterate_GPU_steps(2)
    for k in range(2, 8):
        a.save(str(tmp_path / "s"))
        b.load(str(tmp_path / "s"))
        before = a._get_particles_int("device_slot")
        for s in (a, b):
            s.iterate_GPU(k * sc.dt, k)
        slots = a._get_particles_int("device_slot")
        assert np.array_equal(np.sort(slots), np.arange(n)), k
        assert np.array_equal(slots, b._get_particles_int("device_slot")), k
        assert np.mean(slots != before) > 0.5, k
    a.close()
    b.close()
