"""A batch of impacts off its lattice, with every node of a particle's stencil taking weight: the GPU
against the FP64 restatement over the steps in which the first particles yield and are damaged.

The Drucker-Prager law with damage returns a stress only where F > 0 and I1 < 0, with a finite jump
across I1 = 0, so a particle that sits on the gate takes one of two branches on the rounding of the
node sums.  What has to hold is that all other particles agree, and that those on the gate are as few
as runs of the restatement from positions a rounding apart show."""
import numpy as np
import pytest

from tests.helpers import oracle_ensemble, rel_l2, run_gpu

pytestmark = pytest.mark.gpu

MANY_STEP_TOL = 1e-3


@pytest.mark.parametrize("seed", [0, 1])
def test_off_lattice_batch_against_fp64_ensemble(gpu_lib, oracle_built, seed):
    from graphyt_gb300 import scenes
    sc = scenes.impact_batch(n_inst=5, seed=3, n_min=4000, n_max=20000)
    rng = np.random.default_rng(seed)
    sc.pos = sc.pos + 0.02 * sc.psep * rng.uniform(-1.0, 1.0, sc.pos.shape)
    for c in range(3):  # a smooth flow over the impact speed
        k = rng.uniform(0.5, 2.0, 3) * 2.0 * np.pi / max(sc.L)
        sc.vel[:, c] += 0.5 * np.sin(sc.pos @ k + rng.uniform(0.0, 2.0 * np.pi))
    steps = 50
    gpu = run_gpu(sc, steps)
    base, spread = oracle_ensemble(sc, [steps], ("vel", "stress", "eqps"), members=4)[steps]
    for f in base:
        got = gpu._get_particles(f)
        assert np.isfinite(got).all() and np.linalg.norm(base[f]) > 0, f
        assert rel_l2(got, base[f]) <= max(MANY_STEP_TOL, 2 * spread[f]), (f, rel_l2(got, base[f]), spread[f])
        # particle by particle: one in a thousand may sit on the gate, no more
        off = np.abs(got - base[f]).reshape(sc.n, -1).max(axis=1)
        rms = np.sqrt(np.mean(base[f] ** 2))
        assert np.mean(off > 10 * MANY_STEP_TOL * rms) <= 1e-3, (f, np.mean(off > 10 * MANY_STEP_TOL * rms))
    gpu.close()
