"""2D sets past the whole-step launch whose candidate rows are too long for their
masks, everywhere or in places, also across the seam of a small bucket grid, with
one and two phases, alone and in a batch: against the oracle bit for bit."""
import numpy as np
import pytest

from oracle.oracle import JACOBI, OracleWorld
from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu


def graded(n, near, far):
    side = int(np.ceil(np.sqrt(n)))
    i = np.arange(n)
    rng = np.random.default_rng(n)
    x = np.concatenate([[0.0], np.cumsum(near + (far - near) * np.arange(side) / (side - 1))[:-1]])
    q = np.zeros((n, 4), np.float32)
    q[:, 0] = x[i % side]
    q[:, 1] = (i // side) * 0.5 * (near + far)
    q[:, :2] += 0.01 * rng.standard_normal((n, 2))
    q[:, 2:] = 0.2 * rng.standard_normal((n, 2))
    return q


def worlds(q, phases):
    from phi_eng_b200.world import World2

    w, o = World2(), OracleWorld(cap=len(q))
    cfg = default_config()
    ph = None
    if phases:
        cfg.phase_count = 2
        cfg.phase_rest_density[1] = 0.5
        cfg.phase_mass[1] = 0.03125
        cfg.artificial_viscosity = 0.2
        ph = (np.arange(len(q)) % 3 == 0).astype(np.uint8)
    w.fluid.config = cfg
    o.set_config(cfg)
    w.fluid.set_cap(len(q))
    w.fluid.add_particles(q[:, :2]) if ph is None else w.fluid.add_particles_phase(q[:, :2], ph)
    o.add_particles(q[:, :2], ph)
    w.fluid.set_state(q)
    o.set_state(q)
    return w, o


@pytest.mark.parametrize("phases", [False, True])
@pytest.mark.parametrize("grid", [None, (2, 3), (5, 5)])
@pytest.mark.parametrize("near, far", [(0.1, 0.1), (0.1, 0.25), (0.2, 0.14)])
@pytest.mark.parametrize("n", [4200, 9001])
def test_dense_sets_match_the_oracle(n, near, far, grid, phases):
    w, o = worlds(graded(n, near, far), phases)
    if grid:
        w.set_grid(*grid, -3, 1)
    for _ in range(2):
        w.step(1 / 600)
        o.step(1 / 600, JACOBI)
    np.testing.assert_array_equal(w.fluid.particles, o.state())


def test_dense_scenes_of_a_batch():
    from phi_eng_b200.batch import Batch

    qs = [graded(700, 0.1, 0.25), graded(5000, 0.2, 0.14), graded(64, 0.1, 0.1)]
    pairs = [worlds(q, False) for q in qs]
    b = Batch([w for w, _ in pairs])
    b.step(1 / 600, 2)
    for k, (_, o) in enumerate(pairs):
        for _ in range(2):
            o.step(1 / 600, JACOBI)
        np.testing.assert_array_equal(b.scene_particles(k), o.state())
