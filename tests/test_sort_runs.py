"""The placement of the general bucket sort from the previous sort's order:
buckets of 31 to 33 particles (the longest finished as one run is 32), runs
across its blocks of 256 slots, ids in and out of slot order, particles that
enter and leave buckets between steps; 2D and 3D against the oracle bit for bit."""
import numpy as np
import pytest

from oracle.oracle import JACOBI, OracleWorld, OracleWorld3
from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu


def clusters(n, dims, h, speed, shuffled):
    """Cells three apart with 1, 2, 30 .. 34 or 70 particles near their middle."""
    rng = np.random.default_rng(7)
    sizes = [1, 2, 30, 31, 32, 33, 34, 70]
    cell = []
    while len(cell) < n:
        cell += [len(cell)] * sizes[rng.integers(len(sizes))]
    cell = np.unique(cell[:n], return_inverse=True)[1]
    side = int(np.ceil((cell.max() + 1) ** (1 / dims)))
    at = np.stack([cell // side**a % side for a in range(dims)], -1)
    q = np.zeros((n, 2 * dims), np.float32)
    q[:, :dims] = (3 * at + 0.5 + 0.9 * (rng.random((n, dims)) - 0.5)) * h
    q[:, dims:] = speed * rng.standard_normal((n, dims))
    return q[rng.permutation(n)] if shuffled else q


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("speed", [0.0, 3.0])
@pytest.mark.parametrize("n", [8193, 9001])
def test_2d_matches_the_oracle(n, speed, shuffled):
    from phi_eng_b200.world import World2

    cfg = default_config()
    q = clusters(n, 2, cfg.smoothing_length, speed, shuffled)
    w, o = World2(), OracleWorld(cap=n)
    w.fluid.set_cap(n)
    w.fluid.config = cfg
    o.set_config(cfg)
    assert w.fluid.add_particles(q[:, :2]) == n
    o.add_particles(q[:, :2])
    w.fluid.set_state(q)
    o.set_state(q)
    for _ in range(4):
        w.step(1 / 240)
        o.step(1 / 240, JACOBI)
    np.testing.assert_array_equal(w.fluid.particles, o.state())
    # a new state meets the order of the old one
    w.fluid.set_state(q[::-1].copy())
    o.set_state(q[::-1].copy())
    for _ in range(2):
        w.step(1 / 240)
        o.step(1 / 240, JACOBI)
    np.testing.assert_array_equal(w.fluid.particles, o.state())


@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("speed", [0.0, 3.0])
def test_3d_matches_the_oracle(speed, shuffled):
    from phi_eng_b200.world3 import World3

    n = 9001
    cfg = default_config()
    q = clusters(n, 3, cfg.smoothing_length, speed, shuffled)
    w, o = World3(), OracleWorld3(cap=n)
    w.fluid.set_cap(n)
    w.fluid.config = cfg
    o.set_config(cfg)
    assert w.fluid.add_particles(q[:, :3]) == n
    o.add_particles(q[:, :3])
    w.fluid.set_state(q)
    o.set_state(q)
    for _ in range(4):
        w.step(1 / 240)
        o.step(1 / 240, JACOBI)
    np.testing.assert_array_equal(w.fluid.particles, o.state())
