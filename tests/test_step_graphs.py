"""Several steps per call (four substeps per graph launch once the parameters
have run sixteen) against the same steps one call each: the same bits, substep
counts and clock, before and after a change of the time step; 2D, 3D, batches."""
import numpy as np
import pytest

from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu

CALLS = [(1 / 240, 3), (1 / 240, 22), (1 / 240, 5), (1 / 300, 21)]


def block(n, dims):
    side = int(np.ceil(n ** (1 / dims)))
    i = np.arange(n)
    rng = np.random.default_rng(11)
    q = np.zeros((n, 2 * dims), np.float32)
    q[:, :dims] = 0.25 * np.stack([i // side**a % side for a in range(dims)], -1) + 0.02 * rng.random((n, dims))
    q[:, dims:] = 0.3 * rng.standard_normal((n, dims))
    return q


def world(dims):
    if dims == 2:
        from phi_eng_b200.world import World2 as World
    else:
        from phi_eng_b200.world3 import World3 as World
    n = 9001
    q = block(n, dims)
    w = World()
    w.fluid.set_cap(n)
    w.fluid.config = default_config()
    assert w.fluid.add_particles(q[:, :dims]) == n
    w.fluid.set_state(q)
    return w


@pytest.mark.parametrize("dims", [2, 3])
def test_calls_of_many_steps(dims):
    a, b = world(dims), world(dims)
    for dt, k in CALLS:
        a.step_n(dt, k)
        for _ in range(k):
            b.step(dt)
    np.testing.assert_array_equal(a.fluid.particles, b.fluid.particles)
    assert a.time == b.time
    assert a.status().substeps == b.status().substeps == sum(k for _, k in CALLS)


def test_batch_calls_of_many_steps():
    from phi_eng_b200.batch import Batch

    a, b = (Batch([world(2), world(2)]) for _ in range(2))
    for dt, k in CALLS:
        a.world.step_n(dt, k)
        for _ in range(k):
            b.world.step_n(dt, 1)
    np.testing.assert_array_equal(a.world.fluid.particles, b.world.fluid.particles)
