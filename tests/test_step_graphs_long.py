"""As test_step_graphs, with enough steps that the graph of four substeps is made:
in one long call, over several short ones, and dropped again by another time
step."""
import numpy as np
import pytest

from test_step_graphs import world

pytestmark = pytest.mark.gpu

CALLS = [(1 / 240, 3), (1 / 240, 51), (1 / 300, 20), (1 / 300, 20), (1 / 300, 20), (1 / 300, 6), (1 / 240, 47),
         (1 / 240, 48)]


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
