"""Small worlds where the GPU cannot hold the whole-step launch's cluster (a GPU
partition with few multiprocessors; here the world is told so): they step pass
by pass, without an error and with the same bits, also when the answer changes
between steps."""
import numpy as np
import pytest

from phi_eng_b200 import _abi
from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu


def world(n, mode, cfl):
    from phi_eng_b200.world import Box, World2

    side = int(np.ceil(np.sqrt(n)))
    i = np.arange(n)
    w = World2()
    w.precision = mode
    c = default_config()
    if cfl:
        c.cfl, c.max_substeps = 0.4, 5
    w.fluid.config = c
    w.fluid.set_cap(n)
    w.add_static_body((5.0, -0.55), Box(10.0, 0.5))
    rng = np.random.default_rng(n)
    w.fluid.add_particles((np.stack([i % side, i // side], -1) + 0.1 * rng.random((n, 2))) * 0.25)
    return w


@pytest.mark.parametrize("cfl", [False, True])
@pytest.mark.parametrize("mode", [_abi.EXACT, _abi.TOLERANCE])
@pytest.mark.parametrize("n", [60, 500, 1100, 4096])
def test_passes_take_over(n, mode, cfl):
    a, b = world(n, mode, cfl), world(n, mode, cfl)
    for w, plan in ((a, (0, 0, 0)), (b, (1, 0, 1))):
        for off in plan:
            assert w._lib.phieng_sph_debug_no_cluster(w._h, off) == 1
            w.step_n(1 / 60, 3)
            w.step(1 / 60)
            if off:  # the host took the count and knows it at once
                assert w.status().substeps >= 4
        w.sync()
        assert w.status().error == _abi.OK
    assert a.status().substeps == b.status().substeps
    np.testing.assert_array_equal(a.fluid.particles, b.fluid.particles)
    for x, y in zip(a.fluid.density_pressure(), b.fluid.density_pressure()):
        np.testing.assert_array_equal(x, y)


def test_null_world():
    assert _abi.load().phieng_sph_debug_no_cluster(None, 1) == 0
