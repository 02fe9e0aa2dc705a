"""Worlds that grow while they run: every addition past the capacity moves the
particle arrays to new memory. Sizes around the arrays' alignment, against the
oracle bit for bit."""
import numpy as np
import pytest

from oracle.oracle import JACOBI, OracleWorld, OracleWorld3
from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phases", [False, True])
@pytest.mark.parametrize("dim", [2, 3])
def test_added_particles(dim, phases):
    from phi_eng_b200.world import World2
    from phi_eng_b200.world3 import World3

    w = World2() if dim == 2 else World3()
    o = (OracleWorld if dim == 2 else OracleWorld3)(cap=1 << 16)
    cfg = default_config()
    if phases:
        cfg.phase_count = 2
        cfg.phase_rest_density[1] = 0.5
        cfg.phase_mass[1] = 0.03125
    w.fluid.config = cfg
    o.set_config(cfg)
    w.fluid.set_cap(1 << 16)
    rng = np.random.default_rng(dim)
    side = 64 if dim == 2 else 20
    first = 0
    for count in (1, 62, 1, 960, 1, 1024, 3, 2048, 5000, 7):
        i = first + np.arange(count)
        p = np.stack([i // side**d % side for d in range(dim)], -1) + 0.5 + 0.1 * rng.random((count, dim))
        p = np.ascontiguousarray(0.25 * p, np.float32)
        if phases:
            ph = (i % 3 == 0).astype(np.uint8)
            assert w.fluid.add_particles_phase(p, ph) == count
            o.add_particles(p, ph)
        else:
            assert w.fluid.add_particles(p) == count
            o.add_particles(p)
        first += count
        for _ in range(2):
            w.step(1 / 600)
            o.step(1 / 600, JACOBI)
        np.testing.assert_array_equal(w.fluid.particles, o.state())
    for a, b in zip(w.fluid.density_pressure(), o.density_pressure()):
        np.testing.assert_array_equal(a, b)
