"""Rows that are not finite (set_state_device takes them; they live under the
sentinel key, no other particle sees them): a world that steps in whole-step
launches against the same world stepped pass by pass, which timing the phases
makes it do, in both modes."""
import numpy as np
import pytest

from phi_eng_b200 import _abi
from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu

ROWS = {
    "position": (np.nan, 1.0, 0.5, -0.25),
    "infinite_position": (1.0, np.inf, 0.5, -0.25),
    "velocity": (1.0, 1.0, np.nan, 0.5),
    "infinite_velocity": (1.0, 1.0, 0.5, -np.inf),
}


@pytest.mark.parametrize("mode", [_abi.EXACT, _abi.TOLERANCE])
@pytest.mark.parametrize("n", [1, 96, 1100])
@pytest.mark.parametrize("row", list(ROWS))
def test_whole_step_launch_matches_the_passes(row, n, mode):
    import torch

    from phi_eng_b200.world import World2

    side = int(np.ceil(np.sqrt(n)))
    i = np.arange(n)
    q = np.zeros((n, 4), np.float32)
    rng = np.random.default_rng(1)
    q[:, :2] = (np.stack([i % side, i // side], -1) + 0.5 + 0.1 * (rng.random((n, 2)) - 0.5)) * 0.25
    bad = q.copy()
    bad[n // 2] = ROWS[row]
    bad[-1] = ROWS[row]
    t = torch.from_numpy(bad).cuda()
    got = []
    for passes in (False, True):
        w = World2()
        w.precision = mode
        w.fluid.config = default_config()
        w.fluid.set_cap(n)
        w.fluid.add_particles(q[:, :2])
        w.set_profiling(passes)
        w.step(1 / 600)
        w.set_state_device(t.data_ptr(), n)
        w.step_n(1 / 600, 1)
        one = w.fluid.particles
        w.step_n(1 / 600, 3)
        got.append((one, w.fluid.particles, *w.fluid.density_pressure()))
        w.close()
    for a, b in zip(*got):
        np.testing.assert_array_equal(a, b)
