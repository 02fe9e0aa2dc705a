"""3D sets whose candidate rows are long in some places and short in others, so
that a warp holds particles with one mask word per row, with two and with none,
and rows past the terms that the small sets' density pass keeps; also far from
the origin, where the quick distance test does not apply. Against the oracle bit
for bit, in the passes of small and of large sets, and in the tolerance mode
against the same set beside a distant one."""
import numpy as np
import pytest

from oracle.oracle import JACOBI, OracleWorld3
from phi_eng_b200 import _abi
from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu


def graded(n, near, far, offset=0.0):
    """A block whose spacing grows from `near` to `far` along x (cells of h = 0.5:
    0.25 gives rows of 24 slots, 0.2 of 47, 0.17 of 77, 0.14 of 137)."""
    side = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    a = np.stack([i % side, i // side % side, i // side**2], -1)
    rng = np.random.default_rng(n)
    step = near + (far - near) * np.arange(side) / max(side - 1, 1)
    x = np.concatenate([[0.0], np.cumsum(step)[:-1]])
    p = np.stack([x[a[:, 0]], a[:, 1] * 0.5 * (near + far), a[:, 2] * 0.5 * (near + far)], -1)
    q = np.zeros((n, 6), np.float32)
    q[:, :3] = p + 0.02 * rng.standard_normal((n, 3))
    q[:, 0] += offset
    q[:, 3:] = 0.2 * rng.standard_normal((n, 3))
    return q


def world(q, mode=_abi.EXACT):
    from phi_eng_b200.world3 import World3

    w = World3()
    w.precision = mode
    w.fluid.config = default_config()
    w.fluid.set_cap(len(q))
    assert w.fluid.add_particles(q[:, :3]) == len(q)
    w.fluid.set_state(q)
    return w


@pytest.mark.parametrize("offset", [0.0, 40000.0])
@pytest.mark.parametrize("near, far", [(0.25, 0.2), (0.25, 0.15), (0.2, 0.17), (0.14, 0.25)])
@pytest.mark.parametrize("n", [700, 9000, 30000, 52000])
def test_graded_blocks_match_the_oracle(n, near, far, offset):
    q = graded(n, near, far, offset)
    w = world(q)
    o = OracleWorld3(cap=max(4096, n))
    o.set_config(default_config())
    o.add_particles(q[:, :3])
    o.set_state(q)
    for _ in range(2):
        w.step(1 / 600)
        o.step(1 / 600, JACOBI)
    np.testing.assert_array_equal(w.fluid.particles, o.state())
    for a, b in zip(w.fluid.density_pressure(), o.density_pressure()):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("near, far", [(0.25, 0.15), (0.14, 0.25)])
@pytest.mark.parametrize("n", [9000, 30000])
def test_tolerance_mode_beside_a_distant_block(n, near, far):
    a, b = graded(n, near, far), graded(52000, 0.25, 0.2)
    b[:, 0] += 200.0
    w1, w2 = world(a, _abi.TOLERANCE), world(np.concatenate([a, b]), _abi.TOLERANCE)
    for w in (w1, w2):
        w.step_n(1 / 600, 2)
    np.testing.assert_array_equal(w1.fluid.particles, w2.fluid.particles[:n])
