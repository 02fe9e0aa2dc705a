"""3D passes over the sizes at which their launch shape changes (one-launch
sort up to 8,192 particles; a thread per candidate row and eight lanes per
particle up to 49,152, in the tolerance mode 24,576), against the oracle bit for bit, and a
block alone against the same block beside a distant one large enough to send
the world through the one-thread passes: the same bits in both modes."""
import numpy as np
import pytest

from oracle.oracle import JACOBI, OracleWorld3
from phi_eng_b200 import _abi
from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 33, 1023, 1025, 8191, 8192, 8193, 24577, 49152, 49153]


def block(n, spacing=0.25, seed=3, order="zyx"):
    side = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    a, b, c = i % side, i // side % side, i // side**2
    p = np.stack([a, b, c] if order == "zyx" else [c, b, a], -1) + 0.5
    rng = np.random.default_rng(seed)
    q = np.zeros((n, 6), np.float32)
    q[:, :3] = (p + 0.1 * (rng.random((n, 3)) - 0.5)) * spacing
    q[:, 3:] = 0.2 * rng.standard_normal((n, 3))
    return q


def config(terms):
    c = default_config()
    if terms:
        c.artificial_viscosity = 0.2
        c.surface_tension = 8.0
        c.wall_friction = 0.3
        c.phase_count = 2
        c.phase_rest_density[1] = 0.5
        c.phase_mass[1] = 0.03125
    return c


def walls(w, lo=-0.05, hi=9.0):
    from phi_eng_b200.world3 import Box3, Sphere

    w.add_static_body((hi / 2, lo - 0.5, hi / 2), Box3(hi, 0.5, hi))
    w.add_static_body((lo - 0.5, hi / 2, hi / 2), Box3(0.5, hi, hi))
    w.add_static_body((1.0, 0.0, 1.0), Sphere(0.4))


def gpu_world(q, cfg, phases=None, mode=_abi.EXACT):
    from phi_eng_b200.world3 import World3

    w = World3()
    w.precision = mode
    walls(w)
    w.fluid.config = cfg
    w.fluid.set_cap(len(q))
    assert (w.fluid.add_particles(q[:, :3]) if phases is None else
            w.fluid.add_particles_phase(q[:, :3], phases)) == len(q)
    w.fluid.set_state(q)
    return w


class OracleWalls:
    """walls() on the oracle."""

    def __init__(self, o):
        self.o = o

    def add_static_body(self, pos, shape):
        d = getattr(shape, "radius", None)
        if d is not None:
            self.o.add_body(0, *pos, d)
        else:
            self.o.add_body(1, *pos, shape.hx, shape.hy, shape.hz)


def oracle_world(q, cfg, phases=None):
    o = OracleWorld3(cap=max(4096, len(q)))
    walls(OracleWalls(o))
    o.set_config(cfg)
    if phases is None:
        o.add_particles(q[:, :3])
    else:
        o.add_particles(q[:, :3], phases)
    o.set_state(q)
    return o


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("terms", [False, True])
def test_steps_match_the_oracle(n, terms):
    q = block(n, order="zyx" if n % 2 else "xyz")
    ph = (np.arange(n) % 3 == 0).astype(np.uint8) if terms else None
    cfg = config(terms)
    w, o = gpu_world(q, cfg, ph), oracle_world(q, cfg, ph)
    for _ in range(2):
        w.step(1 / 60)
        o.step(1 / 60, JACOBI)
    np.testing.assert_array_equal(w.fluid.particles, o.state())


@pytest.mark.parametrize("spacing", [0.25, 0.22, 0.2, 0.17, 0.12, 0.06])
@pytest.mark.parametrize("n", [3000, 50000])
def test_dense_blocks_match_the_oracle(spacing, n):
    """Rows past the 32 slots of a mask word (0.22, 0.2), past its two words
    (0.17, 0.12) and neighbour lists past their buffers (0.06: ~2,400
    neighbours), in the passes of small and of large sets."""
    if spacing < 0.1 and n > 3000:
        pytest.skip("2,400 neighbours of 50,000 particles: minutes on the oracle")
    q = block(n, spacing)
    cfg = default_config()
    w, o = gpu_world(q, cfg), oracle_world(q, cfg)
    w.step(1 / 60)
    o.step(1 / 60, JACOBI)
    np.testing.assert_array_equal(w.fluid.particles, o.state())


@pytest.mark.parametrize("mode", [_abi.EXACT, _abi.TOLERANCE])
@pytest.mark.parametrize("n, spacing", [(700, 0.25), (9000, 0.25), (30000, 0.25), (9000, 0.2), (30000, 0.15)])
def test_block_beside_a_distant_one(n, spacing, mode):
    a = block(n, spacing)
    far = block(50000)
    far[:, 0] += 100.0
    w1, w2 = gpu_world(a, default_config(), mode=mode), gpu_world(np.concatenate([a, far]), default_config(), mode=mode)
    for _ in range(3):
        w1.step(1 / 60)
        w2.step(1 / 60)
    np.testing.assert_array_equal(w1.fluid.particles, w2.fluid.particles[:n])


@pytest.mark.parametrize("n, spacing", [(2000, 0.25), (2000, 0.17), (52000, 0.25), (52000, 0.2)])
@pytest.mark.parametrize("shift", [0.0, 1.7, -3.3, 1e5])
def test_blocks_across_the_seam_match_the_oracle(n, spacing, shift):
    """The bucket grid is planned for the first positions; the block is then
    moved so that its x cells wrap (and, at 1e5, so far out that the quick
    distance test does not apply)."""
    q = block(n, spacing)
    w, o = gpu_world(q, default_config()), oracle_world(q, default_config())
    w.step(1 / 60)  # plans the grid
    o.step(1 / 60, JACOBI)
    s = o.state()
    s[:, 3] = shift * 60 * 20 if abs(shift) > 100 else shift * 60
    cfg = default_config()
    cfg.max_velocity = 1e9
    for x in (w.fluid, o):
        x.set_config(cfg)
    o.set_state(s)
    w2 = gpu_world(s, cfg)  # the same state, its grid planned before it moves
    for _ in range(3):
        w2.step(1 / 60)
        o.step(1 / 60, JACOBI)
    np.testing.assert_array_equal(w2.fluid.particles, o.state())
