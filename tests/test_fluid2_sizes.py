"""2D steps over the sizes at which their launch shape changes (whole steps in
one cluster launch of 1, 2, 4, 8 or 16 blocks up to 4,096 particles), against
the oracle bit for bit: optional terms, CFL substeps counted on the device,
wrapped and dense grids, steps taken one by one or several per call; and a
block alone against the same block beside a distant one that makes the world
too large for that launch: the same bits in both modes."""
import numpy as np
import pytest

from oracle.oracle import JACOBI, OracleWorld
from phi_eng_b200 import _abi, scenes
from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 31, 33, 255, 256, 257, 512, 1024, 1025, 2048, 2049, 4095, 4096, 4097]
BOXES = [(5.0, -0.55, 10.0, 0.5), (-0.55, 5.0, 0.5, 10.0)]


def block(n, spacing=0.25, seed=5):
    side = int(np.ceil(np.sqrt(n)))
    i = np.arange(n)
    rng = np.random.default_rng(seed)
    q = np.zeros((n, 4), np.float32)
    q[:, :2] = (np.stack([i % side, i // side], -1) + 0.5 + 0.1 * (rng.random((n, 2)) - 0.5)) * spacing
    q[:, 2:] = 0.3 * rng.standard_normal((n, 2))
    return q


def config(kind):
    c = default_config()
    if kind == "tait":
        c.gamma = 7.0
    if kind == "terms":
        c.artificial_viscosity = 0.2
        c.surface_tension = 8.0
        c.wall_friction = 0.3
        c.phase_count = 2
        c.phase_rest_density[1] = 0.5
        c.phase_mass[1] = 0.03125
    if kind in ("terms", "cfl"):
        c.cfl = 0.4
        c.max_substeps = 5
    return c


def worlds(q, cfg, phases=None, mode=_abi.EXACT, oracle=True):
    from phi_eng_b200.world import Box, Circle, World2

    w = World2()
    w.precision = mode
    w.fluid.set_cap(len(q))
    o = OracleWorld(cap=len(q)) if oracle else None
    for px, py, hx, hy in BOXES:
        w.add_static_body((px, py), Box(hx, hy))
        if o:
            o.add_box(px, py, hx, hy, (1.0, 0.0, -0.0, 1.0))
    w.add_static_body((1.5, 0.0), Circle(0.4))
    w.fluid.config = cfg
    got = w.fluid.add_particles(q[:, :2]) if phases is None else w.fluid.add_particles_phase(q[:, :2], phases)
    assert got == len(q)
    w.fluid.set_state(q)
    if o:
        o.add_circle(1.5, 0.0, 0.4)
        o.set_config(cfg)
        o.add_particles(q[:, :2]) if phases is None else o.add_particles(q[:, :2], phases)
        o.set_state(q)
    return w, o


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("kind", ["plain", "tait", "terms", "cfl"])
def test_steps_match_the_oracle(n, kind):
    q = block(n)
    ph = (np.arange(n) % 3 == 0).astype(np.uint8) if kind == "terms" else None
    w, o = worlds(q, config(kind), ph)
    for _ in range(3):
        w.step(1 / 60)
        o.step(1 / 60, JACOBI)
    w.step_n(1 / 60, 3)
    for _ in range(3):
        o.step(1 / 60, JACOBI)
    np.testing.assert_array_equal(w.fluid.particles, o.state())
    d, p = w.fluid.density_pressure()
    od, op = o.density_pressure()
    np.testing.assert_array_equal(d, od)
    np.testing.assert_array_equal(p, op)
    if kind in ("plain", "tait"):
        assert w.status().substeps == 6
    else:
        assert 6 <= w.status().substeps <= 30


@pytest.mark.parametrize("spacing", [0.12, 0.08, 0.03])
def test_dense_blocks_match_the_oracle(spacing):
    """More neighbours than a particle's list holds (0.12: ~54), rows past the
    32 slots of a mask (0.08), one bucket with most particles (0.03)."""
    q = block(2500, spacing)
    w, o = worlds(q, default_config())
    for _ in range(2):
        w.step(1 / 60)
        o.step(1 / 60, JACOBI)
    np.testing.assert_array_equal(w.fluid.particles, o.state())


@pytest.mark.parametrize("grid", [(2, 2), (3, 4), (6, 6)])
def test_wrapped_grids_match_the_oracle(grid):
    q = block(1500)
    w, o = worlds(q, config("terms"))
    w.set_grid(*grid, -3, 1)
    for _ in range(3):
        w.step(1 / 60)
        o.step(1 / 60, JACOBI)
    np.testing.assert_array_equal(w.fluid.particles, o.state())


@pytest.mark.parametrize("mode", [_abi.EXACT, _abi.TOLERANCE])
@pytest.mark.parametrize("n", [96, 1100, 4000])
def test_block_beside_a_distant_one(n, mode):
    a = block(n)
    far = block(4200)
    far[:, 0] += 500.0
    w1, _ = worlds(a, config("tait"), mode=mode, oracle=False)
    w2, _ = worlds(np.concatenate([a, far]), config("tait"), mode=mode, oracle=False)
    dt = scenes.fine_dt(config("tait"))
    w1.step_n(dt, 20)
    w2.step_n(dt, 20)
    np.testing.assert_array_equal(w1.fluid.particles, w2.fluid.particles[:n])
