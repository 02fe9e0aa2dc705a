"""Worlds of different sizes stepped in turn and from several threads (one world
per thread; ctypes releases the interpreter lock during a call): the launches of
one world leave those of another as they are. 2D worlds of whole-step launches
and 3D worlds of one-launch sorts, whose kernels take more shared memory the
larger the world, against the oracle bit for bit."""
import threading

import numpy as np
import pytest

from oracle.oracle import JACOBI, OracleWorld, OracleWorld3
from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu

SIZES = {2: (96, 4096, 700, 2500), 3: (500, 8000, 1200, 4100)}


def lattice(n, dim):
    side = int(np.ceil(n ** (1 / dim)))
    i = np.arange(n)
    q = np.zeros((n, 2 * dim), np.float32)
    rng = np.random.default_rng(n)
    for d in range(dim):
        q[:, d] = (i // side**d % side + 0.5 + 0.1 * (rng.random(n) - 0.5)) * 0.25
    q[:, dim:] = 0.1 * rng.standard_normal((n, dim))
    return q


def world(n, dim):
    from phi_eng_b200.world import World2
    from phi_eng_b200.world3 import World3

    w = World2() if dim == 2 else World3()
    q = lattice(n, dim)
    w.fluid.config = default_config()
    w.fluid.set_cap(n)
    w.fluid.add_particles(q[:, :dim])
    w.fluid.set_state(q)
    return w


def oracle(n, dim, dts):
    o = (OracleWorld if dim == 2 else OracleWorld3)(cap=max(4096, n))
    q = lattice(n, dim)
    o.set_config(default_config())
    o.add_particles(q[:, :dim])
    o.set_state(q)
    for dt in dts:
        o.step(dt, JACOBI)
    return o.state()


# a time step of its own for every step: the 3D worlds' graphs are captured anew
DTS = [1 / 600 * (1 + 1e-3 * k) for k in range(60)]


@pytest.mark.parametrize("dim", [2, 3])
def test_worlds_stepped_in_turn(dim):
    ws = [world(n, dim) for n in SIZES[dim]]
    for k, dt in enumerate(DTS[:6]):
        for w in ws if k % 2 else reversed(ws):
            w.step(dt)
    for w, n in zip(ws, SIZES[dim]):
        np.testing.assert_array_equal(w.fluid.particles, oracle(n, dim, DTS[:6]))


@pytest.mark.parametrize("dim", [2, 3])
def test_worlds_stepped_by_threads(dim):
    ws = [world(n, dim) for n in SIZES[dim]]
    errors = []
    gate = threading.Barrier(len(ws))

    def run(w):
        try:
            gate.wait(30)
            for dt in DTS:
                w.step(dt)
        except Exception as e:  # reported by the main thread
            errors.append(e)

    ts = [threading.Thread(target=run, args=(w,)) for w in ws]
    for t in ts:
        t.start()
    for t in ts:
        t.join(120)
    assert not errors
    for w, n in zip(ws, SIZES[dim]):
        np.testing.assert_array_equal(w.fluid.particles, oracle(n, dim, DTS))
