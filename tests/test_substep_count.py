"""Substep counts of small worlds whose CFL substeps the GPU counts: equal to the
sum of the oracle's, also where status is read in between and the world leaves
the whole-step launch and comes back; and status never waits for queued steps."""
import numpy as np
import pytest

from oracle.oracle import JACOBI, OracleWorld
from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu

DT = 1 / 60


def config():
    c = default_config()
    c.cfl = 0.4
    c.max_substeps = 5
    return c


def state(n):
    side = int(np.ceil(np.sqrt(n)))
    i = np.arange(n)
    q = np.zeros((n, 4), np.float32)
    rng = np.random.default_rng(n)
    q[:, :2] = (np.stack([i % side, i // side], -1) + 0.5 + 0.1 * (rng.random((n, 2)) - 0.5)) * 0.25
    q[:, 2:] = 3.0 * rng.standard_normal((n, 2))
    return q


def world(n):
    from phi_eng_b200.world import World2

    w = World2()
    w.fluid.config = config()
    w.fluid.set_cap(n)
    w.fluid.add_particles(state(n)[:, :2])
    w.fluid.set_state(state(n))
    return w


@pytest.mark.parametrize("n", [96, 1100, 4096])
def test_counts_match_the_oracle(n):
    w, o = world(n), OracleWorld(cap=n)
    o.set_config(config())
    o.add_particles(state(n)[:, :2])
    o.set_state(state(n))
    total = [0]

    def advance(steps, one_by_one):
        for _ in range(steps):
            total[0] += o.cfl_substeps(DT)
            o.step(DT, JACOBI)
        for _ in range(steps if one_by_one else 1):
            w.step_n(DT, 1 if one_by_one else steps)

    def check():
        w.sync()
        assert w.status().substeps == total[0]
        assert w.status().substeps == total[0]

    advance(4, True)
    w.status()
    advance(3, False)
    check()
    for x in (w, o):  # turbulence: one launch per pass, the host counts
        x.set_turbulence(0.5, seed=3)
    advance(2, True)
    check()
    for x in (w, o):
        x.set_turbulence(0.5, seed=3, enabled=False)
    advance(70, False)  # more than one launch takes
    advance(2, True)
    check()
    np.testing.assert_array_equal(w.fluid.particles, o.state())


def test_status_does_not_wait():
    import torch

    w = world(4000)
    s = torch.cuda.Stream()
    w.set_stream(s.cuda_stream)
    w.step(DT)
    s.synchronize()
    done = torch.cuda.Event()
    w.step_n(DT, 256)  # some 10 ms
    done.record(s)
    before = w.status().substeps
    w.check()
    assert not done.query()
    s.synchronize()
    assert 1 <= before <= w.status().substeps >= 257
    w.close()
