"""The caller's buffers belong to the caller again as soon as a call returns, also
page-locked ones, which the GPU reads and writes directly: a state passed from
page-locked memory with steps still queued, its buffer refilled at once, against
the same state from ordinary memory."""
import numpy as np
import pytest

from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu


def lattice(n, dim, seed):
    side = int(np.ceil(n ** (1 / dim)))
    i = np.arange(n)
    q = np.zeros((n, 2 * dim), np.float32)
    rng = np.random.default_rng(seed)
    for d in range(dim):
        q[:, d] = (i // side**d % side + 0.5 + 0.1 * (rng.random(n) - 0.5)) * 0.25
    q[:, dim:] = 0.2 * rng.standard_normal((n, dim))
    return q


def world(q):
    from phi_eng_b200.world import World2
    from phi_eng_b200.world3 import World3

    dim = q.shape[1] // 2
    w = World2() if dim == 2 else World3()
    w.fluid.config = default_config()
    w.fluid.set_cap(len(q))
    assert w.fluid.add_particles(q[:, :dim]) == len(q)
    return w


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [700, 9000, 150000])
def test_state_from_page_locked_memory(n, dim):
    import torch

    first, second = lattice(n, dim, 1), lattice(n, dim, 2)
    pinned = torch.empty(first.shape, dtype=torch.float32, pin_memory=True).numpy()
    got = []
    for buf in (pinned, first.copy()):
        w = world(first)
        w.step_n(1 / 600, 200)  # still running when the state arrives
        buf[:] = second
        w.fluid.set_state(buf)
        buf[:] = 0.5
        w.step_n(1 / 600, 2)
        got.append(w.fluid.particles)
        w.close()
    np.testing.assert_array_equal(got[0], got[1])


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [700, 150000])
def test_state_read_into_page_locked_memory(n, dim):
    import ctypes as C

    import torch

    q = lattice(n, dim, 3)
    w = world(q)
    w.fluid.set_state(q)
    w.step_n(1 / 600, 40)
    pinned = torch.empty(q.shape, dtype=torch.float32, pin_memory=True).numpy()
    get = w._lib.phieng_world_fluid_get if dim == 2 else w._lib.phieng_world3_fluid_get
    assert get(w._h, pinned.ctypes.data_as(C.POINTER(C.c_float)), n) == n
    np.testing.assert_array_equal(pinned, w.fluid.particles)
    w.close()
