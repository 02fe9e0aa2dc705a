"""A world stepped and read by a thread other than the one that made it (a new
thread's current device is device 0; with a second GPU the world lives on that
one, where the launches of these calls must go), and the thread's current device
is what it was afterwards."""
import threading

import numpy as np
import pytest

from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim, n", [(2, 500), (2, 9000), (3, 500), (3, 9000)])
def test_calls_from_another_thread(dim, n):
    import torch

    from phi_eng_b200.world import World2
    from phi_eng_b200.world3 import World3

    dev = torch.cuda.device_count() - 1
    side = int(np.ceil(n ** (1 / dim)))
    i = np.arange(n)
    q = np.zeros((n, 2 * dim), np.float32)
    for d in range(dim):
        q[:, d] = (i // side**d % side + 0.5) * 0.25

    def make():
        w = World2() if dim == 2 else World3()
        w.fluid.config = default_config()
        w.fluid.set_cap(n)
        w.fluid.add_particles(q[:, :dim])
        w.fluid.set_state(q)
        w.step(1 / 600)
        return w

    def calls(w, out):
        w.step_n(1 / 600, 100)
        out.append(w.fluid.particles)
        w.step_n(1 / 600, 3)
        out.append(w.fluid.particles)
        out.append(torch.cuda.current_device())

    with torch.cuda.device(dev):
        a, b = make(), make()
        here, there = [], []
        calls(a, here)
        t = threading.Thread(target=calls, args=(b, there))
        t.start()
        t.join(120)
        assert len(there) == 3 and there[2] == 0 and here[2] == dev
        for x, y in zip(here[:2], there[:2]):
            np.testing.assert_array_equal(x, y)
        a.close()
        b.close()
