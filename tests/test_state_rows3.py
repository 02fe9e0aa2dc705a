"""Host copies of a 3D world's state: reads (whole, partial, repeated), writes and
the calls between them always see the latest state, on both sides of the sizes
at which the world keeps rows on the host (4,096 written, 4,096 and 131,072
read), against a world of the same particles that is only stepped and read."""
import ctypes as C

import numpy as np
import pytest

from phi_eng_b200._abi import default_config

pytestmark = pytest.mark.gpu

F = C.POINTER(C.c_float)
SIZES = [1, 700, 4096, 4097, 8192, 8193, 131072, 131073]


def lattice(n, seed):
    side = int(np.ceil(n ** (1 / 3)))
    i = np.arange(n)
    q = np.zeros((n, 6), np.float32)
    rng = np.random.default_rng(seed)
    for d in range(3):
        q[:, d] = (i // side**d % side + 0.5 + 0.1 * (rng.random(n) - 0.5)) * 0.25
    q[:, 3:] = 0.2 * rng.standard_normal((n, 3))
    return q


def world(q, cfl=False):
    from phi_eng_b200.world3 import World3

    w = World3()
    c = default_config()
    if cfl:
        c.cfl, c.max_substeps = 0.4, 4
    w.fluid.config = c
    w.fluid.set_cap(len(q) + 10)
    assert w.fluid.add_particles(q[:, :3]) == len(q)
    return w


def read(w, k):
    out = np.full((k, 6), np.nan, np.float32)
    assert w._lib.phieng_world3_fluid_get(w._h, out.ctypes.data_as(F), k) == k
    return out


def reference(q, steps, cfl=False):
    """The state set on a fresh world, stepped."""
    w = world(q, cfl)
    w.fluid.set_state(q)
    if steps:
        w.step_n(1 / 600, steps)
    s = read(w, len(q))
    w.close()
    return s


@pytest.mark.parametrize("n", SIZES)
def test_reads_and_writes(n):
    a, b = lattice(n, 1), lattice(n, 2)
    w = world(a)
    w.step(1 / 600)
    w.fluid.set_state(b)
    np.testing.assert_array_equal(read(w, n), b)  # read before any step
    np.testing.assert_array_equal(read(w, min(n, 7)), b[:7])
    w.step(1 / 600)
    r1 = reference(b, 1)
    np.testing.assert_array_equal(read(w, min(n, 7)), r1[:7])  # a part, the whole, again, a part
    for _ in range(3):
        np.testing.assert_array_equal(read(w, n), r1)
    np.testing.assert_array_equal(read(w, min(n, 7)), r1[:7])
    w.step(1 / 600)
    np.testing.assert_array_equal(read(w, n), reference(b, 2))
    w.fluid.set_state(a)
    w.fluid.set_state(b)  # twice before a step
    w.step(1 / 600)
    np.testing.assert_array_equal(read(w, n), r1)
    w.close()


@pytest.mark.parametrize("n", [2, 700, 6000, 9000])
def test_calls_between(n):
    a, b = lattice(n, 1), lattice(n, 2)
    r1 = reference(b, 1)
    # a part of the state replaced after a read, and after a whole write
    for steps in (0, 1):
        w = world(a)
        w.step(1 / 600)
        w.fluid.set_state(b)
        if steps:
            w.step(1 / 600)
            read(w, n)
        w.fluid.set_state(a[:1])
        c = (r1 if steps else b).copy()
        c[0] = a[0]
        np.testing.assert_array_equal(read(w, n), c)
        w.step(1 / 600)
        np.testing.assert_array_equal(read(w, n), reference(c, 1))
        w.close()
    # particles added, the configuration changed, a snapshot taken before the upload
    w = world(a)
    w.step(1 / 600)
    w.fluid.set_state(b)
    blob = w.save_fluid_block()
    extra = np.array([[-3.0, -3.0, -3.0]], np.float32)
    w.fluid.add_particles(extra)
    s = read(w, n + 1)
    np.testing.assert_array_equal(s[:n], b)
    np.testing.assert_array_equal(s[n], [-3, -3, -3, 0, 0, 0])
    w.load_fluid_block(blob)
    np.testing.assert_array_equal(read(w, n), b)
    w.step(1 / 600)
    w.fluid.set_state(b)
    cfg = w.fluid.config
    cfg.smoothing_length = np.float32(0.4)
    w.fluid.config = cfg
    w.step(1 / 600)
    got = read(w, n)
    w2 = world(a)
    w2.fluid.config = cfg
    w2.fluid.set_state(b)
    w2.step(1 / 600)
    np.testing.assert_array_equal(got, read(w2, n))
    w.fluid.clear()
    assert w.fluid.add_particles(extra) == 1
    np.testing.assert_array_equal(read(w, 1), [[-3, -3, -3, 0, 0, 0]])
    w.close()
    w2.close()


@pytest.mark.parametrize("n", [700, 9000])
def test_cfl_substeps_after_a_write(n):
    a, b = lattice(n, 1), lattice(n, 2)
    b[:, 3:] *= 20
    w = world(a, cfl=True)
    w.step(1 / 600)
    w.fluid.set_state(b)
    w.step_n(1 / 600, 2)
    np.testing.assert_array_equal(read(w, n), reference(b, 2, cfl=True))
    w.close()


@pytest.mark.parametrize("n", [64, 4096])
def test_writes_in_quick_succession(n):
    """A written state that its step has not taken yet is not overwritten by the next."""
    import torch

    a = [lattice(n, k) for k in range(6)]
    w = world(a[0])
    s = torch.cuda.Stream()
    w.set_stream(s.cuda_stream)
    got, busy = [], torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
    for q in a:
        with torch.cuda.stream(s):
            for _ in range(8):
                busy.fill_(1)  # the step below waits behind these
        w.fluid.set_state(q)
        w.step(1 / 600)
    got.append(read(w, n))
    np.testing.assert_array_equal(got[0], reference(a[-1], 1))
    for q in a:
        w.fluid.set_state(q)
        w.debug_forces()  # takes the state without stepping
    w.step(1 / 600)
    np.testing.assert_array_equal(read(w, n), reference(a[-1], 1))
    w.close()
