"""An Adam step from a caller's gradient vector uses, and reads, its NPARAMS
gradient entries only: the same step from a vector that ends there as from one
with the loss entry behind them, whatever that holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_vector_without_the_loss_entry():
    import torch

    from phi_eng_b200.closure import NPARAMS, Mlp

    rng = torch.Generator(device="cuda").manual_seed(4)
    x = torch.randn(4096, 16, device="cuda", generator=rng)
    t = torch.randn(4096, 2, device="cuda", generator=rng)
    got = []
    for ends in (NPARAMS + 1, NPARAMS, NPARAMS + 1):
        m = Mlp(seed=7)
        for k in range(3):
            g = m.shard_grad(x, t, 0, 1024, 1024, 11)
            if len(got) == 2:
                g[NPARAMS] = float("nan")
            m.apply_grad(g[:ends].clone(), 1e-3)
        assert m.steps == 3
        got.append(m.get()[0])
    np.testing.assert_array_equal(got[0], got[1])
    np.testing.assert_array_equal(got[0], got[2])
    assert not np.array_equal(got[0], Mlp(seed=7).get()[0])
