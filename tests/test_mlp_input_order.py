"""A fit that is given no stream, after set_params, trains on inputs that the default stream is still
writing when set_params is called: the call orders the engine's stream after the default one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_targets_written_before_set_params_are_the_ones_trained():
    import torch
    import ucb

    rows, eng = 20000, ucb.Engine(0)
    net = ucb.Mlp(eng, fourier=64, hidden=256, layers=2, seed=3, batch=1024, train_steps=4)
    gen = torch.Generator(device="cuda").manual_seed(2)
    u = torch.rand(rows, 2, device="cuda", generator=gen)
    target = torch.sin(5 * u[:, 0]) + u[:, 1]
    start = net.get_params()
    torch.cuda.synchronize()

    def fit(y):
        net.set_params(start)
        loss = net.fit(u.data_ptr(), y.data_ptr(), rows)
        return loss, net.get_params()

    ref = fit(target)
    for _ in range(5):
        y = torch.full_like(target, 50.0)
        torch.cuda.synchronize()
        a = torch.ones(4096, 4096, device="cuda")
        for _ in range(8):
            a = torch.matmul(a, a) * 1e-4
        y.copy_(target)
        got = fit(y)
        assert got[0] == ref[0]
        np.testing.assert_array_equal(got[1], ref[1])
    net.close()
    eng.close()
