"""Parameters set from host memory are the ones the next training step starts from: the
upload and the kernel that makes the BF16 copies are ordered on one stream."""
import numpy as np
import pytest


@pytest.fixture(scope="module")
def ucb_engine():
    import ucb

    eng = ucb.Engine(0)
    yield eng
    eng.close()


@pytest.mark.gpu
def test_parameters_set_from_the_host_are_the_ones_trained(ucb_engine):
    import torch
    import ucb

    net = ucb.Mlp(ucb_engine, fourier=64, hidden=256, layers=5, seed=7, batch=16384, train_steps=1)
    try:
        gen = torch.Generator(device="cuda").manual_seed(1)
        u = torch.rand(100000, 2, device="cuda", generator=gen)
        y = torch.sin(7 * u[:, 0]) * u[:, 1]
        torch.cuda.synchronize()
        start = net.get_params()

        def step(times):
            for _ in range(times):
                net.set_params(start)
            net.fit(u.data_ptr(), y.data_ptr(), u.shape[0])
            return net.get_params()

        step(1)
        ref = step(3)  # the second and third upload find the values already in place
        for _ in range(12):
            # the step before moved every parameter, so a copy made too early would differ
            assert np.array_equal(step(1), ref)
    finally:
        net.close()
