"""A network created, or first used, while the default stream still has work ahead of it has the
parameters and predictions of one created on an idle device: its buffers are cleared on that
stream and filled on another."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ucb_engine():
    import ucb

    eng = ucb.Engine(0)
    yield eng
    eng.close()


def busy(torch):
    """Some 20 ms of ordinary work on the default stream, queued and not waited for."""
    a = torch.ones(4096, 4096, device="cuda")
    for _ in range(8):
        a = torch.matmul(a, a) * 1e-4
    return a


# fused prediction (128, 256) and the layer-by-layer one with buffers of its own (384)
@pytest.mark.parametrize("hidden", [128, 256, 384])
def test_network_created_behind_queued_work(ucb_engine, hidden):
    import torch
    import ucb

    rows = 1000
    u = torch.rand(rows, 2, device="cuda", generator=torch.Generator(device="cuda").manual_seed(5))

    def network(queued):
        torch.cuda.synchronize()
        kept = busy(torch) if queued else None
        net = ucb.Mlp(ucb_engine, fourier=64, hidden=hidden, layers=2, seed=11, batch=1024, train_steps=1)
        torch.cuda.synchronize()
        mean = torch.empty(rows, device="cuda")
        std = torch.empty(rows, device="cuda")
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        kept = busy(torch) if queued else kept
        net.predict(u.data_ptr(), rows, mean.data_ptr(), std.data_ptr(), stream.cuda_stream)
        torch.cuda.synchronize()
        out = net.get_params(), net.fourier(), mean.cpu().numpy(), std.cpu().numpy()
        net.close()
        del kept
        return out

    ref = network(False)
    assert (ref[0] != 0).any() and (ref[2] != 0).any()
    for _ in range(5):
        for a, b in zip(network(True), ref):
            np.testing.assert_array_equal(a, b)
