"""The one-launch forward pass of a training batch (hidden widths 128 and 256): loss and gradient
against the CPU oracle where it can go wrong: one tile, rows that are padded, a second tile on
some CTAs. A width of 384 goes a layer a launch; its weight gradients, like all, read the
activations and dL/dZ row-major, here over three column tiles."""
import numpy as np
import pytest

from oracle import mlp_oracle as MO


@pytest.fixture(scope="module")
def ucb_engine():
    import ucb

    eng = ucb.Engine(0)
    yield eng
    eng.close()


# 148 SMs: 149 tiles give one CTA a second tile
@pytest.mark.gpu
@pytest.mark.parametrize("hidden,layers,rows", [(128, 1, 5), (128, 3, 128), (128, 2, 300), (128, 3, 149 * 128 - 7),
                                                (256, 1, 128), (256, 2, 73 * 128 + 1), (256, 2, 150 * 128), (384, 2, 300)])
def test_gradient_matches_the_oracle(ucb_engine, hidden, layers, rows):
    import ucb

    rng = np.random.default_rng(hidden + layers + rows)
    net = ucb.Mlp(ucb_engine, fourier=64, hidden=hidden, layers=layers, seed=3, batch=1024, train_steps=1)
    try:
        net.set_target_scale(0.2, 1.7)
        u = rng.uniform(size=(rows, 2)).astype(np.float32)
        y = rng.normal(size=rows).astype(np.float32)
        loss, g = net.loss_grad(u, y)
        again, h = net.loss_grad(u, y)
        assert again == loss and np.array_equal(g, h)
        lo, go = MO.loss_and_grad(net.get_params(), net.fourier(), u, y,
                                  hidden, layers, beta=0.5, y_mean=0.2, y_std=1.7, bf16=True)
        assert abs(loss - lo) < 2e-3 * max(1.0, abs(lo))
        # BF16 operands (2^-9 a rounding) on both sides, rounded at values that differ by FP32
        # rounding and the hardware tanh: the gradients agree to a few BF16 steps of their norm
        off = 0
        for o, i in MO.layer_shapes(64, hidden, layers):
            for k in (o * i, o):
                a, b = g[off:off + k], go[off:off + k]
                assert np.linalg.norm(a - b) < 2e-2 * np.linalg.norm(go) + 2e-2 * np.linalg.norm(b)
                off += k
        assert off == len(g)
    finally:
        net.close()
