"""The U-Net's gradient sums where they take several CTAs and two passes: more
than 4096 pixels a channel, more than 16 tiles (a ragged last group), odd
batches; against the CPU oracle with the gradient bounds of its other tests.
The sums are those of both convolution paths; the FP32 one follows the oracle's
ReLU and pooling decisions, the tensor-core one (split activations) not always:
one flipped pixel of 64 x 64 is worth 4e-4 of the gradient."""
import numpy as np
import pytest

from conftest import rel
from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h, n, cores", [(72, 3, False), (72, 3, True), (64, 1, True)])
def test_gradient_sums_match_oracle(gpulib, monkeypatch, h, n, cores):
    from sparseimaging_b200 import warmstart
    if cores:
        monkeypatch.setenv("MFISTA_UNET_CUDA_CORES", "1")
    rng = np.random.default_rng(h)
    net = warmstart.UNet(h, h, n)
    p = net.params()
    x = rng.standard_normal((n, 2, h, h)).astype(np.float32)
    t = np.abs(rng.standard_normal((n, h, h))).astype(np.float32)
    _, g = net.grad(x, t)
    _, g_ref = U.UNetOracle(p).loss_and_grad(x, t)
    assert rel(g, g_ref) < 1e-4
    lay, hw, hb, _ = U.layout()
    for w0, b0 in lay + [(hw, hb)]:  # weights, then the biases behind them
        assert rel(g[w0:b0], g_ref[w0:b0]) < 1e-3
        assert rel(g[b0:b0 + 16], g_ref[b0:b0 + 16]) < 1e-3
    net.close()


@pytest.mark.parametrize("h", [24, 72])  # widths 3 and 9 at the coarsest level
def test_weight_copies_follow_training(gpulib, h):
    """The convolutions' rounded weight copies after training steps are those of
    the parameters: a fresh net with them gives the same output and gradient."""
    from sparseimaging_b200 import warmstart
    rng = np.random.default_rng(h)
    x = rng.standard_normal((2, 2, h, h)).astype(np.float32)
    t = np.abs(rng.standard_normal((2, h, h))).astype(np.float32)
    net, fresh = warmstart.UNet(h, h, 2), warmstart.UNet(h, h, 2)
    for _ in range(3):
        net.train_step(x, t, 1e-3)
    before = fresh.forward(x)
    fresh.set_params(net.params())
    y = net.forward(x)
    assert not np.array_equal(y, before)
    np.testing.assert_array_equal(y, fresh.forward(x))
    np.testing.assert_array_equal(net.grad(x, t)[1], fresh.grad(x, t)[1])
    net.close()
    fresh.close()
