"""The U-Net's gradient sums where they take several CTAs and two passes: more
than 4096 pixels a channel, more than 16 tiles (a ragged last group), odd
batches; against the CPU oracle with the bounds of its other tests."""
import numpy as np
import pytest

from conftest import rel
from oracle import unet_oracle as U

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h, n", [(72, 3), (64, 1)])
def test_gradient_sums_match_oracle(gpulib, h, n):
    from sparseimaging_b200 import warmstart
    rng = np.random.default_rng(h)
    net = warmstart.UNet(h, h, n)
    p = net.params()
    x = rng.standard_normal((n, 2, h, h)).astype(np.float32)
    t = np.abs(rng.standard_normal((n, h, h))).astype(np.float32)
    loss, g = net.grad(x, t)
    loss_ref, g_ref = U.UNetOracle(p).loss_and_grad(x, t)
    assert abs(loss - loss_ref) <= 1e-5 * loss_ref
    assert rel(g, g_ref) < 1e-4
    lay, hw, hb, _ = U.layout()
    for w0, b0 in lay + [(hw, hb)]:  # weights, then the biases behind them
        assert rel(g[w0:b0], g_ref[w0:b0]) < 1e-3
        assert rel(g[b0:b0 + 16], g_ref[b0:b0 + 16]) < 1e-3
    net.close()
