"""FP32 weight gradients on both sides of the rule that takes few pixels and channels to the one-launch
kernel, and the tiled kernel with few channels and narrow images beyond it."""
import numpy as np
import pytest

from oracle import cnn_oracle as CO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers,ch,H,W,B", [
    (3, 16, 32, 64, 1),   # 2048 pixels x 256 channel pairs: the last that the rule takes
    (3, 17, 32, 64, 1),   # one channel more: the hidden layer beyond it, the outer ones within
    (3, 16, 3, 683, 1),   # 2049 pixels
    (3, 32, 8, 8, 8),     # 512 pixels x 1024 pairs: the last by pairs
    (3, 33, 2, 5, 1),     # 1089 pairs
    (2, 1, 2049, 1, 1),   # the tiled kernel on a column one pixel wide
    (3, 5, 700, 3, 1),
    (3, 8, 41, 17, 3),
    (3, 4, 9, 260, 1),    # five 64-column pieces, the last of 4 columns
])
def test_loss_and_gradients_match_oracle(layers, ch, H, W, B):
    """FP32 sums of at most 2049 products per thread or piece, then pairwise or in FP64: 1e-5 as the other
    FP32 gradient tests."""
    import optimizec_b200 as P

    rng = np.random.default_rng(ch * 1000 + W)
    net = P.CNN(layers, ch, seed=9)
    x = rng.standard_normal((B, 3, H, W)).astype(np.float32)
    t = rng.standard_normal((B, 1, H, W)).astype(np.float32)
    loss, g = net.loss_grad(x, t)
    _, g2 = net.loss_grad(x, t)
    p = net.params().astype(np.float64)
    net.close()
    loss_ref, g_ref = CO.loss_grad(p, layers, ch, x, t)
    assert loss == pytest.approx(loss_ref, rel=1e-5)
    off = 0
    for ci, co in CO.layer_shapes(layers, ch):
        n = co * ci * 9
        assert np.linalg.norm(g[off:off + n] - g_ref[off:off + n]) <= 1e-5 * np.linalg.norm(g_ref[off:off + n])
        off += n + co
    assert np.linalg.norm(g - g_ref) <= 1e-5 * np.linalg.norm(g_ref)
    np.testing.assert_array_equal(g, g2)


def test_sums_over_threads_lose_nothing():
    """One pixel per thread, so every sum of the one-launch kernel is over threads only, in FP64: with all
    weights zero the output is 0, dout = -2 t / 256 and the last bias gradient is its exact sum.  In FP32 the 1
    is lost beside 2^25."""
    import optimizec_b200 as P

    net = P.CNN(2, 1, seed=1)
    net.set_params(np.zeros(net.num_params(), dtype=np.float32))
    t = np.zeros((1, 1, 16, 16), dtype=np.float32)
    t.flat[0], t.flat[1], t.flat[128] = 2.0 ** 25, -2.0 ** 25, 1.0
    _, g = net.loss_grad(np.ones((1, 3, 16, 16), dtype=np.float32), t)
    net.close()
    assert g[-1] == -2.0 / 256
