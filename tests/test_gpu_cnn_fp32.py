"""FP32 convolutions and weight gradients at the edges of their tiles: images smaller than a tile,
widths that are no multiple of 4 or of a 64-column piece, channels beyond one tile of 32 and no
multiple of 8, fewer output channels than a tile."""
import numpy as np
import pytest

from oracle import cnn_oracle as CO

pytestmark = pytest.mark.gpu


def P():
    import optimizec_b200 as mod

    return mod


@pytest.mark.parametrize("layers,ch,H,W,B", [
    (2, 1, 1, 1, 1),      # one pixel: every tap is that pixel
    (3, 5, 1, 3, 2),      # one row, narrower than a pixel group
    (3, 8, 2, 17, 3),     # a second tile of one column
    (3, 9, 33, 16, 1),    # 9 output channels: a tile of 32 mostly empty; 33 rows: a last tile of one row
    (4, 40, 12, 20, 2),   # two input and two output channel tiles
    (3, 33, 7, 130, 1),   # three 64-column pieces, the last of 2 columns
    (3, 64, 9, 64, 2),
])
def test_loss_and_gradients_match_oracle(layers, ch, H, W, B):
    """FP32 sums of up to B H W products per CTA, then FP64: 1e-5 as the other FP32 gradient tests."""
    rng = np.random.default_rng(ch + W)
    net = P().CNN(layers, ch, seed=9)
    x = rng.standard_normal((B, 3, H, W)).astype(np.float32)
    t = rng.standard_normal((B, 1, H, W)).astype(np.float32)
    loss, g = net.loss_grad(x, t)
    _, g2 = net.loss_grad(x, t)
    y = net.forward(x)
    p = net.params().astype(np.float64)
    net.close()
    loss_ref, g_ref = CO.loss_grad(p, layers, ch, x, t)
    y_ref, _ = CO.forward(p, layers, ch, x)
    assert np.linalg.norm(y - y_ref) <= 1e-5 * np.linalg.norm(y_ref)
    assert loss == pytest.approx(loss_ref, rel=1e-5)
    assert np.linalg.norm(g - g_ref) <= 1e-5 * np.linalg.norm(g_ref)
    np.testing.assert_array_equal(g, g2)
