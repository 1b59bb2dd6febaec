"""Tensor-core training on chunk planes at its narrowest networks and at the edges of its tiles: a tile of the
convolutions is 128 consecutive pixels of the padded image (W + 2 to a row), an item of the weight gradient
64 consecutive image pixels."""
import numpy as np
import pytest

from oracle import cnn_oracle as CO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers,ch,H,W,B", [
    (3, 4, 64, 16, 1),    # 64 rows of 18: nine whole tiles; 4 channels, the fewest
    (3, 4, 7, 16, 2),     # 126 padded pixels: one tile, two positions to spare
    (2, 4, 1, 16, 3),     # items of three images' rows
    (3, 5, 8, 48, 1),     # items that begin within a row and end in the next
    (3, 17, 9, 80, 1),    # a second chunk pair with one channel; rows of 1.25 items
    (3, 31, 3, 144, 2),
])
def test_gradients_match_fp32(layers, ch, H, W, B):
    """Against the FP32 path with the tolerances of the tensor-core training tests (bf16 operands)."""
    import optimizec_b200 as P

    rng = np.random.default_rng(H * 11 + W)
    net = P.CNN(layers, ch, seed=5)
    x = rng.standard_normal((B, 3, H, W)).astype(np.float32)
    t = rng.standard_normal((B, 1, H, W)).astype(np.float32)
    y_ref = net.forward(x)
    loss_ref, g_ref = net.loss_grad(x, t)
    net.set_train_tc(True)
    y = net.forward(x)
    loss, g = net.loss_grad(x, t)
    net.close()
    assert np.linalg.norm(y - y_ref) <= 1e-2 * np.linalg.norm(y_ref)
    assert loss == pytest.approx(loss_ref, rel=2e-2)
    off = 0
    for ci, co in CO.layer_shapes(layers, ch):
        n = co * ci * 9 + co
        assert np.linalg.norm(g[off:off + n] - g_ref[off:off + n]) <= 5e-2 * np.linalg.norm(g_ref[off:off + n])
        off += n
    assert np.linalg.norm(g - g_ref) <= 2e-2 * np.linalg.norm(g_ref)
