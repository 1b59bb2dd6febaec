"""Tensor-core training on chunk planes (cnn_train.cuh) at the edges of its tiles: few rows, few
channels, column segments and batches that end within a tile."""
import numpy as np
import pytest

from oracle import cnn_oracle as CO

pytestmark = pytest.mark.gpu


def P():
    import optimizec_b200 as mod

    return mod


@pytest.mark.parametrize("layers,ch,H,W,B", [
    (3, 8, 16, 16, 1),    # one chunk, 8 image rows per weight-gradient item
    (2, 32, 1, 16, 3),    # one row: both halo rows are the image row itself
    (4, 16, 5, 48, 2),    # two chunks, 2 rows per item, a last item of one row
    (3, 24, 9, 144, 1),   # 24 channels in 4 chunks, a second column segment of 16
    (6, 32, 24, 32, 2),
    (4, 32, 7, 272, 1),   # three column segments
    (3, 3, 33, 128, 2),   # a tile per row start, 3 hidden channels
])
def test_gradients_match_fp32_at_the_edges(layers, ch, H, W, B):
    """Forward, loss and every layer's gradient against the FP32 path, with the tolerances of the
    tensor-core training tests (bf16 operands); a wrong halo column, tap or chunk is a fault of at least
    1 / sqrt(W) in the gradients."""
    rng = np.random.default_rng(H * 7 + W)
    net = P().CNN(layers, ch, seed=5)
    x = rng.standard_normal((B, 3, H, W)).astype(np.float32)
    t = rng.standard_normal((B, 1, H, W)).astype(np.float32)
    y_ref = net.forward(x)
    loss_ref, g_ref = net.loss_grad(x, t)
    net.set_train_tc(True)
    y = net.forward(x)
    loss, g = net.loss_grad(x, t)
    _, g2 = net.loss_grad(x, t)
    net.close()
    assert np.linalg.norm(y - y_ref) <= 1e-2 * np.linalg.norm(y_ref)
    assert loss == pytest.approx(loss_ref, rel=2e-2)
    off = 0
    for ci, co in CO.layer_shapes(layers, ch):
        n = co * ci * 9 + co
        assert np.linalg.norm(g[off:off + n] - g_ref[off:off + n]) <= 5e-2 * np.linalg.norm(g_ref[off:off + n])
        off += n
    assert np.linalg.norm(g - g_ref) <= 2e-2 * np.linalg.norm(g_ref)
    np.testing.assert_array_equal(g, g2)


def test_batches_and_sizes_in_turn():
    """The operand buffers are laid out anew for each batch and size: a smaller pass after a larger one
    gives what a fresh network gives; batches larger than one gather launch holds are drawn whole."""
    rng = np.random.default_rng(1)
    a, b = P().CNN(4, 32, seed=2), P().CNN(4, 32, seed=2)
    for n in (a, b):
        n.set_train_tc(True)
    big = [rng.standard_normal((3, c, 40, 64)).astype(np.float32) for c in (3, 1)]
    small = [rng.standard_normal((2, c, 12, 16)).astype(np.float32) for c in (3, 1)]
    a.loss_grad(*big)
    la, ga = a.loss_grad(*small)
    lb, gb = b.loss_grad(*small)
    assert la == lb
    np.testing.assert_array_equal(ga, gb)
    x, t = (rng.standard_normal((600, c, 4, 16)).astype(np.float32) for c in (3, 1))
    l_ref, _ = a.loss_grad(x, t)
    a.set_dataset(x, t)
    assert a.train(1, 600, 1e-4, seed=3)[0] == pytest.approx(l_ref, rel=1e-6)
    a.close()
    b.close()
