"""Networks of different depth and width trained on several host threads at once: the tensor-core
kernels' shared-memory limit belongs to the function, not to a network or a layer."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# layers, channels: operands of 2 and of 4 chunks, so kernels of different shared memory
NETS = [(6, 32), (3, 8), (5, 24), (2, 16)]


@pytest.mark.parametrize("H,W", [
    (16, 16),  # chunk planes
    (12, 20),  # im2col GEMMs (a width that is no multiple of 16)
])
def test_gradients_on_threads_equal_serial_ones(H, W):
    import optimizec_b200 as P

    rng = np.random.default_rng(W)
    x = rng.standard_normal((2, 3, H, W)).astype(np.float32)
    t = rng.standard_normal((2, 1, H, W)).astype(np.float32)
    nets = [P.CNN(l, c, seed=i) for i, (l, c) in enumerate(NETS)]
    for n in nets:
        n.set_train_tc(True)
    serial = [n.loss_grad(x, t) for n in nets]

    def many(n):
        return [n.loss_grad(x, t) for _ in range(300)]

    with ThreadPoolExecutor(len(nets)) as pool:
        got = list(pool.map(many, nets))
    for n in nets:
        n.close()
    for (loss, g), runs in zip(serial, got):
        for l, h in runs:
            assert l == loss
            np.testing.assert_array_equal(h, g)
