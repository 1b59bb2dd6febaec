"""A closed run captures the attached network's launches in CUDA graphs: the network's buffers have to
be there before the capture, whatever the network was used for until then."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, L = 64, 96


def P():
    import optimizec_b200 as mod

    return mod


def closed_state(net):
    s = P().Solver(N, 1e4, 4.0, 0.1)
    s.init_k4(3)
    s.next_dt()
    s.attach_closure(net, (1.0, 1.0, 1.0, 0.05), energy_check=1)
    return s


def test_network_trained_on_the_tensor_cores_then_attached():
    """In training mode the closure evaluates the network as im2col GEMMs; training at this width runs on
    chunk planes and leaves their buffers unallocated."""
    rng = np.random.default_rng(4)
    x, t = (rng.standard_normal((2, c, L, L)).astype(np.float32) for c in (3, 1))
    runs = []
    for warmed in (False, True):
        net = P().CNN(4, 16, seed=11)
        net.set_train_tc(True)
        net.set_dataset(x, t)
        net.train(2, 2, 1e-4, seed=1)
        s = closed_state(net)
        if warmed:
            s.closure_forcing()  # not captured
        s.step(4)
        runs.append(s.om2())
        s.close()
        net.close()
    np.testing.assert_array_equal(runs[0], runs[1])


@pytest.mark.parametrize("N_,channels", [(64, 16), (256, 32)])  # FP32 network; tensor-core inference (L = 384)
def test_network_used_otherwise_between_closed_steps(N_, channels):
    """Calls on the attached network with another image size or a larger batch replace its buffers; the
    closed run goes on as if they had not been made."""
    rng = np.random.default_rng(7)
    L_ = 3 * N_ // 2
    runs = []
    for used in (False, True):
        net = P().CNN(4, channels, seed=11)
        s = P().Solver(N_, 1e4, 4.0, 0.1)
        s.init_k4(3)
        s.next_dt()
        s.attach_closure(net, (1.0, 1.0, 1.0, 0.05), energy_check=1)
        for B, H, W in [(1, 16, 16), (3, L_, L_), (2, 128, 128)]:
            s.step(3)
            s.sync()
            if used:
                x, t = (rng.standard_normal((B, c, H, W)).astype(np.float32) for c in (3, 1))
                net.loss_grad(x, t)
                if channels == 32 and W % 128 == 0:
                    net.forward_tc(x)
        s.step(3)
        runs.append((s.om2(), s.closure_forcing()))
        s.close()
        net.close()
    np.testing.assert_array_equal(runs[0][0], runs[1][0])
    np.testing.assert_array_equal(runs[0][1], runs[1][1])
