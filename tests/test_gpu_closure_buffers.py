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
