"""Order of the warm-start network's copies and products while the device's legacy
stream is busy with another thread's work."""
import threading

import numpy as np
import pytest


@pytest.mark.gpu
def test_new_parameters_are_ordered_with_training():
    """set_params clears the moments of the updates before the training that
    follows reads them, also when the legacy stream is held up (by kernels of
    some 10 ms that another thread goes on queueing): the parameters after an
    epoch are those of the same calls on an idle device, bit for bit."""
    torch = pytest.importorskip("torch")
    from pdal_gb300.learn import MLP

    rng = np.random.default_rng(5)
    net = MLP(200, 64, 90, seed=1)
    first, second = net.get_params(), (0.05 * rng.standard_normal(net.get_params().size)).astype(np.float32)
    net.set_data(rng.standard_normal((64, 200)).astype(np.float32), rng.standard_normal((64, 90)).astype(np.float32))

    def calls():
        net.set_params(first)
        net.train(2, 16, 1e-3, seed=3)    # moments that would show
        net.set_params(second)
        net.train(1, 16, 1e-3, seed=4)
        return net.get_params()

    idle = calls()
    stop = threading.Event()

    def hold():
        pending = []
        while not stop.is_set():
            torch.cuda._sleep(20_000_000)
            e = torch.cuda.Event()
            e.record()
            pending.append(e)
            if len(pending) > 3:
                pending.pop(0).synchronize()

    t = threading.Thread(target=hold)
    t.start()
    try:
        busy = [calls() for _ in range(5)]
    finally:
        stop.set()
        t.join()
        torch.cuda.synchronize()
    assert all(np.array_equal(idle, b) for b in busy)
