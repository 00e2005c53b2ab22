"""Parameters and gradients of one network read by several threads at a time:
each call's values are its own."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import femgpu  # noqa: E402


def test_concurrent_readers():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    net = femgpu.UNet(seed=4)
    rng = np.random.default_rng(0)
    net.loss_grad(rng.standard_normal((1, 9, 9, 9, 2)).astype(np.float32),
                  rng.standard_normal((1, 9, 9, 9)).astype(np.float32))
    want = {"get_params": net.get_params(), "get_grads": net.get_grads()}
    wrong = []

    def read(name):
        for _ in range(200):
            if not np.array_equal(getattr(net, name)(), want[name]):
                wrong.append(name)

    threads = [threading.Thread(target=read, args=(name,)) for name in ("get_params", "get_grads") * 2]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
