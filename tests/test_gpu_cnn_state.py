"""What a network keeps between calls (its device buffers, up to 256 MiB), and calls of
several threads on one network."""
import numpy as np
import pytest

from mantle_convection_lab_gb300 import api

pytestmark = pytest.mark.gpu

KEEP = 256 << 20


@pytest.mark.parametrize("batch, kept", [(4, True), (24, False)])
def test_kept_memory_is_bounded(batch, kept):
    import torch

    # activations of one sample: 8 + 5*32 + 3 channels of 160 x 160 FP32, 17.5 MB
    x = np.zeros((batch, api.GUESS_CIN, 160, 160), np.float32)
    net = api.Cnn(width=32, depth=6)
    net.forward(x[:1, :, :16, :16])   # the context and the kernels are loaded
    before = torch.cuda.mem_get_info()[0]
    net.forward(x)
    held = before - torch.cuda.mem_get_info()[0]
    assert held <= KEEP
    assert (held > batch * 8 << 20) == kept
    net.close()
    assert before - torch.cuda.mem_get_info()[0] <= 0


def test_calls_of_several_threads_do_not_mix():
    """Gradients, forward passes and training of one network at the same time: a
    training whose steps round to nothing leaves the parameters as they are, so every
    call gives what it gives alone, to the bit."""
    import threading

    r = np.random.default_rng(3)
    net = api.Cnn(width=32, depth=4, seed=1)
    net.set_params(0.1 * r.standard_normal(net.nparam))
    p = net.params()

    def data(b, h, w):
        return (r.standard_normal((b, api.GUESS_CIN, h, w)).astype(np.float32),
                r.standard_normal((b, api.GUESS_COUT, h, w)).astype(np.float32))

    small, large = data(1, 33, 17), data(6, 97, 130)   # partial sums of different sizes
    want = [net.gradient(*small), net.gradient(*large)]
    y = net.forward(large[0])
    wrong = []

    def check(k, d):
        for _ in range(15):
            loss, g = net.gradient(*d)
            if loss != want[k][0] or not np.array_equal(g, want[k][1]):
                wrong.append(k)

    def forward():
        for _ in range(15):
            if not np.array_equal(net.forward(large[0]), y):
                wrong.append("forward")

    jobs = [threading.Thread(target=check, args=(0, small)), threading.Thread(target=check, args=(1, large)),
            threading.Thread(target=forward),
            threading.Thread(target=lambda: net.train(*data(4, 64, 64), batch=2, iters=60, lr=1e-30))]
    for t in jobs:
        t.start()
    for t in jobs:
        t.join()
    assert not wrong, wrong
    np.testing.assert_array_equal(net.params(), p)
    net.close()
