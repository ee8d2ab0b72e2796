"""What a network keeps between calls: its device buffers, up to 256 MiB."""
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
