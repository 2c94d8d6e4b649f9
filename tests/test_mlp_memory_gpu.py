"""A closed proposal network leaves no device memory behind."""
import numpy as np
import pytest

from brian_b200._lib import MLPHandle

pytestmark = pytest.mark.gpu


def test_handles_give_their_memory_back(gpu_table):
    import torch
    X = np.zeros((128, 64), np.float32)

    def use():
        h = MLPHandle()
        h.forward(X)
        h.close()

    use()
    free = torch.cuda.mem_get_info()[0]
    for _ in range(600):
        use()
    # the device hands out 2 MB at a time: 600 times the smallest buffer a
    # handle has (its bias gradients, 8 KB) would be two of them
    assert free - torch.cuda.mem_get_info()[0] < 2 << 20
