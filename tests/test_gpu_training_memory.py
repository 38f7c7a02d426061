"""A network's training buffers are allocated when it is made: its first training call takes no device memory of any
size, so a network that could be made does not fail there."""
import numpy as np
import pytest

from xmcml_b200 import surrogate as SG

pytestmark = pytest.mark.gpu


def _net():
    m = SG.MLP(15, 1000, 256, 4, max_rows=512)
    m.set_params(SG.he_uniform(np.random.default_rng(0), 15, 256, 4, 1000))
    return m


def _data(n):
    rng = np.random.default_rng(1)
    return rng.standard_normal((n, 15)).astype(np.float32), rng.standard_normal((n, 1000)).astype(np.float32)


@pytest.mark.parametrize("call", ["gradients", "train"])
def test_first_training_call_allocates_next_to_nothing(call):
    import torch

    def free_before_the_first_call(m):
        if call == "train":
            m.set_dataset(*_data(600))
        free = torch.cuda.mem_get_info()[0]
        if call == "train":
            m.train(1, batch=512)
        else:
            m.gradients(*_data(512))
        return free

    warm, m = _net(), _net()
    free_before_the_first_call(warm)  # loads the kernels
    before = free_before_the_first_call(m)
    taken = before - torch.cuda.mem_get_info()[0]
    m.close()
    warm.close()
    assert taken <= 8 << 20  # the recorded graph of a step; the partial sums alone are 71 MB
