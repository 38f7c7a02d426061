"""Arrays of the wrong shape are refused before a pointer to them reaches the library, which reads rows x n_in
(rows x n_out for targets) floats from it. The library is a stand-in that notes its calls: no GPU needed."""
import ctypes as C

import numpy as np
import pytest

from xmcml_b200 import surrogate as SG

N_IN, N_OUT = 15, 20


class _Library:
    def __init__(self):
        self.rows = []

    def _note(self, handle, x, rows, *_):
        self.rows.append(rows)
        return 0

    def _note_two(self, handle, x, t, rows, *_):
        self.rows.append(rows)
        return 0

    xmc_mlp_forward_rows = _note
    xmc_mlp_gradients = xmc_mlp_set_dataset = _note_two

    def xmc_mlp_destroy(self, handle):
        return 0


def _net(max_rows=256):
    m = SG.MLP.__new__(SG.MLP)
    m._lib, m._m = _Library(), C.c_void_p()
    m.n_in, m.n_out, m.max_rows, m.n_params = N_IN, N_OUT, max_rows, 1
    return m


@pytest.mark.parametrize("shape", [(N_IN,), (1, N_IN + 1), (5, N_IN - 1), (5, N_IN + 1), (128, N_IN - 1), (128, N_IN + 1),
                                   (300, N_IN - 1), (N_IN * 128,), (2, 5, N_IN), (2, 3, 5)])
def test_forward_refuses_other_shapes(shape):
    m = _net()
    with pytest.raises(ValueError):
        m.forward(np.zeros(shape, np.float32))
    assert m._lib.rows == []


@pytest.mark.parametrize("n", [0, 1, 5, 128, 300, 600])
def test_forward_takes_rows_of_n_in(n):
    m = _net()
    y, _ = m.forward(np.zeros((n, N_IN), np.float32))
    assert y.shape == (n, N_OUT) and sum(m._lib.rows) == n


def test_ensemble_mean_refuses_a_flat_query():
    s = SG.Surrogate.__new__(SG.Surrogate)
    s.members = [_net(), _net()]
    s.x_mean, s.x_std, s.y_mean, s.y_std = np.zeros(N_IN), np.ones(N_IN), np.zeros(N_OUT), np.ones(N_OUT)
    with pytest.raises(ValueError):
        s.mean_log10(np.zeros(N_IN))
    assert s.members[0]._lib.rows == []


@pytest.mark.parametrize("call", ["gradients", "set_dataset"])
@pytest.mark.parametrize("x,t", [((128, N_IN - 1), (128, N_OUT)), ((128, N_IN + 1), (128, N_OUT)), ((128, N_IN), (128, N_OUT - 1)),
                                 ((128, N_IN), (127, N_OUT)), ((128 * N_IN,), (128, N_OUT)), ((128, N_IN), (128,))])
def test_training_arrays_of_other_shapes_are_refused(call, x, t):
    m = _net()
    with pytest.raises(ValueError):
        getattr(m, call)(np.zeros(x, np.float32), np.zeros(t, np.float32))
    assert m._lib.rows == []


@pytest.mark.parametrize("call", ["gradients", "set_dataset"])
@pytest.mark.parametrize("t", [(128, N_OUT), (128, 4, 5), (200, N_OUT)])
def test_training_takes_targets_laid_out_as_rings_and_bins(call, t):
    m = _net()
    getattr(m, call)(np.zeros((128, N_IN), np.float32), np.zeros(t, np.float32))
    assert m._lib.rows == [128]
