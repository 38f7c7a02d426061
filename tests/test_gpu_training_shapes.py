"""Training kernels at the edges of their shapes: tile widths 64 to 256, output counts that are no multiple of 4
or of a tile, one to eight hidden layers, the smallest and larger batches; gradients against the FP64 oracle
with its BF16 roundings, and one Adam step of a minibatch against the gradients of the same rows."""
import ctypes as C

import numpy as np
import pytest

from oracle import mlp_ref as R
from xmcml_b200 import _lib
from xmcml_b200 import surrogate as SG

pytestmark = pytest.mark.gpu

SHAPES = [(15, 128, 1, 3, 128), (15, 128, 2, 301, 384), (7, 256, 3, 1000, 1024), (15, 256, 2, 1026, 2048),
          (64, 256, 1, 64, 4096), (15, 128, 8, 40, 256)]


def _net(n_in, hidden, n_hidden, n_out, rows, seed):
    rng = np.random.default_rng(seed)
    p = R.init_params(rng, n_in, hidden, n_hidden, n_out)
    m = SG.MLP(n_in, n_out, hidden, n_hidden, max_rows=rows)
    m.set_params(p)
    return m, p, rng


@pytest.mark.parametrize("n_in,hidden,n_hidden,n_out,rows", SHAPES)
def test_gradients(n_in, hidden, n_hidden, n_out, rows):
    m, p, rng = _net(n_in, hidden, n_hidden, n_out, rows, rows + n_out)
    x = rng.standard_normal((rows, n_in)).astype(np.float32)
    dims = dict(n_in=n_in, hidden=hidden, n_hidden=n_hidden, n_out=n_out)
    t = (R.forward(p, x, **dims) + rng.normal(0, 0.5, (rows, n_out))).astype(np.float32)
    g, loss = m.gradients(x, t)
    again, _ = m.gradients(x, t)
    m.close()
    gr, lr_ = R.gradients(p, x, t, **dims)
    assert np.array_equal(g, again)
    assert loss == pytest.approx(lr_, rel=1e-3)
    o = 0
    for i, (r, c) in enumerate(R.shapes(n_in, hidden, n_hidden, n_out)):
        for sz in (r * c, r):
            rel = np.linalg.norm(g[o:o + sz] - gr[o:o + sz]) / np.linalg.norm(gr[o:o + sz])
            o += sz
            assert rel < 1e-2, (i, sz, rel)  # BF16 flips through up to eight layers; 2e-3 through four


@pytest.mark.parametrize("n_in,hidden,n_hidden,n_out,rows", SHAPES)
def test_minibatch_step(n_in, hidden, n_hidden, n_out, rows):
    """Rows drawn by the counter generator, gradients as xmc_mlp_gradients gives them for those rows, Adam."""
    m, p, rng = _net(n_in, hidden, n_hidden, n_out, rows, rows)
    ds = 517
    x = rng.standard_normal((ds, n_in)).astype(np.float32)
    t = rng.standard_normal((ds, n_out)).astype(np.float32)
    seed = 0x1234_5678_9ABC
    key, out, src = (C.c_uint32 * 2)(seed & 0xFFFFFFFF, seed >> 32), (C.c_uint32 * 4)(), []
    for r in range(rows):
        _lib.load().xmc_philox4x32_10((C.c_uint32 * 4)(r, 1, 0x6D6C70, 0), key, out)
        src.append((out[0] * ds) >> 32)
    g, loss = m.gradients(x[src], t[src])
    m.set_dataset(x, t)
    losses, _ = m.train(1, batch=rows, lr=1e-3, seed=seed)
    got = m.get_params().astype(np.float64)
    m.set_dataset(x[:40], t[:40])  # another data set: the recorded step must not read the old one
    m.train(2, batch=rows, lr=1e-3, seed=seed)
    assert np.all(np.isfinite(m.get_params()))
    m.close()
    assert losses[0] == pytest.approx(loss, rel=1e-5)  # FP32 sums in another order
    g = g.astype(np.float64)
    want, _, _ = R.adam_step(p.astype(np.float64), g, np.zeros_like(g), np.zeros_like(g), 1, 1e-3)
    sure = np.abs(g) > 1e-5 * np.abs(g).max()  # eps and FP32 rounding of tiny moments aside
    assert np.max(np.abs(got - want)[sure]) < 2e-6 + 1e-3 * 1e-2
