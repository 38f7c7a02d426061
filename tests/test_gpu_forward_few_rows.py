"""The fused forward pass with few rows (one tile per CTA, and one output chunk per CTA while the SMs suffice)
gives the rows that the same rows get inside a large batch, bit for bit; at the edges of both rules."""
import numpy as np
import pytest

from xmcml_b200 import surrogate as SG

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,n_hidden,n_out", [(256, 4, 1000), (128, 2, 36), (256, 1, 4), (256, 3, 2052)])
def test_few_rows_equal_the_large_batch(hidden, n_hidden, n_out):
    rng = np.random.default_rng(n_out)
    big = 128 * 300
    m = SG.MLP(15, n_out, hidden, n_hidden, max_rows=big)
    m.set_params(SG.he_uniform(rng, 15, hidden, n_hidden, n_out))
    x = rng.standard_normal((big, 15)).astype(np.float32)
    whole, _ = m.forward(x)  # 300 tiles: two slots per CTA
    chunks = (n_out + 255) // 256
    for tiles in {1, 2, 148 // chunks, 148 // chunks + 1, 148, 149}:
        for rows in {128 * tiles, 128 * tiles - 127, 128 * tiles - 1}:
            y, _ = m.forward(x[:rows])
            assert y.shape == (rows, n_out) and np.array_equal(y, whole[:rows]), (tiles, rows)
    m.close()
