"""A photon's path does not depend on the kernel that walks it, nor on the order in which a launch starts and hands
over its photons: 1e7 photons through mesh scenes in two launch shapes, bit for bit. A sum of products that one
kernel rounds in another order than the other shows in fewer (with the order of every such sum changed, already
2e6 photons differ)."""
import numpy as np
import pytest

from xmcml_b200 import api, scenes
from xmcml_b200 import structs as S

pytestmark = pytest.mark.gpu

COUNTS = ["steps", "n_escaped_top", "n_escaped_bottom", "n_area", "n_cut", "n_roulette", "n_glass", "n_invalid", "n_detected"]


def _biased():
    sc = scenes.planar(n_rings=20, time_bins=7, time_finish=40.0)
    sc.bias_target, sc.bias_factor = (0, 0, 2), 1.0
    sc.bias_integral_precision, sc.bias_table_precision = 16, 256
    return sc


SCENES = {
    "heightfield": (lambda: scenes.height_field_tissue(grid=128, n_rings=20, time_bins=7), 10_000_000, dict()),
    "ellipsoid": (lambda: scenes.ellipsoid_target(subdiv=5, n_rings=20, time_bins=7), 10_000_000, dict()),
    "biased": (_biased, 1_000_000, dict()),
}


@pytest.mark.parametrize("name", list(SCENES))
def test_ten_million_photons_in_two_launch_shapes(tmp_path, name):
    make, n, kw = SCENES[name]
    m = api.Model(*make().write(str(tmp_path), name))
    got = []
    for shape in (dict(), dict(block_size=192, blocks_per_sm=1, photons_per_chunk=7, query_batch=5)):
        t = api.Transport(m, **kw, **shape)
        led = t.run(n, seed=21)
        got.append((led, t.tallies()))
        t.close()
    for k in got[0][1]:
        assert np.array_equal(got[0][1][k], got[1][1][k]), k
    for k in [x + "_fx" for x in S.LEDGER_TERMS] + COUNTS:
        assert got[0][0][k] == got[1][0][k], k
