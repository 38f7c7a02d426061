"""Which runs the tail kernel walks whole: up to a share of the grid's threads that depends on the walk. At the line and
one photon past it the tallies are those of the run's pieces, bit for bit, and the library counts the runs
that went there."""
import ctypes as C

import numpy as np
import pytest

from xmcml_b200 import _lib, api, scenes

from helpers import rich_planar

pytestmark = pytest.mark.gpu


def _biased():
    sc = scenes.planar(n_rings=5)
    sc.bias_target, sc.bias_factor = (0, 0, 2), 1.0
    sc.bias_integral_precision, sc.bias_table_precision = 16, 256
    return sc


CASES = {
    "biased": (_biased, dict(), (1, 1)),
    "no_area_loss": (lambda: scenes.planar(n_rings=5), dict(roulette=True, area_kill=False), (4, 5)),
    "mesh": (lambda: scenes.ellipsoid_target(subdiv=3, n_rings=5, time_bins=2), dict(), (3, 5)),
    "mesh_no_area_loss": (lambda: scenes.height_field_tissue(grid=17, n_rings=5, time_bins=2), dict(area_kill=False), (4, 5)),
    "planes": (lambda: scenes.planar(n_rings=5), dict(roulette=True), (1, 3)),
    "glass": (lambda: rich_planar(), dict(), (1, 3)),
}


def _whole_in_tail():
    v = (C.c_uint64 * 1)()
    _lib.load().xmc_debug_counts(v, 1)
    return v[0]


@pytest.mark.parametrize("name", list(CASES))
def test_both_sides_of_the_line(tmp_path, name):
    import torch

    make, kw, (a, b) = CASES[name]
    m = api.Model(*make().write(str(tmp_path), name))
    t = api.Transport(m, block_size=64, blocks_per_sm=1, **kw)
    threads = 64 * torch.cuda.get_device_properties(0).multi_processor_count
    line = threads * a // b

    def run(first, n, whole):
        before = _whole_in_tail()
        t.run(n, seed=6, first_photon=first)
        assert _whole_in_tail() - before == (1 if whole else 0), (first, n)
        return t.tallies()

    at, past, last, half = run(0, line, True), run(0, line + 1, False), run(line, 1, True), run(0, line // 2, True)
    rest = run(line // 2, line - line // 2, True)
    t.close()
    for k in at:
        assert np.array_equal(at[k] + last[k], past[k]), k
        assert np.array_equal(half[k] + rest[k], at[k]), k
