"""The ray queries of the transport kernel itself: runs of several times as many photons as the grid has threads, so
that the tail kernel gets only the last of them. The warp-cooperative query (rectangles of up to 100 cells, kept cells
flushed 128 at a time), the lane-by-lane walk of up to 4 cells and the BVH find the same hits: every tally and map is the
same bit for bit, over grids and media in which a segment covers one cell or dozens."""
import ctypes as C

import numpy as np
import pytest

from xmcml_b200 import _lib, api, scenes
from xmcml_b200 import structs as S

pytestmark = pytest.mark.gpu

SHAPE = dict(block_size=128, blocks_per_sm=1)  # 18,944 threads on 148 SMs


def _thin(sc, factor):
    """The scene with its scattering coefficients divided: longer segments."""
    for layer in sc.layers:
        layer.mus /= factor
    return sc


SCENES = {
    "heightfield": lambda: scenes.height_field_tissue(grid=128, n_rings=10, time_bins=5),
    "heightfield_long_segments": lambda: _thin(scenes.height_field_tissue(grid=128, n_rings=10, time_bins=5), 5.0),
    "ellipsoid": lambda: scenes.ellipsoid_target(subdiv=4, n_rings=10, time_bins=5),
    "ellipsoid_long_segments": lambda: _thin(scenes.ellipsoid_target(subdiv=5, n_rings=10, time_bins=5), 6.0),
}


def _whole_in_tail():
    v = (C.c_uint64 * 1)()
    _lib.load().xmc_debug_counts(v, 1)
    return v[0]


@pytest.mark.parametrize("name", list(SCENES))
def test_query_schemes_of_the_transport_kernel_agree(tmp_path, name):
    n = 100_000
    m = api.Model(*SCENES[name]().write(str(tmp_path), name))
    maps = name == "heightfield"
    before = _whole_in_tail()
    got = []
    for kw in (dict(), dict(lane_queries=True), dict(query_batch=1, grid_cell_tris=2), dict(query_batch=31, grid_cell_tris=2),
               dict(lane_queries=True, grid_cell_tris=32, query_batch=16), dict(grid_cell_tris=32, smem_nodes=-1)):
        t = api.Transport(m, roulette=True, scattering=maps, trajectories=maps, **SHAPE, **kw)
        led = t.run(n, seed=23)
        got.append((t.tallies(), t.maps(), led))
        t.close()
    assert _whole_in_tail() == before
    for tal, mp, led in got[1:]:
        for k in tal:
            assert np.array_equal(tal[k], got[0][0][k]), k
        for k in mp:
            assert np.array_equal(mp[k], got[0][1][k]), k
        for k in [x + "_fx" for x in S.LEDGER_TERMS] + ["steps", "n_detected", "n_plane_crossings"]:
            assert led[k] == got[0][2][k], k
    # the schemes did run: they look at different numbers of cells and nodes
    assert len({led["n_node_visits"] for _, _, led in got}) >= 4
    assert got[0][2]["n_triangle_tests"] > 0


@pytest.mark.parametrize("log", [0, 16])
def test_maps_of_the_transport_kernel_agree_with_the_replay(tmp_path, log):
    """The crossing log against the replay of every detected photon, in the transport kernel."""
    n = 100_000
    m = api.Model(*scenes.height_field_tissue(grid=65, n_rings=10, time_bins=5).write(str(tmp_path), "log"))
    before = _whole_in_tail()
    got = []
    for rows in (-1, log):
        t = api.Transport(m, roulette=True, scattering=True, trajectories=True, trajectory_log=rows, **SHAPE)
        led = t.run(n, seed=29)
        assert led["n_replay_mismatch"] == 0
        got.append((t.maps(), t.tallies()["det_count"], led["n_trajectory_replayed"]))
        t.close()
    assert got[1][2] < got[0][2] and (log == 0 or got[1][2] > 0)
    assert _whole_in_tail() - before <= 2  # the replays alone may be small
    for k in got[0][0]:
        assert np.array_equal(got[0][0][k], got[1][0][k]), k
    assert np.array_equal(got[0][1], got[1][1])
