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


def _stack():
    """Four height fields 0.2 mm apart: a walk among triangles wherever it goes, so that warps take rounds in which
    every lane takes the general step."""
    sc = scenes.height_field_tissue(grid=33, n_rings=10, time_bins=5)
    top, upper, lower, bottom = sc.surfaces
    sc.surfaces = [top, upper] + [scenes.height_field(0.25 + 0.2 * i, 0.09, 2.0, 33, 10.0) for i in range(4)] + [lower, bottom]
    a, l1, l2, l3 = sc.layers
    inner = [scenes.Layer(l2.n, l2.mua, l2.mus, l2.g, [s, s + 1]) for s in range(1, 6)]
    sc.layers = [scenes.Layer(a.n, 0, 0, 0, [0, 7]), scenes.Layer(l1.n, l1.mua, l1.mus, l1.g, [0, 1])] + inner + \
                [scenes.Layer(l3.n, l3.mua, l3.mus, l3.g, [6, 7])]
    return sc


@pytest.mark.parametrize("maps", [False, True])
def test_rounds_of_general_steps_change_nothing(tmp_path, maps):
    """The tail kernel has no such rounds: pieces of a run that it walks whole add up to the run."""
    m = api.Model(*_stack().write(str(tmp_path), "stack"))
    t = api.Transport(m, roulette=True, scattering=maps, trajectories=maps, **SHAPE)
    n, piece = 40_000, 10_000
    before = _whole_in_tail()
    led = t.run(n, seed=31)
    whole, maps_whole = t.tallies(), t.maps()
    assert _whole_in_tail() == before
    steps, total, maps_total = 0, None, None
    for first in range(0, n, piece):
        steps += t.run(piece, seed=31, first_photon=first)["steps"]
        tal, mp = t.tallies(), t.maps()
        total = tal if total is None else {k: total[k] + tal[k] for k in tal}
        maps_total = mp if maps_total is None else {k: maps_total[k] + mp[k] for k in mp}
    assert _whole_in_tail() - before >= n // piece  # (and replays)
    t.close()
    assert steps == led["steps"] and led["n_detected"] > 100
    for k in whole:
        assert np.array_equal(whole[k], total[k]), k
    for k in maps_whole:
        assert np.array_equal(maps_whole[k], maps_total[k]), k
