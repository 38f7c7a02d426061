"""How many lanes of a warp wait for a general step, and the launch shapes that the autotuner times: query_batch as the
option has it for cooperative queries, but not below the number that is faster than every smaller one, and no part of
the lane-by-lane scheme, whatever a caller's options (or options kept from an earlier tuning) say."""
import ctypes as C

import pytest

from xmcml_b200 import _lib, api
from xmcml_b200 import structs as S


@pytest.mark.parametrize("batch,lanes", [(0, 12), (1, 12), (2, 12), (8, 12), (12, 12), (13, 13), (16, 16), (31, 31), (32, 32)])
def test_waiting_lanes(batch, lanes):
    lib = _lib.load()
    assert lib.xmc_debug_waiting_lanes(C.byref(api.options(query_batch=batch))) == lanes
    assert lib.xmc_debug_waiting_lanes(C.byref(api.options(query_batch=batch, lane_queries=True))) == 12


def test_shapes_that_are_timed():
    lib = _lib.load()
    base = api.options(roulette=True, scattering=True, chance=0.2, beam_radius=0.3, grid_cell_tris=8)
    n = lib.xmc_debug_launch_shapes(C.byref(base), None, 0)
    out = (S.XmcOptions * n)()
    assert lib.xmc_debug_launch_shapes(C.byref(base), out, n) == n
    seen = set()
    for o in out:
        lane = bool(o.flags & S.XMC_LANE_QUERIES)
        # what is timed is what a run with these options does
        seen.add((lane, o.block_size, o.photons_per_chunk, lib.xmc_debug_waiting_lanes(C.byref(o))))
        assert o.query_batch == lib.xmc_debug_waiting_lanes(C.byref(o))
        assert o.flags & ~S.XMC_LANE_QUERIES == base.flags and (o.roulette_chance, o.beam_radius) == (0.2, 0.3)
        assert o.grid_cell_tris == 8 and o.blocks_per_sm == 0
    assert len(seen) == n == 12
    assert {x[3] for x in seen if not x[0]} == {12, 16} and {x[3] for x in seen if x[0]} == {12}
