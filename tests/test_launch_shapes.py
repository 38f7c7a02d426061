"""The launch shapes that the autotuner times: both query schemes with the same shapes and the same numbers of
waiting lanes, everything else as the caller's options have it."""
import ctypes as C

from xmcml_b200 import _lib, api
from xmcml_b200 import structs as S


def test_both_query_schemes_are_tuned_alike():
    lib = _lib.load()
    base = api.options(roulette=True, scattering=True, chance=0.2, beam_radius=0.3, grid_cell_tris=8)
    n = lib.xmc_debug_launch_shapes(C.byref(base), None, 0)
    out = (S.XmcOptions * n)()
    assert lib.xmc_debug_launch_shapes(C.byref(base), out, n) == n
    shapes = {True: [], False: []}
    for o in out:
        lane = bool(o.flags & S.XMC_LANE_QUERIES)
        shapes[lane].append((o.block_size, o.photons_per_chunk, o.query_batch))
        assert o.flags & ~S.XMC_LANE_QUERIES == base.flags and (o.roulette_chance, o.beam_radius) == (0.2, 0.3)
        assert o.grid_cell_tris == 8 and o.blocks_per_sm == 0
    assert sorted(shapes[True]) == sorted(shapes[False]) and len(set(shapes[True])) == n // 2
    assert {q for _, _, q in shapes[True]} == {8, 12, 16}
