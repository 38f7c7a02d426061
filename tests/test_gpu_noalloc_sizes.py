"""xmc_run_noalloc against xmc_create / xmc_run over the numbers of photons at which its ways change (one kernel or
both, with or without a clearance grid) and over models that leave room for all of its optional tables in the
scratch, for some or for hardly any: the same tallies and ledger bit for bit, and no device memory taken by a call."""
import ctypes as C

import numpy as np
import pytest

from xmcml_b200 import _lib, api, scenes
from xmcml_b200 import structs as S

pytestmark = pytest.mark.gpu

SCENES = {
    "planar": lambda: scenes.planar(n_rings=10, time_bins=3, time_finish=20.0),
    "heightfield": lambda: scenes.height_field_tissue(grid=64, n_rings=10, time_bins=3),
    "ellipsoid": lambda: scenes.ellipsoid_target(subdiv=4, n_rings=10, time_bins=3),
    "no_room_for_the_tail_list": lambda: scenes.height_field_tissue(grid=130, n_rings=10, time_bins=3),  # 1 MB left
    "no_room_for_the_clearance_grid": lambda: scenes.height_field_tissue(grid=138, n_rings=10, time_bins=3),  # 0.1 MB
}


@pytest.mark.parametrize("kw", [dict(roulette=True), dict(area_kill=False, roulette=True, beam_radius=0.2), dict(lane_queries=True)])
@pytest.mark.parametrize("name", list(SCENES))
def test_noalloc_equals_a_context_at_every_size(tmp_path, name, kw):
    import torch

    lib = _lib.load()
    m = api.Model(*SCENES[name]().write(str(tmp_path), name))
    opts = api.options(**kw)
    D, T, G = m.n_detectors, m.info.timeScaleSize, int(np.prod(m.grid_shape))
    bufs = [torch.full((k,), 7, dtype=torch.int64, device="cuda") for k in (G, 4 * D, 4 * D * T, 32)]
    t = api.Transport(m, opts)
    t.run(1)
    free = None
    for seed, n in enumerate((1, 20_000, 39_000, 60_000, 200_000)):
        st = lib.xmc_run_noalloc(C.byref(m.info), C.byref(opts), seed, 100 * seed, n, *[b.data_ptr() for b in bufs],
                                 torch.cuda.current_stream().cuda_stream)
        assert st == S.XMC_OK, _lib.last_error()
        led, tal = t.run(n, seed=seed, first_photon=100 * seed), t.tallies()
        absorption, det, bins, raw = [b.cpu().numpy().view(np.uint64) for b in bufs]
        assert np.array_equal(absorption, tal["absorption"]), n
        for k, what in enumerate(["weight", "count", "target", "weight2"]):
            assert np.array_equal(det.reshape(D, 4)[:, k], tal["det_" + what]), (n, what)
            assert np.array_equal(bins.reshape(D, T, 4)[:, :, k], tal["time_" + what]), (n, what)
        for k, slot in (("photons_launched", 0), ("photons_terminated", 1), ("steps", 2), ("n_detected", 11), ("absorbed_fx", 15)):
            assert int(raw[slot]) == led[k], (n, k)
        if free is not None:
            assert torch.cuda.mem_get_info()[0] == free, n
        free = torch.cuda.mem_get_info()[0]
    t.close()
