"""The tail kernel of a transport run against the transport kernel: a photon takes the same path whichever
of the two walks it, so the tallies of a run that uses both are, bit for bit, the sums over pieces of the run
that are small enough for the tail kernel to walk whole. Also the edges of that rule: one photon, as many
photons as the grid has threads, one more."""
import numpy as np
import pytest

from xmcml_b200 import api, scenes
from xmcml_b200 import structs as S

from helpers import rich_planar

pytestmark = pytest.mark.gpu

LEDGER = [k + "_fx" for k in S.LEDGER_TERMS] + ["photons_launched", "photons_terminated", "steps", "n_escaped_top",
                                               "n_escaped_bottom", "n_area", "n_cut", "n_roulette", "n_glass", "n_invalid",
                                               "n_detected", "absorbed_target_fx", "bias_gained_fx", "bias_lost_fx",
                                               "n_plane_crossings"]


def _biased():
    sc = scenes.planar(n_rings=20, time_bins=7, time_finish=40.0)
    sc.bias_target, sc.bias_factor = (0, 0, 2), 1.0
    sc.bias_integral_precision, sc.bias_table_precision = 16, 256
    return sc


SCENES = {
    "planar": (lambda: scenes.planar(n_rings=20, time_bins=7, time_finish=40.0), dict(roulette=True, area_kill=False)),
    "cover": (lambda: rich_planar(), dict(beam_radius=0.2)),
    "heightfield": (lambda: scenes.height_field_tissue(grid=33, n_rings=20, time_bins=7), dict()),
    "ellipsoid": (lambda: scenes.ellipsoid_target(subdiv=3, n_rings=20, time_bins=7), dict(roulette=True)),
    "biased": (_biased, dict()),
}


@pytest.mark.parametrize("maps", [False, True])
@pytest.mark.parametrize("name", list(SCENES))
def test_whole_run_equals_its_small_pieces(tmp_path, name, maps):
    make, kw = SCENES[name]
    xml, surf = make().write(str(tmp_path), name)
    m = api.Model(xml, surf)
    kw = dict(kw, block_size=32, blocks_per_sm=1)  # one warp per SM
    if maps and name != "ellipsoid":
        kw.update(scattering=True, trajectories=True, trajectory_log=64)  # short log: some photons are replayed
    t = api.Transport(m, **kw)
    threads = 32 * _sms()
    sizes = [1, threads, 31, threads - 5]
    led, pieces, maps_sum = [], None, None
    for i, n in enumerate(sizes):
        led.append(t.run(n, seed=9, first_photon=sum(sizes[:i])))
        tal, mp = t.tallies(), t.maps()
        pieces = tal if pieces is None else {k: pieces[k] + tal[k] for k in tal}
        maps_sum = mp if maps_sum is None else {k: maps_sum[k] + mp[k] for k in mp}
    whole = t.run(sum(sizes), seed=9)
    tal, mp = t.tallies(), t.maps()
    t.close()
    for k in tal:
        assert np.array_equal(tal[k], pieces[k]), k
    for k in mp:
        assert np.array_equal(mp[k], maps_sum[k]), k
    for k in LEDGER:
        assert whole[k] == sum(x[k] for x in led), k


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def test_one_more_photon_than_threads(tmp_path):
    """n = threads goes to the tail kernel whole, n = threads + 1 through both: they differ by the last
    photon's own run."""
    xml, surf = scenes.planar(n_rings=10).write(str(tmp_path), "edge")
    m = api.Model(xml, surf)
    t = api.Transport(m, block_size=32, blocks_per_sm=1, roulette=True)
    n = 32 * _sms()
    out = []
    for first, count in ((0, n), (n, 1), (0, n + 1)):
        t.run(count, seed=4, first_photon=first)
        out.append(t.tallies())
    t.close()
    for k in out[0]:
        assert np.array_equal(out[0][k] + out[1][k], out[2][k]), k


def test_step_budget_in_both_kernels(tmp_path):
    """Photons that reach the step budget end in the ledger's budget term in either kernel."""
    xml, surf = scenes.planar(n_rings=10).write(str(tmp_path), "budget")
    m = api.Model(xml, surf)
    t = api.Transport(m, block_size=32, blocks_per_sm=1, max_steps=37)
    n = 32 * _sms() + 77
    a = t.run(n, seed=4, allow_budget=True)
    b = [t.run(c, seed=4, first_photon=f, allow_budget=True) for f, c in ((0, n - 1000), (n - 1000, 1000))]
    t.close()
    assert a["n_budget"] > 0
    for k in LEDGER + ["n_budget"]:
        assert a[k] == sum(x[k] for x in b), k


def test_contexts_of_different_shared_memory_run_in_turn(tmp_path):
    """A context that stages much in shared memory still runs, through either kernel, after one was created that
    stages little."""
    big = api.Model(*scenes.height_field_tissue(grid=97, n_rings=20, time_bins=5).write(str(tmp_path), "big"))
    small = api.Model(*scenes.planar(n_rings=2).write(str(tmp_path), "small"))
    a = api.Transport(big)
    first = [a.run(n, seed=3)["absorbed_fx"] for n in (500, 90_000)]
    b = api.Transport(small)
    b.run(500)
    assert [a.run(n, seed=3)["absorbed_fx"] for n in (500, 90_000)] == first
    b.run(90_000)
    a.close()
    b.close()
