"""The batch kernel and its tail kernel against each other: a run of fewer photons than the grid has threads is
walked by the tail kernel alone, with a grid of one warp per SM the same run goes through both, and the
integer tallies are the same bit for bit. Instances at the edges of what a batch accepts."""
import numpy as np
import pytest

from xmcml_b200 import batch as XB
from xmcml_b200 import structs as S

pytestmark = pytest.mark.gpu


def _instances(photons):
    mua = [[0.3, 0.05, 0.02], [0.0, 0.01, 0.005], [5.0, 0.2, 0.1], [0.1, 0.1, 0.1], [1e-4, 1e-4, 1.0], [30.0, 30.0, 30.0]]
    mus = [[10.0, 20.0, 15.0], [40.0, 5.0, 20.0], [1.0, 2.0, 3.0], [10.0, 10.0, 10.0], [5.0, 60.0, 10.0], [0.0, 1.0, 2.0]]
    g = [[0.8, 0.9, 0.85], [0.0, -0.5, 0.7], [0.95, 0.99, 0.0], [0.9, 0.9, 0.9], [-0.9, 0.0, 0.5], [0.0, 0.0, 0.0]]
    n = [[1.4, 1.4, 1.37], [1.0, 1.6, 1.2], [1.4, 1.3, 1.5], [1.33, 1.33, 1.33], [1.5, 1.0, 1.5], [1.4, 1.4, 1.4]]
    th = [[0.1, 1.0, 50.0], [1e-4, 0.5, 2.0], [0.01, 0.01, 0.01], [1e-3, 1e4, 1.0], [0.2, 1e-5, 3.0], [1.0, 1.0, 1.0]]
    return XB.make_instances(mua, mus, g, n, th, photons, np.arange(6) + 40, [0.0, 0.3, 0.0, 1.0, 0.0, 0.2],
                             [1.0, 1.3, 1.0, 1.0, 1.5, 1.0], [1.0, 1.0, 1.4, 1.0, 1.0, 1.0])


@pytest.mark.parametrize("photons", [1, 33, 3000])
@pytest.mark.parametrize("spec", [dict(), dict(min_weight=0.0, max_steps_per_photon=3000), dict(min_weight=0.4),
                                  dict(max_steps_per_photon=17)])
@pytest.mark.parametrize("scheme", [0, 1])
def test_tail_and_batch_kernels_agree(photons, spec, scheme):
    inst = _instances(photons)
    got = []
    for small in (False, True):
        b = XB.Batch(n_rings=17, n_time=5, max_instances=6, **spec)
        if small:
            b.set_tuning(block_size=32, blocks_per_sm=1, photons_per_chunk=32, tally_scheme=scheme)
        out = b.run(inst, allow_budget=True)
        got.append((b.tallies(), out))
        b.close()
    for k in got[0][0]:
        assert np.array_equal(got[0][0][k], got[1][0][k]), k
    for k, _ in S.BatchResult._fields_:
        assert np.array_equal(got[0][1][k], got[1][1][k]), k
    led = got[0][0]["ledger"]
    assert np.all(led[:, 0] == photons) and np.all(led[:, 8:12].sum(1) == photons)


def test_long_walks_are_handed_over_and_rows_keep_the_callers_order():
    """Photons of more than 4,000 steps, instances that are started in another order than the caller's."""
    mua = [[1.0], [0.005], [0.3], [0.002]]
    inst = XB.make_instances(mua, [[10.0], [40.0], [20.0], [60.0]], [[0.8]] * 4, [[1.4]] * 4, [[50.0]] * 4, 6000, [1, 2, 3, 4])
    got = []
    for shape in (None, dict(block_size=32, blocks_per_sm=1), dict(block_size=64, blocks_per_sm=2, tally_scheme=0)):
        b = XB.Batch(n_layers=1, n_rings=10, n_time=3, max_instances=4)
        if shape:
            b.set_tuning(photons_per_chunk=64, **shape)
        b.run(inst)
        got.append(b.tallies())
        b.close()
    for other in got[1:]:
        for k in got[0]:
            assert np.array_equal(got[0][k], other[k]), k
    steps = got[0]["ledger"][:, 1] / 6000.0
    assert steps[0] < steps[2] < steps[1] < steps[3]
    for k in range(4):  # each row is its own instance's run
        b = XB.Batch(n_layers=1, n_rings=10, n_time=3, max_instances=1)
        b.run(inst.subset([k]))
        one = b.tallies()
        b.close()
        for key in one:
            assert np.array_equal(one[key][0], got[0][key][k]), (k, key)
