"""The autotuners time the kernels whose shapes they choose: a sample of fewer photons than the grid has threads,
which a run would give to the tail kernel whole, goes through the main kernel while they do, and runs
afterwards take the tail kernel again."""
import ctypes as C

import numpy as np
import pytest

from xmcml_b200 import _lib, api, scenes
from xmcml_b200 import batch as XB

pytestmark = pytest.mark.gpu


def _whole_in_tail():
    v = (C.c_uint64 * 1)()
    assert _lib.load().xmc_debug_counts(v, 1) >= 1
    return v[0]


def test_transport_samples_go_through_the_transport_kernel(tmp_path):
    m = api.Model(*scenes.planar(n_rings=5).write(str(tmp_path), "t"))
    before = _whole_in_tail()
    best, ms = api.autotune(m, sample_photons=2_000, roulette=True)
    assert _whole_in_tail() == before and ms > 0
    t = api.Transport(m, best)
    t.run(2_000)
    assert _whole_in_tail() == before + 1
    t.close()


def test_batch_samples_go_through_the_batch_kernel():
    inst = XB.sample_instances(3, 3, budget=(2000, 2000))
    b = XB.Batch(n_rings=10, n_time=3, max_instances=3)
    b.run(inst)
    whole, before = b.tallies(), _whole_in_tail()
    best = b.autotune(inst, photons_cap=1000)
    assert _whole_in_tail() == before and best["ms"] > 0
    b.run(inst)
    assert _whole_in_tail() == before + 1
    again = b.tallies()
    b.close()
    for k in whole:
        assert np.array_equal(whole[k], again[k]), k
