"""xmc_run_noalloc builds a clearance grid only for runs that pay for it: the call of a model that exceeds its scratch,
which ends after the host image is built and before the GPU is touched, leaves the count of built grids as it is
with few photons and raises it with many."""
import ctypes as C

import numpy as np

from xmcml_b200 import _lib, api, scenes
from xmcml_b200 import structs as S


def _grids_built(lib):
    v = (C.c_uint64 * 2)()
    assert lib.xmc_debug_counts(v, 2) >= 2
    return v[1]


def test_short_runs_build_no_clearance_grid(tmp_path):
    lib = _lib.load()
    m = api.Model(*scenes.height_field_tissue(photons=1).write(str(tmp_path), "big"))
    before = _grids_built(lib)
    opts, dummy = api.options(), C.c_void_p(1)
    for n, grids in ((10, 0), (39_999, 0), (40_000, 1)):
        assert lib.xmc_run_noalloc(C.byref(m.info), C.byref(opts), 1, 0, n, dummy, dummy, dummy, dummy, None) == S.XMC_ERR_RANGE
        assert _grids_built(lib) == before + grids
    f, i = np.zeros(1, np.float32), np.zeros(1, np.int32)
    pf, pi = C.POINTER(C.c_float), C.POINTER(C.c_int)
    _lib.check(lib.xmc_debug_nearest(C.byref(m.info), 0, f.ctypes.data_as(pf), 0.0, 1.0, f.ctypes.data_as(pf),
                                     i.ctypes.data_as(pi), None, 4))
    assert _grids_built(lib) == before + 2
