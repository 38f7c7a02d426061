"""The clearance grid of meshes large enough that several host threads build it, against the ray query it saves: a
segment that it calls clear has no hit by the BVH search over the same device image."""
import ctypes as C

import numpy as np
import pytest

from xmcml_b200 import _lib, api, scenes

LARGE = {"heightfield": lambda: scenes.height_field_tissue(grid=257), "ellipsoid": lambda: scenes.ellipsoid_target(subdiv=6)}


def _query(info, r, tmax, flags):
    n = len(r)
    r = np.ascontiguousarray(r, dtype=np.float32)
    t, s = np.zeros(n, np.float32), np.zeros(n, np.int32)
    pf, pi = C.POINTER(C.c_float), C.POINTER(C.c_int)
    _lib.check(_lib.load().xmc_debug_nearest(C.byref(info), n, r.ctypes.data_as(pf), 0.0, tmax, t.ctypes.data_as(pf),
                                             s.ctypes.data_as(pi), None, flags))
    return t, s


@pytest.mark.parametrize("name", list(LARGE))
def test_clear_segments_of_a_large_mesh_have_no_hit(tmp_path, name):
    m = api.Model(*LARGE[name]().write(str(tmp_path), name))
    rng = np.random.default_rng(11)
    n = 100_000
    o = rng.uniform((-2.6, -2.6, -0.2), (2.6, 2.6, 4.0), (n, 3))
    o[: n // 3, 2] = rng.uniform(-0.06, 0.2, n // 3)
    d = rng.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    r = np.concatenate([o, d], 1)
    for tmax in (0.01, 0.3):
        clear, _ = _query(m.info, r, tmax, 4)
        _, surf = _query(m.info, r, tmax, 0)
        assert not np.any((clear == 1.0) & (surf >= 0))
        assert clear.mean() > 0.3 and (surf >= 0).any()
