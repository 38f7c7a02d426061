"""The clearance grid against the ray query it saves: a segment that the grid calls clear has no hit by the
BVH search over the same device image. Short and long segments, inside and around the meshes, towards
surfaces and along them, from points on the voxels' and the bounds' edges."""
import ctypes as C

import numpy as np
import pytest

from xmcml_b200 import _lib, api, scenes


def _query(info, r, tmax, flags):
    lib = _lib.load()
    n = len(r)
    r = np.ascontiguousarray(r, dtype=np.float32)
    t, s = np.zeros(n, np.float32), np.zeros(n, np.int32)
    pf, pi = C.POINTER(C.c_float), C.POINTER(C.c_int)
    _lib.check(lib.xmc_debug_nearest(C.byref(info), n, r.ctypes.data_as(pf), 0.0, tmax, t.ctypes.data_as(pf),
                                     s.ctypes.data_as(pi), None, flags))
    return t, s


def _steep():
    """A box-like closed mesh with vertical walls and a needle, beside a plane stack."""
    sc = scenes.planar(n_rings=2)
    v = np.array([[x, y, z] for z in (0.3, 0.8) for x, y in ((-1, -1), (1, -1), (1, 1), (-1, 1))], float)
    f = np.array([[0, 1, 2], [0, 2, 3], [4, 5, 6], [4, 6, 7], [0, 1, 5], [0, 5, 4], [1, 2, 6], [1, 6, 5], [2, 3, 7], [2, 7, 6],
                  [3, 0, 4], [3, 4, 7]], np.int32)
    needle = np.array([[2.0, 2.0, 0.2], [2.001, 2.0, 0.9], [2.0, 2.001, 0.9]]), np.array([[0, 1, 2]], np.int32)
    sc.surfaces += [(v, f), needle]
    return sc


SCENES = {
    "ellipsoid": lambda: scenes.ellipsoid_target(subdiv=4),
    "heightfield": lambda: scenes.height_field_tissue(grid=65),
    "heightfield_coarse": lambda: scenes.height_field_tissue(grid=9, amp=0.04),
    "steep": _steep,
    "planar": lambda: scenes.planar(),
}


@pytest.mark.parametrize("tmax", [0.003, 0.05, 0.4, 3.0])
@pytest.mark.parametrize("name", list(SCENES))
def test_clear_segments_have_no_hit(tmp_path, name, tmax):
    m = api.Model(*SCENES[name]().write(str(tmp_path), name))
    rng = np.random.default_rng(len(name) * 100 + int(tmax * 1000))
    n = 60_000
    o = rng.uniform((-2.6, -2.6, -0.2), (2.6, 2.6, 4.0), (n, 3))
    o[: n // 4, 2] = rng.uniform(-0.06, 0.2, n // 4)                    # the height fields' depths
    o[n // 4: n // 2, :2] *= 0.4                                        # about the ellipsoid's axis
    o[::7] = np.round(o[::7], 2)                                        # coordinates that many edges share
    d = rng.standard_normal((n, 3))
    d[::5, 2] *= 0.02                                                   # along the layers
    d[::11, :2] *= 1e-3                                                 # straight down and up
    d /= np.linalg.norm(d, axis=1)[:, None]
    r = np.concatenate([o, d], 1)
    clear, _ = _query(m.info, r, tmax, 4)
    _, surf = _query(m.info, r, tmax, 0)
    assert not np.any((clear == 1.0) & (surf >= 0))
    if name == "planar":
        assert not clear.any()  # no small triangles: no grid
    elif tmax < 0.1:
        assert clear.mean() > 0.1 and (surf >= 0).any()
