"""The depths between which the batch kernels take a step for one that reaches no plane, from the compiled rule
(xmc_debug_free_depths): safe against the division that finds a plane's distance in FP32, with 4 ulp to spare for
the device's approximate quotient, and wide enough to be of use in layers given as practically semi-infinite."""
import ctypes as C

import numpy as np
import pytest

from xmcml_b200 import _lib

F = np.float32


def _depths(top, bottom, mfp):
    lo, hi = C.c_float(), C.c_float()
    _lib.load().xmc_debug_free_depths(top, bottom, mfp, C.byref(lo), C.byref(hi))
    return F(lo.value), F(hi.value)


LAYERS = [(0.0, 0.05), (0.0, 1e-5), (0.1, 1.1), (1.1, 51.1), (0.3, 0.3001), (50.0, 1e4), (1e4, 1e4 + 1.0), (0.0, 1e6), (0.0, 1e8),
          (0.7, 1e8), (0.3, np.inf)]


@pytest.mark.parametrize("mfp", [1e-3, 0.05, 1.0, 30.0, 1e5])
@pytest.mark.parametrize("top,bottom", LAYERS)
def test_inside_the_depths_no_plane_is_reached(top, bottom, mfp):
    rng = np.random.default_rng(int(min(bottom, 1e6) * 7) + int(1e3 * mfp))
    n = 400_000
    zt, zb = F(top), F(bottom)
    zlo, zhi = _depths(top, bottom, mfp)
    deep = min(float(zb), float(zt) + 40 * mfp)  # where the upper plane can be reached, and the lower one's neighbourhood
    pz = rng.uniform(float(zt), deep, n).astype(F)
    if np.isfinite(zb):
        pz[::2] = rng.uniform(max(float(zt), float(zb) - 40 * mfp), float(zb), n)[::2].astype(F)
    pz = np.clip(pz, zt, zb)
    pz[: n // 8] = zt
    dz = rng.uniform(-1, 1, n).astype(F)
    dz[n // 4: n // 2] *= F(1e-4)
    ahead = np.where(dz > 0, zb, zt)
    with np.errstate(divide="ignore", invalid="ignore", over="ignore"):
        near = ((ahead - pz) / dz).astype(F)
        step = (near * rng.uniform(1 - 1e-4, 1 + 1e-6, n)).astype(F)  # ends near the plane ahead
        step[::3] = (mfp * rng.exponential(1.0, n)).astype(F)[::3]
        longest = F(-np.log(2.0 ** -25) * mfp)
        step = np.where(np.isfinite(step) & (step >= 0) & (step <= longest), step, F(0.2 * mfp))
        zn = (step.astype(np.float64) * dz.astype(np.float64) + pz.astype(np.float64)).astype(F)
        free = (zn > zlo) & (zn < zhi)
        reaches = np.maximum(near, F(0.0)) * F(1 - 4 * 2.0 ** -23) <= step
    assert not np.any(free & reaches)


@pytest.mark.parametrize("top,bottom", [x for x in LAYERS if x[1] - x[0] >= 50])
@pytest.mark.parametrize("mfp", [0.01, 0.1, 1.0])
def test_steps_near_the_upper_plane_of_a_thick_layer_are_free(top, bottom, mfp):
    zlo, zhi = _depths(top, bottom, mfp)
    assert zlo <= F(top) * F(1 + 8e-6) + F(2e-4 * mfp)   # far below a mean free path from the plane
    assert zlo < F(top + 1.0) < zhi
    assert zhi >= F(bottom) * F(1 - 8e-6)
