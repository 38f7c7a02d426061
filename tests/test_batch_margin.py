"""The batch kernels take a step that ends between zlo and zhi of its layer for one that reaches no plane,
without the division that finds a plane's distance. This checks the rule against that division in FP32, with
4 ulp to spare for the device's approximate quotient, on steps that end near the planes."""
import numpy as np
import pytest

F = np.float32


@pytest.mark.parametrize("top,bottom", [(0.0, 0.05), (0.0, 1e-5), (0.1, 1.1), (1.1, 51.1), (0.3, 0.3001), (50.0, 1e4),
                                        (1e4, 1e4 + 1.0), (0.0, 1e6)])
def test_inside_the_margin_no_plane_is_reached(top, bottom):
    rng = np.random.default_rng(int(bottom * 7) + 1)
    n = 400_000
    zt, zb = F(top), F(bottom)
    zlo = (F(4e-6) * zb + zt).astype(F)
    zhi = (zb - F(4e-6) * zb).astype(F)
    pz = np.clip(rng.uniform(float(zt), float(zb), n).astype(F), zt, zb)
    pz[: n // 8], pz[n // 8: n // 4] = zt, zb
    dz = rng.uniform(-1, 1, n).astype(F)
    dz[n // 4: n // 2] *= F(1e-4)
    ahead = np.where(dz > 0, zb, zt)
    with np.errstate(divide="ignore", invalid="ignore", over="ignore"):
        near = ((ahead - pz) / dz).astype(F)
        step = (near * rng.uniform(1 - 1e-4, 1 + 1e-6, n)).astype(F)   # ends near the plane ahead
        step[::3] = rng.exponential(1.0, n).astype(F)[::3]
        step = np.where(np.isfinite(step) & (step >= 0), step, F(0.01))
        zn = (step.astype(np.float64) * dz.astype(np.float64) + pz.astype(np.float64)).astype(F)
        free = (zn > zlo) & (zn < zhi)
        tb = np.maximum(near, F(0.0))
        reaches = tb * F(1 - 4 * 2.0 ** -23) <= step
    assert not np.any(free & reaches)
    if bottom - top > 1e-3 * bottom:
        assert free.any()
