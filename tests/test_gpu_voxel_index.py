"""The free step's voxel index, made from the bits of the scaled coordinates, in both transport kernels: on grids of up to
4,096 partitions along an axis (XMC_LARGE_GRID), summed over blocks of voxels, it gives the coarse grid's tallies bit
for bit, and voxel (255, 255, 255), which the reference's byte indices exclude, is excluded exactly where it is."""
import numpy as np
import pytest

from xmcml_b200 import api, scenes

pytestmark = pytest.mark.gpu

SHAPE = dict(block_size=128, blocks_per_sm=1)
RUNS = [10_000, 100_000]  # the tail kernel alone; both kernels


def _run(tmp_path, name, sc, n, **kw):
    m = api.Model(*sc.write(str(tmp_path), name))
    t = api.Transport(m, **SHAPE, **kw)
    led = t.run(n, seed=33)
    a = t.tallies()["absorption"].reshape(m.grid_shape)
    t.close()
    return a, led


@pytest.mark.parametrize("n", RUNS)
@pytest.mark.parametrize("times", [(2, 2, 2), (4, 2, 4), (16, 1, 4), (1, 16, 8)])
def test_fine_grids_add_up_to_the_coarse_one(tmp_path, n, times):
    grid = (256, 3, 250)
    coarse, a = _run(tmp_path, "c", scenes.planar(n_rings=2, area_partitions=grid), n, roulette=True)
    fine_grid = tuple(p * k for p, k in zip(grid, times))
    fine, b = _run(tmp_path, "f", scenes.planar(n_rings=2, area_partitions=fine_grid), n, roulette=True, large_grid=True)
    x, y, z = times
    summed = fine.reshape(grid[0], x, grid[1], y, grid[2], z).sum(axis=(1, 3, 5))
    assert coarse.any() and np.array_equal(summed, coarse)
    # (not the steps: a point on a surface counts as inside Area within 1e-4 of a voxel, so a photon that leaves there
    # is lost one step later on the coarser grid)
    assert a["absorbed_fx"] == b["absorbed_fx"] and a["n_area"] == b["n_area"]


@pytest.mark.parametrize("n", RUNS)
def test_the_excluded_voxel_counts_as_outside(tmp_path, n):
    """An Area whose last voxel lies on the beam, 0.5 mm deep."""
    side, w = 10.24, 0.04
    sc = scenes.planar(n_rings=2, area_corner=(w - side - 0.02, w - side - 0.02, 0.5 + w - side), area_length=(side,) * 3,
                       area_partitions=(256, 256, 256))
    with_it, a = _run(tmp_path, "w", sc, n, roulette=True, area_kill=False, large_grid=True)
    without, b = _run(tmp_path, "o", sc, n, roulette=True, area_kill=False)
    last = int(with_it[255, 255, 255])
    assert last > 0 and without[255, 255, 255] == 0
    with_it[255, 255, 255] = 0
    assert np.array_equal(with_it, without)
    assert a["absorbed_fx"] - b["absorbed_fx"] == last == b["absorbed_outside_fx"] - a["absorbed_outside_fx"]
    assert a["steps"] == b["steps"] and a["n_escaped_top"] == b["n_escaped_top"]
