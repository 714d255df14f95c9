"""The octree's tiles: CTAs with one step, with several tiles of one step, and
with tiles of 2 x 2 steps (from 592 of them on a device of 148 SMs), with ragged
last tiles and levels thinner than a tile, twice in one context: every level
against the oracle's."""
import numpy as np
import pytest

from helpers import mid_iso, to_cuda, u32

pytestmark = pytest.mark.gpu

# block grids (z, y, x) of block edge 2
GRIDS = [(1, 1, 2), (9, 17, 33), (60, 161, 161), (67, 161, 481), (1, 1501, 3201)]


@pytest.mark.parametrize("grid", GRIDS)
def test_octree_levels(oracle, grid):
    from meshtrex_b200 import api
    shape = tuple(2 * n for n in grid)
    a = np.random.default_rng(sum(grid)).integers(0, 256, shape, dtype=np.uint8)
    want = oracle.pyramid(oracle.minmax_halo(a, 2), oracle.block_grid(a.shape, 2))
    c = api.Context(0)
    try:
        voxels = to_cuda(a)
        vol = api.wrap_volume(voxels)
        pc = api.push_constants((shape[2], shape[1], shape[0]), 2, mid_iso(a[:2, :2, :2]))
        for _ in range(2):  # the second launch starts from the counter the first one left
            mm = api.compute_min_max_mip(c, vol, pc)
            np.testing.assert_array_equal(u32(mm.all_levels()), want)
            mm.free()
    finally:
        c.close()
