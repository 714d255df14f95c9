"""The leaf min/max pass for any block edge and row alignment (and for uint8
volumes of every layout) against the oracle's (B+1)^3 block min/max, bit for
bit.  Shapes sit at the edges of its work split: strips of exactly a whole
number of blocks and one voxel more or less, rows of one voxel, rows shifted
by 1-3 bytes, volumes whose first and last words reach past the buffer
(a base address that is not word-aligned), runs of one slab, partial slabs,
and block edges with and without a compile-time form."""
import numpy as np
import pytest
import torch

from helpers import TORCH, blob_volume, mid_iso, u32

pytestmark = pytest.mark.gpu

CASES = [
    # shape (z, y, x), dtype, block edge, elements before the volume in its buffer, z-chunk (0: default)
    ((20, 19, 64), np.uint8, 3, 0, 0),     # aligned rows, word-aligned strips of four blocks
    ((20, 19, 123), np.uint8, 3, 0, 0),    # odd rows
    ((13, 17, 124), np.uint8, 3, 1, 1),    # aligned pitch, unaligned base; runs of one slab
    ((11, 9, 125), np.uint8, 4, 3, 0),     # unaligned rows and base
    ((19, 23, 257), np.uint8, 8, 0, 2),    # three strips
    ((24, 24, 256), np.uint8, 8, 0, 0),    # 16-byte rows: the default path of uint8
    ((33, 35, 130), np.uint8, 16, 2, 0),
    ((9, 8, 1), np.uint8, 2, 1, 0),        # rows of one voxel
    ((16, 21, 41), np.uint8, 5, 0, 0),     # run-time edge, aligned by strips of four blocks or not at all
    ((23, 14, 127), np.uint16, 8, 1, 0),
    ((17, 18, 128), np.uint16, 8, 1, 0),   # even rows from an odd element
    ((25, 26, 255), np.uint16, 4, 0, 3),
    ((31, 20, 130), np.uint16, 3, 0, 0),   # word-aligned rows, strips of an even number of blocks
    ((29, 30, 113), np.uint16, 16, 3, 0),
    ((15, 16, 77), np.uint16, 7, 0, 0),
    ((18, 17, 64), np.float32, 8, 1, 0),   # float32 rows off the 16-byte grid
    ((21, 33, 65), np.float32, 16, 0, 0),  # one strip of three blocks and one voxel more
    ((14, 13, 63), np.float32, 3, 2, 2),
    ((12, 11, 250), np.float32, 4, 0, 0),
    ((20, 22, 100), np.float32, 11, 0, 0),
]


@pytest.mark.parametrize("shape,dtype,block,offset,zchunk", CASES)
def test_rows_leaf_matches_oracle(ctx, oracle, shape, dtype, block, offset, zchunk):
    from meshtrex_b200 import api
    a = blob_volume(shape, dtype, seed=sum(shape) * 7 + block)
    n = a.size
    buf = torch.zeros(n + offset, dtype=torch.uint8 if dtype == np.uint8 else torch.int16
                      if dtype == np.uint16 else torch.float32, device="cuda")
    buf[offset:] = torch.from_numpy(a.reshape(-1).view(np.int16) if dtype == np.uint16 else a.reshape(-1)).cuda()
    vol = buf.view(TORCH[np.dtype(dtype)])[offset:].view(shape)
    pc = api.push_constants((shape[2], shape[1], shape[0]), block, mid_iso(a))
    ctx.set_tuning(minmax_zchunk=zchunk)
    try:
        mm = api.compute_min_max_mip(ctx, api.wrap_volume(vol), pc)
        ctx.synchronize()
        leaf = oracle.minmax_halo(a, block)
        np.testing.assert_array_equal(u32(mm.all_levels()), oracle.pyramid(leaf, oracle.block_grid(a.shape, block)))
        mm.free()
    finally:
        ctx.set_tuning()


@pytest.mark.parametrize("block,offset", [(7, 0), (8, 1), (3, 0)])
def test_rows_leaf_keys_of_nan_and_infinities(ctx, block, offset):
    """A NaN of positive sign counts as -0.0, so that it does not take its block
    out of every isovalue's range; one of negative sign and the infinities keep
    their place in the order of the keys."""
    from meshtrex_b200 import api
    rng = np.random.default_rng(5)
    a = rng.standard_normal((2 * block + 1, block + 3, 3 * block + 2)).astype(np.float32)
    r = rng.random(a.shape)
    for lo, v in ((.0, np.float32(np.nan)), (.01, -np.float32(np.nan)), (.02, np.inf), (.03, -np.inf), (.04, -0.0)):
        a[(r >= lo) & (r < lo + .01)] = v
    buf = torch.zeros(a.size + offset, dtype=torch.float32, device="cuda")
    buf[offset:] = torch.from_numpy(a.reshape(-1)).cuda()
    mm = api.compute_min_max_mip(ctx, api.wrap_volume(buf[offset:].view(a.shape)),
                                 api.push_constants(a.shape[::-1], block, 0.0))
    got = u32(mm.level(0))
    mm.free()
    bits = a.view(np.uint32)
    keys = np.where(bits >> 31, ~bits, bits | 0x80000000)
    keys = np.where(keys > 0xff800000, np.uint32(0x7fffffff), keys)
    for z, y, x in np.ndindex(got.shape[:3]):
        s = keys[z * block:(z + 1) * block + 1, y * block:(y + 1) * block + 1, x * block:(x + 1) * block + 1]
        assert (got[z, y, x, 0], got[z, y, x, 1]) == (s.min(), s.max())
