"""The compaction where a CTA takes one, two, three and four tiles (592 CTAs on a
device of 148 SMs; tiles of 4096 blocks, 1024 in the entry point that allocates
nothing), twice in one context, and with a tile withheld between good calls: ids
and ranks against the oracle's."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import to_cuda, u32

pytestmark = pytest.mark.gpu


def _volume(gx, gy, seed):
    """Blocks of edge 2, about a fifth of them active at 127.5."""
    rng = np.random.default_rng(seed)
    a = np.where(rng.random((2, 2 * gy, 2 * gx)) < 0.02, 200, 50).astype(np.uint8)
    return a


def _check(c, a, voxels, want):
    from meshtrex_b200 import api
    pc = api.push_constants((a.shape[2], a.shape[1], a.shape[0]), 2, 127.0)
    mm = api.compute_min_max_mip(c, api.wrap_volume(voxels), pc)
    f = api.filter_active_blocks(c, mm, pc)
    n = api.read_active_block_count(c, f)
    assert n == len(want)
    np.testing.assert_array_equal(u32(f.ids()), want)
    total = int(f.out.totalBlocks)
    rank = u32(api.device_view(f.out.blockRankBuffer.ptr, (total,), torch.int32))
    ref = np.full(total, 0xffffffff, np.uint32)
    ref[want] = np.arange(len(want), dtype=np.uint32)
    np.testing.assert_array_equal(rank, ref)
    return mm, f


@pytest.mark.parametrize("gx,gy", [(4096, 592), (4096, 593), (4096, 1184), (4097, 1185), (4093, 2371)])
def test_tiles_per_cta(oracle, gx, gy):
    from meshtrex_b200 import _lib as L
    from meshtrex_b200 import api
    a = _volume(gx, gy, gx + gy)
    want = oracle.compact(oracle.minmax_halo(a, 2), oracle.U8, 127.0)
    voxels = to_cuda(a)
    c = api.Context(0)
    try:
        for _ in range(2):
            mm, f = _check(c, a, voxels, want)
            nb = int(f.out.totalBlocks)
            ids = torch.full((nb,), -1, dtype=torch.int32, device="cuda")
            rank = torch.full((nb,), -7, dtype=torch.int32, device="cuda")
            words = torch.full((8,), -1, dtype=torch.int32, device="cuda")
            c.synchronize()
            rc = L.lib().mtx_filter_active_blocks_noalloc(
                C.c_void_p(mm.out.minMaxImage.ptr), nb, L.DTYPE_U8, 127.0, C.c_void_p(ids.data_ptr()),
                C.c_void_p(rank.data_ptr()), C.c_void_p(words.data_ptr()), C.c_void_p(words.data_ptr() + 16),
                C.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert rc == 0
            torch.cuda.synchronize()
            assert int(words[0]) == len(want) and int(words[4]) == 0
            np.testing.assert_array_equal(u32(ids[:len(want)]), want)
            assert torch.equal(rank, api.device_view(f.out.blockRankBuffer.ptr, (nb,), torch.int32))
            f.free()
            mm.free()
    finally:
        c.close()


def test_withheld_tile_among_several_a_cta(oracle):
    from meshtrex_b200 import _lib as L
    from meshtrex_b200 import api
    a = _volume(4096, 1300, 5)
    want = oracle.compact(oracle.minmax_halo(a, 2), oracle.U8, 127.0)
    voxels = to_cuda(a)
    c = api.Context(0)
    try:
        _check(c, a, voxels, want)
        pc = api.push_constants((a.shape[2], a.shape[1], a.shape[0]), 2, 127.0)
        mm = api.compute_min_max_mip(c, api.wrap_volume(voxels), pc)
        c.set_waits(max_polls=4096, withhold=1)
        with pytest.raises(L.MtxError):
            f = api.filter_active_blocks(c, mm, pc)
            api.read_active_block_count(c, f)
        c.set_waits()
        _check(c, a, voxels, want)  # the next epoch started all the same
    finally:
        c.close()
