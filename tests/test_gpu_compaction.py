"""The compaction at the edges of its tiles (4096 blocks, rounds of 64 a warp,
two blocks a lane), its look-back words kept between launches of one context,
and the count scan's words zeroed by the count pass: ids and ranks against the
oracle's, in one context over sizes that grow and shrink, and a captured call
replayed on new voxels."""
import numpy as np
import pytest
import torch

from helpers import blob_volume, mid_iso, to_cuda, u32

pytestmark = pytest.mark.gpu

# (z, y, x) at block edge 2: 1, 63, 64, 65, 4095, 4096, 4097, 12289 and 3 blocks
SHAPES = [(2, 2, 2), (2, 14, 18), (4, 8, 16), (2, 10, 26), (6, 42, 130), (2, 32, 512), (2, 34, 482), (2, 2, 24578),
          (2, 2, 6)]


def test_compaction_over_sizes_in_one_context(oracle):
    from meshtrex_b200 import api
    c = api.Context(0)
    try:
        for shape in SHAPES + SHAPES[::-1]:
            a = blob_volume(shape, np.uint8, seed=sum(shape))
            iso = mid_iso(a)
            pc = api.push_constants((shape[2], shape[1], shape[0]), 2, iso)
            mm = api.compute_min_max_mip(c, api.wrap_volume(to_cuda(a)), pc)
            f = api.filter_active_blocks(c, mm, pc)
            n = api.read_active_block_count(c, f)
            ref = oracle.compact(oracle.minmax_halo(a, 2), oracle.U8, iso)
            assert n == len(ref), shape
            np.testing.assert_array_equal(u32(f.ids()), ref)
            total = int(f.out.totalBlocks)
            rank = u32(api.device_view(f.out.blockRankBuffer.ptr, (total,), torch.int32))
            want = np.full(total, 0xffffffff, np.uint32)
            want[ref] = np.arange(len(ref), dtype=np.uint32)
            np.testing.assert_array_equal(rank, want)
            f.free()
            mm.free()
    finally:
        c.close()


def test_captured_call_replayed_on_new_voxels(oracle):
    from meshtrex_b200 import api
    vols = [blob_volume((68, 66, 64), np.uint8, seed=s) for s in (1, 2, 3)]
    iso = mid_iso(vols[0])
    refs = [oracle.extract(a, 4, iso) for a in vols]
    cap_v, cap_t = max(r.n_vertices for r in refs), max(r.n_triangles for r in refs)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        c = api.Context(0, stream)
        vol = to_cuda(vols[0])
        ex = api.AsyncExtractor(c, vol, 4, iso, cap_v, cap_t)
        ex.run()
        c.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            ex.run()
        for k in (1, 2, 0, 2):
            vol.copy_(to_cuda(vols[k]))
            g.replay()
            if k == 2:
                ex.run()  # an eager call between replays
            c.synchronize()
            r = refs[k]
            assert list(u32(ex.counters)[:5]) == [r.n_vertices, 3 * r.n_triangles, len(r.ids), len(r.ids), 0]
            np.testing.assert_array_equal(u32(ex.indices)[:r.n_triangles], r.indices)
            np.testing.assert_array_equal(ex.vertices.cpu().numpy()[:r.n_vertices].view(np.uint32),
                                          r.xyz.view(np.uint32))
        del g
        c.close()
