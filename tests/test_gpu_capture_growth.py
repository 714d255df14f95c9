"""The compaction's look-back words where a capture that grew the scratch was
never replayed."""
import numpy as np
import pytest
import torch

from helpers import blob_volume, mid_iso, to_cuda, u32


@pytest.mark.gpu
def test_words_of_a_capture_that_never_ran(oracle):
    """The look-back words grow inside a capture, whose memset has not run when
    the graph is dropped; the buffer they got held other words before."""
    from meshtrex_b200 import api
    a = blob_volume((136, 128, 136), np.uint8, seed=9)  # 68 x 64 x 68 blocks of edge 2: 73 tiles
    iso = mid_iso(a)
    ref = oracle.extract(a, 2, iso)
    small = blob_volume((16, 16, 16), np.uint8, seed=8)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        c = api.Context(0, stream)
        try:
            v0 = to_cuda(small)
            ex0 = api.AsyncExtractor(c, v0, 2, mid_iso(small), 20000, 40000)
            ex0.run()
            c.synchronize()
            # buffers of the size the words will take, every word "7 blocks up to and with this tile" of an epoch
            size = 8 * 73
            for epoch in range(4):
                words = np.full(73, (2 << 62) | (epoch << 32) | 7, np.uint64).view(np.uint8).reshape(1, 1, size)
                pc = api.push_constants((size, 1, 1), 8, 0.0)
                v, mm = api.upload_compute_min_max_mip(c, words, pc)
                c.synchronize()
                mm.free()
                api.free_volume(c, v)
            vol = to_cuda(a)
            ex = api.AsyncExtractor(c, vol, 2, iso, ref.n_vertices, ref.n_triangles)
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=stream, capture_error_mode="relaxed"):
                ex.run()
            del g
            for _ in range(2):
                ex.counters.fill_(-1)
                ex.run()
                c.synchronize()
                assert list(u32(ex.counters)[:5]) == [ref.n_vertices, 3 * ref.n_triangles, len(ref.ids), len(ref.ids), 0]
                np.testing.assert_array_equal(u32(ex.indices), ref.indices)
        finally:
            c.close()
