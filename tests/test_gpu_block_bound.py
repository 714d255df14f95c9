"""More active blocks than mtx_mesh_buffers::maxActiveBlocks: the call reports
MTX_ERR_CAPACITY and the count it would need, writes no descriptor past the
bound (words behind a caller's buffer of exactly that many keep their values)
and leaves the other totals zero."""
import numpy as np
import pytest
import torch

from helpers import blob_volume, mid_iso, to_cuda, u32

pytestmark = pytest.mark.gpu

CAPACITY = 4  # MTX_ERR_CAPACITY


@pytest.mark.parametrize("shape,block,bound", [
    ((40, 40, 48), 8, lambda n: n // 2),   # bound and count in the scan's only tile of 1024
    ((40, 40, 48), 8, lambda n: 1),
    ((72, 64, 80), 4, lambda n: 1023),     # a tile short of one, two tiles or more by the count
    ((72, 64, 80), 4, lambda n: 1025),
    ((72, 64, 80), 4, lambda n: n - 1),
])
def test_nothing_is_written_past_the_block_bound(ctx, oracle, shape, block, bound):
    from meshtrex_b200 import _lib as L
    from meshtrex_b200 import api
    a = blob_volume(shape, np.uint8, seed=3)
    iso = mid_iso(a)
    ref = oracle.extract(a, block, iso)
    n = len(ref.ids)
    most = bound(n)
    assert 0 < most < n
    desc = torch.full((n + 2048, 4), 0x5a5a5a5a, dtype=torch.int32, device="cuda")
    ex = api.AsyncExtractor(ctx, to_cuda(a), block, iso, ref.n_vertices, ref.n_triangles, max_active_blocks=most)
    ex.bufs.meshlets = desc.data_ptr()
    ex.bufs.meshletCapacity = most
    ex.run()
    with pytest.raises(L.MtxError) as e:
        ctx.synchronize()
    assert e.value.status == CAPACITY
    assert bool((desc[most:] == 0x5a5a5a5a).all())
    assert list(u32(ex.counters)[:5]) == [0, 0, 0, n, CAPACITY]
    # with room for all of them the same buffers give the mesh
    ex.bufs.maxActiveBlocks = ex.bufs.meshletCapacity = n
    ex.run()
    ctx.synchronize()
    assert list(u32(ex.counters)[:5]) == [ref.n_vertices, 3 * ref.n_triangles, n, n, 0]
    np.testing.assert_array_equal(u32(ex.indices[: ref.n_triangles]), ref.indices)
    assert bool((desc[n:] == 0x5a5a5a5a).all())
