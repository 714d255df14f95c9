"""How the count and emit passes share out blocks: more blocks than warps but
fewer than two rounds of them (B = 8, on a device of 148 SMs), CTAs of up to 16
warps for B > 8 whose blocks go round the CTAs, fewer blocks than CTAs, and
explicit warp counts: meshes against the oracle's, staged and in one call."""
import numpy as np
import pytest
import torch

from helpers import to_cuda, u32

pytestmark = pytest.mark.gpu


def _waves(n, dtype):
    """Every block of edge 8 or more is active at 100."""
    z, y, x = np.meshgrid(*(np.arange(k) for k in n), indexing="ij")
    a = 100.3 + 30 * (np.sin(x * 0.9) + np.sin(y * 0.35 + 1) * 0.4 + np.cos(z * 0.3) * 0.3)
    return a.astype(dtype)


@pytest.mark.parametrize("shape,block,dtype,warps", [
    ((145, 145, 145), 8, np.uint8, 0),     # 5832 blocks: one round of 4736 warps and part of another
    ((145, 153, 161), 8, np.float32, 0),   # odd rows
    ((210, 225, 224), 16, np.uint16, 0),   # 2744 blocks: one round of 14 warps an SM and part of another
    ((100, 127, 131), 9, np.uint8, 0),
    ((40, 33, 50), 16, np.float32, 0),     # fewer blocks than CTAs
    ((100, 90, 96), 12, np.uint16, 8),
    ((100, 90, 96), 16, np.uint8, 1),
])
def test_shares(oracle, shape, block, dtype, warps):
    from meshtrex_b200 import api
    a = _waves(shape, dtype)
    iso = 100.0
    ref = oracle.extract(a, block, iso)
    voxels = to_cuda(a)
    c = api.Context(0)
    try:
        if warps:
            c.set_tuning(extract_warps=warps)
        pc = api.push_constants((shape[2], shape[1], shape[0]), block, iso)
        mm = api.compute_min_max_mip(c, api.wrap_volume(voxels), pc)
        f = api.filter_active_blocks(c, mm, pc)
        assert api.read_active_block_count(c, f) == len(ref.ids)
        x = api.extract_meshlet_descriptors(c, mm, f, pc)
        assert (x.vertex_count, x.index_count) == (ref.n_vertices, 3 * ref.n_triangles)
        np.testing.assert_array_equal(u32(x.indices()).reshape(-1, 3), ref.indices)
        np.testing.assert_array_equal(x.vertices().cpu().numpy().view(np.uint32), ref.xyz.view(np.uint32))
        ex = api.AsyncExtractor(c, voxels, block, iso, ref.n_vertices, ref.n_triangles)
        ex.run()
        c.synchronize()
        np.testing.assert_array_equal(u32(ex.indices), ref.indices)
        np.testing.assert_array_equal(ex.vertices.cpu().numpy().view(np.uint32), ref.xyz.view(np.uint32))
    finally:
        c.close()
