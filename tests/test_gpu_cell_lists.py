"""The count and emit passes' cell lists at their edges, against the oracle bit
for bit: blocks whose every cell is listed (noise: full 32-cell steps, job and
vertex queues that wrap, 5 triangles a cell), blocks of one cell, lists of 31-33
cells, cells at the volume's high faces (voxels that own a vertex but start no
cell), dimensions of 1 and 2, and every kind of block edge: compile-time and
run-time, lists handed over (B <= 8) and inside bits handed over (B > 8)."""
import numpy as np
import pytest
import torch

from helpers import to_cuda, u32

pytestmark = pytest.mark.gpu


def _volume(kind, shape, dtype, rng):
    if kind == "noise":
        f = rng.random(shape)
    elif kind == "spikes":
        f = np.zeros(shape)
        for k in range(3):
            f[tuple(rng.integers(0, s) for s in shape)] = 0.9
        f[-1, -1, -1] = f[-1, 0, 0] = f[0, -1, 0] = f[0, 0, -1] = 0.8
    else:  # a plane through the block: about one row of cells a slice
        z, y, x = np.meshgrid(*[np.arange(s) / max(s, 2) for s in shape], indexing="ij")
        f = 0.3 * x + 0.3 * y + 0.4 * z + 0.01 * rng.random(shape)
    return (f * 255).astype(np.uint8) if dtype == np.uint8 else (f * 65535).astype(np.uint16) if dtype == np.uint16 \
        else f.astype(np.float32)


# (z, y, x): x aligned to 16 bytes for the tile path, odd for the plain loads
CASES = [(B, dt, kind, shape)
         for B, dt in ((2, np.uint8), (3, np.uint16), (4, np.float32), (5, np.uint8), (7, np.uint16), (8, np.uint8),
                       (8, np.uint16), (8, np.float32), (9, np.float32), (13, np.uint8), (16, np.uint16), (16, np.float32))
         for kind in ("noise", "spikes", "plane")
         for shape in ((2 * B + 1, B + 2, 16 * ((2 * B + 15) // 16)), (B, 2 * B - 1, 2 * B + 3))]
CASES += [(8, np.uint16, "noise", s) for s in ((1, 19, 24), (9, 1, 16), (11, 13, 1), (2, 2, 2), (9, 9, 9))]


@pytest.mark.parametrize("block,dtype,kind,shape", CASES)
def test_lists_match_oracle(ctx, oracle, block, dtype, kind, shape):
    from meshtrex_b200 import _lib as L
    from meshtrex_b200 import api
    a = _volume(kind, shape, dtype, np.random.default_rng(sum(shape) + block))
    iso = {np.uint8: 120.0, np.uint16: 30000.0, np.float32: 0.45}[dtype]
    ref = oracle.extract(a, block, iso)
    vol = to_cuda(a)
    for staging in (L.STAGING_AUTO, L.STAGING_LDG):
        m = api.extract(vol, block, iso, ctx=ctx, options=api.extract_options(staging=staging))
        np.testing.assert_array_equal(u32(m.active_ids), ref.ids)
        np.testing.assert_array_equal(m.vertices.cpu().numpy().view(np.uint32), ref.xyz.view(np.uint32))
        np.testing.assert_array_equal(u32(m.indices), ref.indices)


@pytest.mark.parametrize("block", [3, 8, 16])
def test_lists_with_normals_match_oracle(ctx, oracle, block):
    from meshtrex_b200 import _lib as L
    from meshtrex_b200 import api
    a = _volume("noise", (block + 3, 2 * block - 1, 2 * block + 5), np.uint16, np.random.default_rng(block))
    ref = oracle.extract(a, block, 30000.0, frame=oracle.FRAME_NDC, want_normals=True)
    m = api.extract(to_cuda(a), block, 30000.0, ctx=ctx,
                    options=api.extract_options(vertex_format=L.VERTEX_DATA, frame=L.FRAME_NDC, normals=True))
    v = m.vertices.cpu().numpy()
    np.testing.assert_array_equal(v[:, :3].copy().view(np.uint32), ref.xyz.view(np.uint32))
    np.testing.assert_array_equal(v[:, 4:7].copy().view(np.uint32), ref.normals.view(np.uint32))
    np.testing.assert_array_equal(u32(m.indices), ref.indices)
