"""The meshlet split's 32-triangle steps at their edges, against the oracle bit
for bit, on index lists made for it: blocks of 0, 1, 31, 32, 33, 64, 65 and 500
triangles, limits that cut inside a step, at its end and never, triangles that
repeat a vertex, ids that all hash near one another, and blocks of one vertex."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import u32

pytestmark = pytest.mark.gpu

TRIS = [0, 1, 31, 32, 33, 64, 65, 500, 32, 7, 126, 127]


def _indices(kind, rng):
    out = []
    for b, n in enumerate(TRIS):
        if kind == "strip":  # two new vertices every other triangle, as a surface has
            base = 1000 * b
            tri = base + np.arange(n)[:, None] // 2 + np.array([0, 1, 2])
        elif kind == "repeats":  # few ids: repeated corners inside a triangle and across steps
            tri = rng.integers(0, 40, (n, 3)) + 17 * b
        elif kind == "spread":  # every corner new
            tri = 3 * n * b + rng.permutation(3 * n).reshape(n, 3)
        elif kind == "stride":  # multiples of a power of two
            tri = rng.integers(0, 300, (n, 3)) * 4096
        else:
            tri = np.full((n, 3), 5 + b)
        out.append(tri)
    return np.concatenate(out).astype(np.uint32)


@pytest.mark.parametrize("limits", [(64, 126), (3, 1), (64, 1024), (5, 32), (64, 32), (64, 33), (33, 31), (9, 64)])
@pytest.mark.parametrize("kind", ["strip", "repeats", "spread", "stride", "one"])
def test_meshlet_steps_match_oracle(ctx, oracle, kind, limits):
    from meshtrex_b200 import _lib as L
    idx = _indices(kind, np.random.default_rng(7))
    nt = np.array(TRIS, np.uint32)
    desc = np.zeros((len(TRIS), 4), np.uint32)
    desc[:, 1] = 3 * np.concatenate([[0], np.cumsum(nt[:-1])])
    desc[:, 3] = nt
    nverts = int(idx.max()) + 1
    verts = torch.rand((nverts, 3), device="cuda")
    d_idx = torch.from_numpy(idx.view(np.int32)).cuda()
    d_desc = torch.from_numpy(desc.view(np.int32)).cuda()
    count = torch.tensor([nverts, 3 * len(idx), len(TRIS)], dtype=torch.int32, device="cuda")
    x = L.ExtractionOutput()
    for f, t in (("vertexBuffer", verts), ("indexBuffer", d_idx), ("meshletDescriptorBuffer", d_desc)):
        getattr(x, f).ptr, getattr(x, f).size = t.data_ptr(), t.numel() * 4
    x.meshletDescriptorCountBuffer.ptr, x.meshletDescriptorCountBuffer.size = count.data_ptr() + 8, 4
    x.meshletCount, x.vertexCount, x.indexCount, x.vertexStride = len(TRIS), nverts, 3 * len(idx), 12
    torch.cuda.synchronize()
    o = L.MeshletOutput()
    L.check(L.lib().mtx_build_meshlets(ctx.handle, C.byref(x), limits[0], limits[1], C.byref(o)), "mtx_build_meshlets",
            ctx.handle)
    from meshtrex_b200 import api
    got_d = u32(api.device_view(o.meshletDescriptorBuffer.ptr, (o.meshletCount, 4), torch.int32))
    got_v = u32(api.device_view(o.meshletVertexBuffer.ptr, (o.vertexCount,), torch.int32))
    got_i = u32(api.device_view(o.indexBuffer.ptr, (o.indexCount // 3, 3), torch.int32))
    want_d, want_v, want_i = oracle.meshlets(nt, idx, *limits)
    np.testing.assert_array_equal(got_d, want_d)
    np.testing.assert_array_equal(got_v, want_v)
    np.testing.assert_array_equal(got_i, want_i)
    L.lib().mtx_meshlet_output_free(ctx.handle, C.byref(o))
