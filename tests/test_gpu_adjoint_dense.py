"""The adjoint on blocks with more cut edges than its shared memory holds
dL/diso terms for (a checkerboard cuts every edge) and on noise, at every kind
of block edge: dL/dfield against the oracle's FP64 adjoint, and
dL/diso bit for bit in the order the kernels state -- each lane over its rows,
axis by axis, the lanes by a butterfly, the blocks in rank order in double."""
import numpy as np
import pytest
import torch

from helpers import to_cuda, u32

pytestmark = pytest.mark.gpu


def _diso(a, block, iso, ids, g):
    """dL/diso in float32 arithmetic in that order; vertices are numbered as the forward numbers them."""
    f32 = np.float32
    Z, Y, X = a.shape
    gx, gy = -(-X // block), -(-Y // block)
    inside = a <= f32(iso)
    rows = (block * block + 31) // 32
    parts, vid = [], 0
    for b in ids:
        lanes = [[[], [], []] for _ in range(32)]
        oz, oy, ox = (int(b) // (gx * gy)) * block, (int(b) // gx % gy) * block, (int(b) % gx) * block
        for q in range(block * block):
            z, y = oz + q // block, oy + q % block
            if z >= Z or y >= Y:
                continue
            for x in range(ox, min(ox + block, X)):
                for k, (dz, dy, dx) in enumerate(((0, 0, 1), (0, 1, 0), (1, 0, 0))):
                    w = (z + dz, y + dy, x + dx)
                    if w[0] >= Z or w[1] >= Y or w[2] >= X or inside[z, y, x] == inside[w]:
                        continue
                    den = f32(f32(a[w]) - f32(a[z, y, x]))
                    lanes[q // rows][k].append(f32(g[vid, k] / den) if abs(den) > f32(1e-5) else f32(0))
                    vid += 1
        s = np.zeros(32, f32)
        for l in range(32):
            for t in lanes[l][0] + lanes[l][1] + lanes[l][2]:
                s[l] = f32(s[l] + t)
        for o in (16, 8, 4, 2, 1):
            s = (s + s[np.arange(32) ^ o]).astype(f32)
        parts.append(s[0])
    assert vid == len(g) and len(parts) <= 1024
    d = np.zeros(1024, np.float64)
    d[: len(parts)] = parts
    h = 512
    while h:
        d[:h] += d[h:2 * h]
        h //= 2
    return f32(d[0])


@pytest.mark.parametrize("block", [2, 3, 4, 5, 6, 7, 8, 9, 16])
@pytest.mark.parametrize("kind", ["checkerboard", "noise"])
@pytest.mark.parametrize("mode", [0, 1])
def test_dense_blocks(ctx, oracle, block, kind, mode):
    from meshtrex_b200 import api
    rng = np.random.default_rng(block)
    shape = (block + 1, block + 2, 2 * block)
    a = rng.random(shape).astype(np.float32)
    if kind == "checkerboard":
        a = (0.4 * a + 0.6 * (np.indices(shape).sum(0) % 2)).astype(np.float32)
    iso = 0.5
    vol_t = to_cuda(a)  # the volume lives as long as the calls that read it
    vol = api.wrap_volume(vol_t)
    pc = api.push_constants(a.shape[::-1], block, iso)
    mm = api.compute_min_max_mip(ctx, vol, pc)
    f = api.filter_active_blocks(ctx, mm, pc)
    api.read_active_block_count(ctx, f)
    x = api.extract_meshlet_descriptors(ctx, mm, f, pc)
    g = rng.standard_normal((x.vertex_count, 3)).astype(np.float32)
    dfield, diso = api.extract_backward(ctx, vol, pc, f, x.out.meshletDescriptorBuffer.ptr, x.vertex_count,
                                        torch.from_numpy(g).cuda(), mode=mode)
    ctx.synchronize()
    ids = u32(f.ids())
    ref, _ = oracle.mc_adjoint(a, block, iso, ids, g)
    scale = max(np.abs(ref).max(), 1.0)  # a voxel's six terms round at most a dozen times, 6e-8 each
    np.testing.assert_allclose(dfield.cpu().numpy(), ref, rtol=1e-5, atol=2e-6 * scale)
    assert np.float32(diso.item()).view(np.uint32) == _diso(a, block, iso, ids, g).view(np.uint32)
    for o in (x, f, mm):
        o.free()
