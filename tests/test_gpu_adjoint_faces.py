"""The adjoint where edges cross from one block into the next, against the
oracle's FP64 adjoint: spikes on block faces, edges and corners (so that a
voxel's terms come from several blocks, and some of those blocks are not
active), noise (every voxel has all its terms), odd and tiny volumes, both
modes, compile-time and run-time block edges."""
import numpy as np
import pytest
import torch

from helpers import to_cuda, u32

pytestmark = pytest.mark.gpu


def _field(kind, shape, block, rng):
    if kind == "noise":
        return rng.random(shape).astype(np.float32)
    f = 0.2 * rng.random(shape).astype(np.float32)
    for _ in range(12):  # voxels at or beside multiples of the block edge
        p = [min(s - 1, max(0, block * int(rng.integers(0, s // block + 1)) + int(rng.integers(-1, 2)))) for s in shape]
        f[tuple(p)] = 0.6 + 0.3 * rng.random()
    return f


@pytest.mark.parametrize("block", [2, 3, 4, 8, 11, 16])
@pytest.mark.parametrize("kind", ["spikes", "noise"])
@pytest.mark.parametrize("mode", [0, 1])
def test_adjoint_across_block_faces_matches_oracle(ctx, oracle, block, kind, mode):
    from meshtrex_b200 import api
    for k, shape in enumerate([(2 * block + 1, 3 * block, 2 * block + 3), (block, block + 1, 4 * block), (2, 1, block + 2)]):
        rng = np.random.default_rng(100 * block + k)
        a = _field(kind, shape, block, rng)
        iso = 0.5
        vol_t = to_cuda(a)
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
        ref, ref_iso = oracle.mc_adjoint(a, block, iso, u32(f.ids()), g)
        # a voxel's six terms round at most a dozen times in float32 (6e-8 each); terms cancel, so relative to
        # the largest gradient, which in a field of this range exceeds every term's partial sums
        scale = max(np.abs(ref).max(), 1.0)
        np.testing.assert_allclose(dfield.cpu().numpy(), ref, rtol=1e-5, atol=2e-6 * scale)
        assert abs(float(diso.item()) - ref_iso) <= 1e-5 * max(abs(ref_iso), scale)
        for o in (x, f, mm):
            o.free()
