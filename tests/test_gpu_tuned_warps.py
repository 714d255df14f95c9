"""The CTA sizes of the count and emit passes, read from a captured call's kernel
nodes: an untuned context and one tuned to the largest warp count that
mtx_autotune tries run the same CTAs at every block edge, and fewer warps, or
threads given with the call, are taken as they are."""
import numpy as np
import pytest
import torch

from helpers import blob_volume, mid_iso, to_cuda, u32

pytestmark = pytest.mark.gpu


def _cta_threads(graph):
    """{kernel name: threads a CTA} of a captured graph's kernels."""
    from cuda.bindings import driver as D
    raw = D.CUgraph(graph.raw_cuda_graph())
    err, _, n = D.cuGraphGetNodes(raw, 0)
    assert err == D.CUresult.CUDA_SUCCESS
    err, nodes, n = D.cuGraphGetNodes(raw, n)
    out = {}
    for node in nodes[:n]:
        err, kind = D.cuGraphNodeGetType(node)
        if kind != D.CUgraphNodeType.CU_GRAPH_NODE_TYPE_KERNEL:
            continue
        err, p = D.cuGraphKernelNodeGetParams(node)
        assert err == D.CUresult.CUDA_SUCCESS
        err, name = D.cuKernelGetName(p.kern) if int(p.kern) else D.cuFuncGetName(p.func)
        assert err == D.CUresult.CUDA_SUCCESS
        out[name.decode()] = p.blockDimX
    return out


def _sizes(a, block, ref, options=None, **tuning):
    from meshtrex_b200 import api
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        c = api.Context(0, stream)
        c.set_tuning(**tuning)
        vol = to_cuda(a)
        ex = api.AsyncExtractor(c, vol, block, mid_iso(a), ref.n_vertices, ref.n_triangles, options=options)
        ex.run()
        c.synchronize()
        np.testing.assert_array_equal(u32(ex.indices), ref.indices)
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g, stream=stream):
            ex.run()
        sizes = _cta_threads(g)
        del g
        c.close()
    count = [t for k, t in sizes.items() if "pmb_count_kernel" in k]
    emit = [t for k, t in sizes.items() if "pmb_emit_kernel" in k]
    assert len(count) == len(emit) == 1, sizes
    return count[0] // 32, emit[0] // 32


@pytest.mark.parametrize("block", [4, 8, 12, 16])
def test_tuned_warps(oracle, block):
    from meshtrex_b200 import api
    a = blob_volume((40, 36, 48), np.uint16, seed=2)
    ref = oracle.extract(a, block, mid_iso(a))
    own = _sizes(a, block, ref)
    assert min(own) >= 8 if block <= 8 else max(own) > 8
    assert _sizes(a, block, ref, extract_warps=8) == own
    assert _sizes(a, block, ref, extract_warps=4) == (4, 4)
    assert _sizes(a, block, ref, extract_warps=8, options=api.extract_options(threads=64)) == (2, 2)


@pytest.mark.parametrize("block", [4, 8, 16])
def test_capped_ctas_keep_their_size(oracle, block):
    """extractCtasPerSm leaves room on each SM: the CTAs it counts stay at four warps."""
    a = blob_volume((40, 36, 48), np.uint16, seed=2)
    ref = oracle.extract(a, block, mid_iso(a))
    assert _sizes(a, block, ref, extract_ctas_per_sm=2) == (4, 4)
    assert _sizes(a, block, ref, extract_ctas_per_sm=2, extract_warps=2) == (2, 2)
