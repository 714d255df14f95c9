"""The accessors' copies where the context's device is not the current one: they
go through torch, whose copy between devices waits for both devices' streams,
and not through a copy on the current stream alone."""
import types

import pytest
import torch

from meshtrex_b200 import api


class _Lib:
    def __init__(self, calls):
        self.calls = calls

    def mtxpy_copy(self, *a):
        self.calls.append("copy")
        return 0


@pytest.mark.parametrize("device,way", [(0, "copy"), (1, "view")])
def test_accessors_copy_by_the_contexts_device(monkeypatch, device, way):
    calls = []
    empty = torch.empty
    monkeypatch.setattr(api.torch.cuda, "current_device", lambda: 0)
    monkeypatch.setattr(api, "_current_stream_ptr", lambda *a: 0)
    monkeypatch.setattr(api.L, "lib", lambda: _Lib(calls))
    monkeypatch.setattr(api.torch, "empty", lambda shape, dtype=None, device=None: empty(shape, dtype=dtype))

    def view(ptr, shape, dtype):
        calls.append("view")
        return torch.zeros(shape, dtype=dtype)

    monkeypatch.setattr(api, "device_view", view)
    ctx = types.SimpleNamespace(device=device, handle=None)
    buf = types.SimpleNamespace(ptr=4096, size=64)
    x = api.Extraction(ctx, types.SimpleNamespace(
        vertexStride=12, vertexCount=4, indexCount=6, meshletCount=1, vertexBuffer=buf, indexBuffer=buf,
        meshletDescriptorBuffer=buf, vertexCountBuffer=buf))
    f = api.Filtering(ctx, types.SimpleNamespace(activeBlockCount=3, compactedBlockIdBuffer=buf))
    m = api.MinMax(ctx, types.SimpleNamespace(minMaxImage=buf, levelExtent=[(2, 2, 2)], levelOffset=[0]))
    shapes = [tuple(t.shape) for t in (x.vertices(), x.indices(), x.meshlets(), x.counters(), f.ids(), m.level(0),
                                       m.all_levels())]
    assert shapes == [(4, 3), (2, 3), (1, 4), (3,), (3,), (2, 2, 2, 2), (8, 2)]
    assert calls == [way] * 7
