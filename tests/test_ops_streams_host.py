"""Devices as ops' workspaces take them: a torch.device, an index, a string, None -- whatever torch.cuda.current_stream does."""
import types

import pytest
import torch


@pytest.mark.parametrize("device,index", [(torch.device("cuda", 1), 1), (torch.device("cuda"), 0), ("cuda", 0), ("cuda:1", 1),
                                          (1, 1), (None, 0)])
def test_every_form_of_a_device_finds_its_stream(monkeypatch, device, index):
    from nanovllm import _C, ops

    def current_stream(dev=None):
        dev = torch.device("cuda", dev) if isinstance(dev, int) else torch.device(dev or "cuda")
        return types.SimpleNamespace(cuda_stream=7000 + (dev.index or 0))

    def raw(i):
        assert type(i) is int
        return 7000 + i
    monkeypatch.setattr(torch.cuda, "current_stream", current_stream)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", raw, raising=False)
    assert ops._stream_of(device) == 7000 + index
    # the two workspaces, one per device and stream
    lib = types.SimpleNamespace(b200_paged_decode_attn_workspace_size=lambda *a: 64, b200_prefill_workspace_size=lambda d: 32)
    monkeypatch.setattr(_C, "load", lambda: lib)
    for name in ("_decode_ws", "_decode_need", "_prefill_ws"):
        monkeypatch.setattr(ops, name, {})
    made = []
    for f in ("zeros", "empty"):
        monkeypatch.setattr(torch, f, lambda n, dtype=None, device=None: made.append((n, device)) or torch.ones(n, dtype=dtype))
    ops.decode_workspace(1, 8, 8, 128, device)
    ops.prefill_workspace(device, 128)
    assert made == [(64, device), (32, device)]
    assert list(ops._decode_ws) == [(device, 7000 + index)] and list(ops._prefill_ws) == [(device, 128, 7000 + index)]
