"""The native calls of ops' attention entry points (csrc/host_calls.cpp): what they take gives what ops' own way gives, bit for bit; what they
do not take is left to ops' own checks."""
import ctypes

import pytest
import torch


def test_nothing_but_cuda_tensors_and_numbers():
    from nanovllm import _C, ops
    calls, t = _C.calls(), torch.zeros(1, 16, 128, dtype=torch.bfloat16)
    never = lambda *a: pytest.fail("asked for a workspace")  # noqa: E731
    assert calls.decode(never, t, t, t, t, t, 1.0, 8, 0, 0.0, 0, 0, 0) is None            # CPU tensors
    assert calls.decode_fp8(never, t, t, t, t, t, 1.0, 8, 0, 1.0, 1.0) is None
    assert calls.prefill(None, t, t, t, t, t, None, 1, 1, 1.0, 8, 0.0, None, 0, 0, 0) is None
    assert calls.decode(never, t, t, t, t, t, "1", 8, 0, 0.0, 0, 0, 0) is None            # not numbers
    assert calls.decode(never, t, t, t, t, t, 1.0, 1 << 70, 0, 0.0, 0, 0, 0) is None
    assert calls.decode(never, 1, 2, 3, 4, 5, 1.0, 8, 0, 0.0, 0, 0, 0) is None            # not tensors
    assert calls.decode() is None and calls.prefill() is None
    with pytest.raises(RuntimeError, match="CUDA only"):
        ops.paged_decode_attn(t, t, t, t, t, 1.0, 8)


def test_without_the_module_ops_goes_its_own_way(monkeypatch, tmp_path, caplog):
    from nanovllm import _C, ops
    assert _C.calls() is not None
    t = torch.zeros(1, 16, 128, dtype=torch.bfloat16)
    _C.load()
    monkeypatch.setenv("B200ATTN_LIB", str(tmp_path / "libb200attn.so"))      # a library elsewhere, without native calls beside it
    for there in (None, "not a module"):
        if there:
            open(_C.calls_path(), "w").write(there)
        monkeypatch.setattr(_C, "_calls", None)
        caplog.clear()
        assert _C.calls() is None and _C.calls() is None and len(caplog.records) == 1
        with pytest.raises(RuntimeError, match="CUDA only"):
            ops.paged_decode_attn(t, t, t, t, t, 1.0, 8)
        with pytest.raises(RuntimeError, match="CUDA only"):
            ops.prefill_varlen_attn(t, t, t, t, t, 1, 1, 1.0, 8)
    monkeypatch.setattr(_C, "_calls", None)
    monkeypatch.setattr(_C, "_lib", None)                                     # and none at all
    assert _C.calls() is None
    with pytest.raises(RuntimeError, match="CUDA only"):
        ops.paged_decode_attn_fp8(t, t, t, t, t, 1.0, 8)


@pytest.mark.gpu
def test_without_the_module_the_answer_is_the_same(monkeypatch):
    from nanovllm import _C, ops
    q, k, v, tables, lens = _step()
    want = ops.paged_decode_attn(q, k, v, tables, lens, 0.125, 2)
    monkeypatch.setattr(_C, "_calls", False)
    assert torch.equal(ops.paged_decode_attn(q, k, v, tables, lens, 0.125, 2), want)


def _step(dtype=torch.bfloat16, fp8=False, B=3, H=8, G=2, D=64, bs=16):
    g = torch.Generator(device="cuda").manual_seed(B)
    q = torch.randn(B, H + 2, D, device="cuda", generator=g).to(dtype)[:, :H]             # a token-strided view
    k, v = (torch.randn(40, bs, G * D, device="cuda", generator=g).to(dtype) for _ in range(2))
    if fp8:
        k, v = k.to(torch.float8_e4m3fn), v.to(torch.float8_e4m3fn).view(torch.uint8)
    tables = torch.randperm(40, device="cuda", generator=g)[:B * 10].view(B, 10).to(torch.int32)
    return q, k, v, tables, torch.tensor([150, 1, 77], dtype=torch.int32, device="cuda")


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_decode_is_the_same_either_way(dtype):
    from nanovllm import _C, ops
    q, k, v, tables, lens = _step(dtype)
    for kw in ({}, dict(window=20, keep_first=3), dict(chunk=32), dict(softcap=5), dict(num_ctas=64)):
        got = ops.paged_decode_attn(q, k, v, tables, lens, 0.125, 2, **kw)
        want = ops.paged_decode_attn(q, k, v, tables, lens, 0.125, 2, out=torch.empty_like(got), **kw)
        assert torch.equal(got, want) and got.dtype == dtype and got.shape == (3, 512), kw
    k4 = k.view(40, 16, 2, 64)
    assert torch.equal(ops.paged_decode_attn(q, k4, v, tables, lens, 0.125, 2), ops.paged_decode_attn(q, k, v, tables, lens, 0.125, 2))
    q8, k8, v8 = _step(dtype, fp8=True)[:3]
    got = ops.paged_decode_attn_fp8(q8, k8, v8, tables, lens, 0.125, 2, 0.5, 2.0)
    assert torch.equal(got, ops.paged_decode_attn_fp8(q8, k8, v8, tables, lens, 0.125, 2, 0.5, 2.0, out=torch.empty_like(got)))
    with pytest.raises(TypeError):
        ops.paged_decode_attn(q, k, v, tables.long(), lens, 0.125, 2)
    with pytest.raises(ValueError):
        ops.paged_decode_attn(q, k[:, :, :64], v, tables, lens, 0.125, 2)
    with pytest.raises(TypeError):
        ops.paged_decode_attn(q.float(), k, v, tables, lens, 0.125, 2)
    with pytest.raises(TypeError):
        ops.paged_decode_attn_fp8(q8, k, v, tables, lens, 0.125, 2)
    with pytest.raises(_C.B200Error):
        ops.paged_decode_attn(q[:, :3], k, v, tables, lens, 0.125, 2)                     # 3 heads over 2


@pytest.mark.gpu
def test_prompts_are_the_same_either_way():
    from nanovllm import ops
    g = torch.Generator(device="cuda").manual_seed(1)
    T, H, G, D = 90, 4, 2, 64
    qkv = torch.randn(T, (H + 2 * G) * D, device="cuda", generator=g).bfloat16()
    q, k, v = (x.unflatten(1, (-1, D)) for x in qkv.split([H * D, G * D, G * D], dim=1))
    cu = torch.tensor([0, 33, 90], dtype=torch.int32, device="cuda")
    sink = torch.randn(H, device="cuda", generator=g)
    for kw in ({}, dict(sink=sink, softcap=20.0), dict(window=16, keep_first=2), dict(chunk=24), dict(workspace=None)):
        got = ops.prefill_varlen_attn(q, k, v, cu, cu, 57, 57, 0.125, G, **kw)
        assert torch.equal(got, ops.prefill_varlen_attn(q, k, v, cu, cu, 57, 57, 0.125, G, out=torch.empty_like(got), **kw)), kw
    one = ops.prefill_varlen_attn(q[:1], k[:1], v[:1], cu[:1].repeat(2) + torch.tensor([0, 1], dtype=torch.int32, device="cuda"),
                                  torch.tensor([0, 1], dtype=torch.int32, device="cuda"), 1, 1, 0.125, G)
    assert torch.allclose(one.view(H, D).float(), v[0].repeat_interleave(H // G, 0).float(), atol=1e-2)
    cache = torch.randn(12, 16, G * D, device="cuda", generator=g).bfloat16()
    table = torch.randperm(12, device="cuda", generator=g).view(2, 6).to(torch.int32)
    ck = torch.tensor([0, 60, 150], dtype=torch.int32, device="cuda")
    got = ops.prefill_varlen_attn(q, cache, cache, cu, ck, 57, 90, 0.125, G, block_tables=table)
    assert torch.equal(got, ops.prefill_varlen_attn(q, cache, cache, cu, ck, 57, 90, 0.125, G, block_tables=table, out=torch.empty_like(got)))
    with pytest.raises(TypeError):
        ops.prefill_varlen_attn(q, k, v, cu.long(), cu, 57, 57, 0.125, G)
    with pytest.raises(ValueError):
        ops.prefill_varlen_attn(q, k.transpose(0, 1).contiguous().transpose(0, 1), v, cu, cu, 57, 57, 0.125, G)


@pytest.mark.gpu
@pytest.mark.parametrize("transform", [lambda f, x: torch.vmap(f)(x[None]), lambda f, x: torch.func.grad(f)(x), lambda f, x: torch.func.jvp(f, (x,), (x,))],
                         ids=["vmap", "grad", "jvp"])
def test_wrapped_tensors_raise(transform):
    """torch.vmap and torch.func wrap what they pass on: torch.Tensor to Python, and without memory."""
    from nanovllm import ops
    q, k, v, tables, lens = _step()
    q8, k8, v8 = _step(fp8=True)[:3]
    cu = torch.tensor([0, 3], dtype=torch.int32, device="cuda")
    kv = torch.randn(3, 2, 64, device="cuda").bfloat16()
    calls = ((q, lambda x: ops.paged_decode_attn(x, k, v, tables, lens, 0.125, 2)),
             (q8, lambda x: ops.paged_decode_attn_fp8(x, k8, v8, tables, lens, 0.125, 2)),
             (q, lambda x: ops.prefill_varlen_attn(x, kv, kv, cu, cu, 3, 3, 0.125, 2)))
    for x, call in calls:
        want = call(x)                                         # (the workspaces are there)
        with pytest.raises(RuntimeError, match="storage"):
            transform(lambda y: call(y).sum(), x)              # noqa: B023
        assert torch.equal(call(x), want)


@pytest.mark.gpu
def test_numbers_are_what_ctypes_takes():
    from nanovllm import ops
    q, k, v, tables, lens = _step()
    with pytest.raises(ctypes.ArgumentError):
        ops.paged_decode_attn(q, k, v, tables, lens, 0.125, 2.0)
    with pytest.raises(ValueError):
        ops.paged_decode_attn(q, k, v, tables, lens, 0.125, 2, window=float("nan"))
    assert torch.equal(ops.paged_decode_attn(q, k, v, tables, lens, 1, 2, window=20.0), ops.paged_decode_attn(q, k, v, tables, lens, 1.0, 2, window=20))
