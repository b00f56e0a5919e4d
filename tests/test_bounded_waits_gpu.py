"""The way out of the bounded waits of recurrence_umma_kernel and attn_split_kernel: where tiles stop coming, every role leaves in order, with
products behind it; the status word is set, the next call raises, and the one after it is right."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def _recurrence(V, lens):
    from nanovllm import ops
    g = torch.Generator(device="cuda").manual_seed(V)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    T, H, G, N = sum(lens), 4, 2, 128
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    q, k, v = rand(T, G * N).bfloat16(), (rand(T, G * N) * N ** -0.5).bfloat16(), rand(T, H * V).bfloat16()
    decay = 0.7 + 0.3 * torch.rand(H, device="cuda", generator=g)
    slots = torch.arange(len(lens), dtype=torch.int32, device="cuda")
    sp = ops.StepSpans(cu, cu, None, max(lens))
    return lambda: ops.linear_recurrence(q, k, v, sp, H, G, N, V, torch.zeros(len(lens), H, N, V, device="cuda"), slots, decay=decay)


def _attention(D, lens):
    from nanovllm import ops
    g = torch.Generator(device="cuda").manual_seed(D)
    rand = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    q, k, v = rand(sum(lens), 8, D), rand(sum(lens), 2, D), rand(sum(lens), 2, D)
    sp = ops.StepSpans(cu, cu, None, max(lens))
    return lambda: ops.attn_generic(q, k, v, sp, D ** -0.5, 2, D)


@pytest.mark.parametrize("make,size,lens,entry", [(_recurrence, 64, [700, 129, 400], "b200_linear_recurrence"), (_recurrence, 128, [500] * 40, "b200_linear_recurrence"),
                                                  (_attention, 128, [600, 300], "b200_attn_generic"), (_attention, 64, [700] * 12, "b200_attn_generic")])
def test_a_wait_that_runs_out_is_reported(monkeypatch, make, size, lens, entry):
    from nanovllm import _C, ops
    call, lib = make(size, lens), _C.load()
    want = call()
    torch.cuda.synchronize()
    ops.check_waits()
    impatient = SimpleNamespace(**{entry + "_step": lambda *a: getattr(lib, entry + "_bounded")(*a[:-1], 0, a[-1])})
    with monkeypatch.context() as m:
        m.setattr(_C, "load", lambda: impatient)
        first = call()
    torch.cuda.synchronize()
    with pytest.raises(_C.B200Error, match="ran out"):
        call()
    assert not torch.equal(first, want)                        # (some CTAs left before their work was done)
    assert torch.equal(call(), want)
    torch.cuda.synchronize()
    ops.check_waits()


@pytest.mark.parametrize("D,lens", [(128, [600, 300]), (64, [700] * 12)])     # (two CTAs to a row tile's keys, and one)
def test_attention_leaves_a_tile_unwritten(monkeypatch, D, lens):
    """A row tile whose products did not all come is not written, also where only a part of its keys is missing: every element is right or as it was."""
    from nanovllm import _C, ops
    call, lib = _attention(D, lens), _C.load()
    want = call()
    torch.cuda.synchronize()
    with monkeypatch.context() as m:
        empty = torch.empty
        m.setattr(torch, "empty", lambda *a, **kw: empty(*a, **kw).fill_(7.0))
        m.setattr(_C, "load", lambda: SimpleNamespace(b200_attn_generic_step=lambda *a: lib.b200_attn_generic_bounded(*a[:-1], 0, a[-1])))
        got = call()
    torch.cuda.synchronize()
    with pytest.raises(_C.B200Error, match="ran out"):
        call()
    assert bool(((got == want) | (got == 7.0)).all()) and bool((got == 7.0).any())
