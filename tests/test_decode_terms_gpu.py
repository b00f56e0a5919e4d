"""Paged decode attention keeps its probabilities in two 16-bit terms: what is left of the error is the rounding of the result,
whatever the number of CTAs; infinite values stay infinite."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(H, G, D, lens, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    need = [-(-n // 16) for n in lens]
    order = torch.randperm(sum(need), generator=g).to(torch.int32)
    table = torch.full((len(lens), max(need)), -1, dtype=torch.int32)
    at = 0
    for b, n in enumerate(need):
        table[b, :n] = order[at:at + n]
        at += n
    k, v = (torch.randn(sum(need), 16, G * D, generator=g).to(dtype) for _ in range(2))
    return torch.randn(len(lens), H, D, generator=g).to(dtype), k, v, table


def _want(q, k, v, table, lens, H, G, D):
    out = []
    for b, n in enumerate(lens):
        kk, vv = (c[table[b, :-(-n // 16)].long()].reshape(-1, G, D)[:n].double().repeat_interleave(H // G, 1) for c in (k, v))
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[b].double(), kk) * D ** -0.5, 1)
        out.append(torch.einsum("hn,nhd->hd", p, vv).reshape(-1))
    return torch.stack(out)


@pytest.mark.parametrize("ctas", [0, 1, 64, 148])
@pytest.mark.parametrize("H,G,D,lens", [(16, 8, 128, [1500]), (32, 8, 64, [700, 33]), (8, 2, 128, [257, 1, 16]), (8, 1, 64, [90])])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_the_result_is_the_rounded_one(H, G, D, lens, dtype, ctas):
    from nanovllm import ops
    q, k, v, table = _case(H, G, D, lens, dtype, H + D)
    ctx = torch.tensor(lens, dtype=torch.int32)
    got = ops.paged_decode_attn(q.cuda(), k.cuda(), v.cuda(), table.cuda(), ctx.cuda(), D ** -0.5, G, num_ctas=ctas).cpu()
    want = _want(q, k, v, table, lens, H, G, D).to(dtype)
    # two terms hold a bf16 probability to 2^-17 (fp16: 2^-22): a result rounds to the other side about once in 2^8 times, a
    # few times as often where it is small against the values it sums. With one term it is every third
    share = 0.04 if dtype == torch.bfloat16 else 0.01
    assert float((got != want).float().mean()) < share, float((got != want).float().mean())


@pytest.mark.parametrize("ctas", [1, 148])
def test_infinite_values(ctas):
    from nanovllm import ops
    H, G, D, lens = 16, 8, 128, [200, 40]
    q, k, v, table = _case(H, G, D, lens, torch.bfloat16, 5)
    flat = v[table[0, 3]]
    flat[7, 5], flat[9, 200], flat[11, 300] = math.inf, -math.inf, math.nan
    v[table[0, 3]] = flat
    ctx = torch.tensor(lens, dtype=torch.int32)
    got = ops.paged_decode_attn(q.cuda(), k.cuda(), v.cuda(), table.cuda(), ctx.cuda(), D ** -0.5, G, num_ctas=ctas).cpu().double()
    want = _want(q, k, v, table, lens, H, G, D)
    fine = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    assert float((got - want)[fine].abs().max()) < 2e-2
