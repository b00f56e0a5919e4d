"""ops.paged_decode_attn_fp8 with heads of 64, whose tiles are taken two at a time (csrc/decode_attn_fp8.cu): lengths around one, two and three
tiles (16 tokens for 8 kv heads, 128 for one pair), alone and split over CTAs, against fp32 attention over the de-quantised cache."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,G,lens", [
    (16, 8, [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 64, 65, 300]),
    (8, 4, [30, 33, 63, 64, 65, 97, 129]),
    (4, 2, [127, 128, 129, 255, 256, 257, 700, 0, 5]),
    (32, 8, [1000]),
])
def test_against_fp32(H, G, lens):
    from nanovllm import ops
    g = torch.Generator(device="cuda").manual_seed(H + len(lens))
    D, bs, B = 64, 16, len(lens)
    need = [-(-n // bs) for n in lens]
    order = torch.randperm(sum(need) + 1, device="cuda", generator=g).to(torch.int32)
    tables = torch.full((B, max(need)), -1, dtype=torch.int32, device="cuda")
    k, v = (torch.randn(sum(need) + 1, bs, G * D, device="cuda", generator=g).to(torch.float8_e4m3fn) for _ in range(2))
    q = torch.randn(B, H, D, device="cuda", generator=g).half()
    at = 0
    for i, n in enumerate(need):
        tables[i, :n] = order[at:at + n]
        at += n
    got = ops.paged_decode_attn_fp8(q, k, v, tables, torch.tensor(lens, dtype=torch.int32, device="cuda"), D ** -0.5, G, 0.5, 2.0).view(B, H, D)
    for i, n in enumerate(lens):
        if n == 0:
            assert not got[i].any()
            continue
        kk, vv = (c[tables[i, :need[i]].long()].float().reshape(-1, G, D)[:n].repeat_interleave(H // G, 1) * s for c, s in ((k, 0.5), (v, 2.0)))
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[i].float(), kk) * D ** -0.5, -1)
        want = torch.einsum("hn,nhd->hd", p, vv)
        # weights and the result are rounded to f16
        assert float((got[i].float() - want).norm() / want.norm()) < 2e-3, n
