"""Prompt attention on the tcgen05 kernel with capped scores around the range of its polynomial, at the edges of its row
and key tiles, with a sink, in both CTA layouts and with the keys split; and cached keys in blocks of every size the
kernel looks up at once. Against a 64-bit evaluation."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


@pytest.mark.parametrize("tiles", [0, 1, 2])
def test_more_sequences_than_the_ordered_list_holds(tiles):
    """300 sequences of 0 to 200 rows: past 256 the items come in the sequences' own order."""
    from nanovllm import _C, ops
    _C.load().b200_prefill_set_query_tiles(tiles)
    g = torch.Generator().manual_seed(5)
    for count in (256, 300):
        lens = torch.randint(0, 40, (count,), generator=g).tolist()
        lens[7], lens[200] = 200, 131
        T, H, G, D = sum(lens), 2, 1, 64
        q, k, v = (torch.randn(T, h, D, generator=g).half() for h in (H, G, G))
        cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
        got = ops.prefill_varlen_attn(q.cuda(), k.cuda(), v.cuda(), cu, cu, max(lens), max(lens), D ** -0.5, G).cpu().to(F64)
        at = 0
        for n in lens:
            if n:
                w = _want(q[at:at + n], k[at:at + n], v[at:at + n], D ** -0.5, 0.0, None)
                assert float((got[at:at + n] - w).abs().max()) < 4e-3, n
            at += n


def _want(q, k, v, scale, cap, sink):
    n, H, _ = q.shape
    m, G, _ = v.shape
    hidden = torch.arange(m)[None] > torch.arange(m - n, m)[:, None]
    out = []
    for h in range(H):
        s = q[:, h].to(F64) @ k[:, h * G // H].to(F64).T * scale
        s = (cap * torch.tanh(s / cap) if cap else s).masked_fill(hidden, -math.inf)
        s = torch.cat([s, sink[h].to(F64).expand(n, 1)], 1) if sink is not None else s
        out.append(torch.softmax(s, -1)[:, :m] @ v[:, h * G // H].to(F64))
    return torch.stack(out, 1).reshape(n, -1)


@pytest.fixture(autouse=True)
def _layout():
    from nanovllm import _C
    yield
    _C.load().b200_prefill_set_query_tiles(0)


@pytest.mark.parametrize("tiles", [0, 1, 2])
@pytest.mark.parametrize("H,G,D,cap,dtype", [(4, 2, 64, 30.0, torch.bfloat16), (3, 1, 128, 30.0, torch.float16),
                                             (6, 2, 64, 4.0, torch.float16), (4, 1, 128, 0.7, torch.bfloat16)])
def test_capped_scores_in_and_out_of_the_polynomial(H, G, D, cap, dtype, tiles):
    """cap 30: every score lies inside the range, but for one loud key that the rows behind it see (their tiles leave the
    polynomial, and the later ones with them); caps 4 and 0.7: most tiles lie outside."""
    from nanovllm import _C, ops
    _C.load().b200_prefill_set_query_tiles(tiles)
    g = torch.Generator().manual_seed(D + int(cap))
    lens = [1, 127, 128, 129, 300, 385]
    T = sum(lens)
    q, k, v = (torch.randn(T, h, D, generator=g).to(dtype) for h in (H, G, G))
    k[T - 200] *= 12
    sink = torch.randn(H, generator=g)
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    got = ops.prefill_varlen_attn(q.cuda(), k.cuda(), v.cuda(), cu, cu, max(lens), max(lens), D ** -0.5, G, softcap=cap,
                                  sink=sink.cuda()).cpu().to(F64)
    at = 0
    # P and the result in 16 bits: a rounding of either is 2^-9 (bf16) or 2^-12 (fp16) of values up to ~4, P V sums them
    tol = 3e-2 if dtype == torch.bfloat16 else 4e-3
    for n in lens:
        w = _want(q[at:at + n], k[at:at + n], v[at:at + n], D ** -0.5, cap, sink)
        assert float((got[at:at + n] - w).abs().max()) < tol, n
        at += n


@pytest.mark.parametrize("tiles", [0, 1, 2])
@pytest.mark.parametrize("H,block,D,spans", [(4, 16, 64, [(40, 700), (1, 17), (130, 130)]), (3, 32, 128, [(129, 641)]),
                                             (3, 64, 64, [(5, 900)]), (2, 128, 128, [(128, 385), (3, 3)]), (1, 256, 64, [(70, 600)])])
def test_cached_keys_in_blocks(H, block, D, spans, tiles):
    from nanovllm import _C, ops
    _C.load().b200_prefill_set_query_tiles(tiles)
    g = torch.Generator().manual_seed(block)
    G = 1
    need = [-(-m // block) for _, m in spans]
    order = torch.randperm(sum(need) + 2, generator=g).tolist()
    kc, vc = (torch.full((len(order), block, G * D), math.nan, dtype=torch.float16) for _ in range(2))
    table = torch.full((len(spans), max(need) + 1), -1, dtype=torch.int32)
    q = torch.randn(sum(n for n, _ in spans), H, D, generator=g).half()
    keys = []
    for s, (_, m) in enumerate(spans):
        k, v = (torch.randn(m, G, D, generator=g).half() for _ in range(2))
        keys.append((k, v))
        for b in range(need[s]):
            blk = table[s, b] = order.pop()
            for c, x in ((kc, k), (vc, v)):
                rows = x[b * block:(b + 1) * block].reshape(-1, G * D)
                c[blk] = 0                                   # rows of an owned block past the sequence hold finite values
                c[blk, :len(rows)] = rows
    cu = lambda i: torch.tensor([0] + [x[i] for x in spans]).cumsum(0).to(torch.int32).cuda()  # noqa: E731
    got = ops.prefill_varlen_attn(q.cuda(), kc.cuda(), vc.cuda(), cu(0), cu(1), max(n for n, _ in spans),
                                  max(m for _, m in spans), D ** -0.5, G, block_tables=table.cuda()).cpu().to(F64)
    at = 0
    for (n, m), (k, v) in zip(spans, keys):
        w = _want(q[at:at + n], k, v, D ** -0.5, 0.0, None)
        assert float((got[at:at + n] - w).abs().max()) < 4e-3, (n, m)
        at += n


@pytest.mark.parametrize("tiles", [1, 2])
@pytest.mark.parametrize("level", [0.05, 0.168, 0.172, 0.348, 0.352, 1.5])
@pytest.mark.parametrize("D,window", [(64, 0), (128, 0), (64, 100)])
def test_caps_on_either_side_of_both_polynomials(D, window, level, tiles):
    """The largest score of a head is `level` caps: the short polynomial, the long one and the function itself, on tiles with and without a mask
    (the maximum of a tile without one is capped by itself). A cap of 40 makes scores of up to 60: a wrong cap or maximum shows."""
    from nanovllm import _C, ops
    _C.load().b200_prefill_set_query_tiles(tiles)
    g = torch.Generator().manual_seed(D + window)
    H, G, lens, cap = 4, 2, [300, 129, 1], 40.0
    T = sum(lens)
    q, k, v = torch.randn(T, H, D, generator=g), torch.randn(T, G, D, generator=g), torch.randn(T, G, D, generator=g).half()
    q, k = q.half(), k.half()
    top = max(float((q[:, h].double() @ k[:, h * G // H].double().T).abs().max()) for h in range(H))
    scale = level * cap / top
    cu = torch.tensor([0] + lens).cumsum(0).to(torch.int32).cuda()
    got = ops.prefill_varlen_attn(q.cuda(), k.cuda(), v.cuda(), cu, cu, max(lens), max(lens), scale, G, softcap=cap, window=window).cpu().to(F64)
    at = 0
    for n in lens:
        out = []
        for h in range(H):
            s = cap * torch.tanh(q[at:at + n, h].to(F64) @ k[at:at + n, h * G // H].to(F64).T * scale / cap)
            i = torch.arange(n)
            seen = (i[None] <= i[:, None]) & ((i[:, None] - i[None] < window) if window else True)
            out.append(torch.softmax(s.masked_fill(~seen, -math.inf), -1) @ v[at:at + n, h * G // H].to(F64))
        want = torch.stack(out, 1).reshape(n, -1)
        # a probability is rounded to 2^-11, a result to 2^-11; scores of 32 bits move a probability of e^60 in all by 60 * 2^-23
        assert float((got[at:at + n] - want).norm() / want.norm()) < 6e-4
        at += n


@pytest.mark.parametrize("cap", [1e-8, 1e-4, 3e4, 1e9])
def test_caps_of_any_size(cap):
    """Scores of up to 0.15 caps, however small or large the cap is: its powers leave the range of 32 bits."""
    from nanovllm import ops
    g = torch.Generator().manual_seed(3)
    n, H, G, D = 200, 2, 1, 64
    q, k, v = (torch.randn(n, h, D, generator=g).bfloat16() for h in (H, G, G))
    top = max(float((q[:, h].double() @ k[:, 0].double().T).abs().max()) for h in range(H))
    q = (q * (0.15 * cap / (top * D ** -0.5))).bfloat16()
    cu = torch.tensor([0, n], dtype=torch.int32).cuda()
    got = ops.prefill_varlen_attn(q.cuda(), k.cuda(), v.cuda(), cu, cu, n, n, D ** -0.5, G, softcap=cap).cpu().to(F64)
    want = _want(q, k, v, D ** -0.5, cap, None)
    # scores up to 1.5e8: their spacing is 16, so that only the largest of a row counts, and near ties fall either way
    assert bool(got.isfinite().all())
    assert float(((got - want).abs().amax(1) > 3e-2).double().mean()) <= (0.02 if cap > 1e6 else 0.0)


@pytest.mark.parametrize("scale", [-0.125, -0.004])
def test_a_negative_scale(scale):
    """Scores far beyond the polynomials' range, and within: what decides is their size, whatever the sign."""
    from nanovllm import ops
    g = torch.Generator().manual_seed(4)
    n, H, G, D = 200, 2, 1, 64
    q, k, v = (torch.randn(n, h, D, generator=g).half() * s for h, s in ((H, 4.0), (G, 1.0), (G, 1.0)))
    cu = torch.tensor([0, n], dtype=torch.int32).cuda()
    got = ops.prefill_varlen_attn(q.cuda(), k.cuda(), v.cuda(), cu, cu, n, n, scale, G, softcap=5.0).cpu().to(F64)
    assert float((got - _want(q, k, v, scale, 5.0, None)).abs().max()) < 4e-3
