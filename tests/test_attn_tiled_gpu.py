"""Prompt portions of ops.attn_generic (csrc/attn_tiled.cu): 64-row, 64-key tiles against a 64-bit evaluation, at the
edges of the tiles, of the vector and scalar staging, and of every mask."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _want(q, k, v, past, scale, window, keep, chunk, cap, sink, gate):
    n, H, _ = q.shape
    m, G, dv = v.shape
    i, j = torch.arange(past, past + n)[:, None], torch.arange(m)[None]
    seen = j <= i
    if window:
        seen &= (i - j < window) | (j < keep)
    if chunk:
        seen &= i // chunk == j // chunk
    out = torch.zeros(n, H, dv, dtype=F64)
    for h in range(H):
        s = q[:, h].to(F64) @ k[:, h * G // H].to(F64).T * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].to(F64).expand(n, 1)], 1)
        p = torch.softmax(s, -1)[:, :m]
        for t in range(n):                                  # a hidden key's value takes no part, whatever it holds
            rows = seen[t]
            out[t, h] = p[t, rows] @ v[rows, h * G // H].to(F64)
        if gate is not None:
            out[:, h] *= torch.sigmoid(gate[:, h].to(F64))[:, None]
    return out


@pytest.mark.parametrize("H,G,dim,dv,dtype,spans,paged,kw", [
    (8, 2, 128, 128, torch.float32, [(64, 64), (1, 200), (63, 129), (2, 2)], 16, {}),
    (4, 4, 64, 64, torch.float32, [(65, 65), (16, 300)], 64, dict(window=33, keep_first=5)),
    (6, 1, 40, 24, torch.float32, [(11, 150), (70, 70)], 0, dict(latent=True, window=19)),
    (3, 3, 13, 21, torch.float32, [(17, 17), (90, 131)], 16, dict(chunk=48, softcap=3.0, sink=True, gate=True)),
    (2, 1, 256, 200, torch.bfloat16, [(64, 127), (9, 9)], 0, dict(sink=True)),
    (4, 2, 72, 136, torch.float16, [(130, 130)], 16, dict(gate=True, softcap=20.0)),
    (2, 2, 30, 66, torch.bfloat16, [(40, 40)], 0, {}),
])
def test_against_64_bit(H, G, dim, dv, dtype, spans, paged, kw):
    from nanovllm import ops
    g = torch.Generator().manual_seed(dim * dv + H)
    rnd = lambda *s: torch.randn(*s, generator=g).to(dtype)  # noqa: E731
    latent, window, keep, chunk = kw.get("latent", False), kw.get("window", 0), kw.get("keep_first", 0), kw.get("chunk", 0)
    cap, scale = kw.get("softcap", 0.0), dim ** -0.5
    T = sum(n for n, _ in spans)
    q = rnd(T, H, dim)
    sink = torch.randn(H, generator=g) if kw.get("sink") else None
    gate = rnd(T, H) if kw.get("gate") else None
    ks = [rnd(m, G, dim) for _, m in spans]
    vs = [k[:, :, :dv] if latent else rnd(m, G, dv) for k, (_, m) in zip(ks, spans)]
    if dtype == torch.float32 and not latent:
        vs[-1][-1] = math.inf                               # seen by the last token alone, in a tile that others share
    cu = lambda i: torch.tensor([0] + [s[i] for s in spans]).cumsum(0).to(torch.int32).cuda()  # noqa: E731
    sp = ops.StepSpans(cu(0), cu(1), None, max(n for n, _ in spans))
    extra = dict(window=window, keep_first=keep, chunk=chunk, softcap=cap, sink=None if sink is None else sink.cuda(),
                 gate=None if gate is None else gate.cuda())
    if paged:
        need = [-(-m // paged) for _, m in spans]
        order = torch.randperm(sum(need) + 2, generator=g).tolist()
        table = torch.full((len(spans), max(need)), -1, dtype=torch.int32)
        kc = torch.full((len(order), paged, G * dim), math.nan, dtype=dtype)     # what no sequence owns is never used
        vc = torch.full((len(order), paged, G * dv), math.nan, dtype=dtype)
        for s, n in enumerate(need):
            for b in range(n):
                blk = order.pop()
                table[s, b] = blk
                rows = ks[s][b * paged:(b + 1) * paged]
                kc[blk, :len(rows)] = rows.reshape(len(rows), -1)
                vc[blk, :len(rows)] = vs[s][b * paged:(b + 1) * paged].reshape(len(rows), -1)
        got = ops.attn_generic(q.cuda(), kc.cuda(), vc.cuda(), sp, scale, G, dv, block_tables=table.cuda(), **extra)
    else:
        got = ops.attn_generic(q.cuda(), torch.cat(ks).cuda(), None if latent else torch.cat(vs).cuda(), sp, scale, G, dv, **extra)
    got, at = got.cpu().to(F64).view(T, H, dv), 0
    # fp32: a score of ~4 sums dim products (a few 2^-24 each), weights and outputs follow it; 16-bit: the rounding of the result
    tol = 2e-5 if dtype == torch.float32 else 2 ** -8 if dtype == torch.bfloat16 else 2 ** -10
    for s, (n, m) in enumerate(spans):
        w = _want(q[at:at + n], ks[s], vs[s], m - n, scale, window, keep, chunk, cap, sink, None if gate is None else gate[at:at + n])
        x = got[at:at + n]
        fine = torch.isfinite(w)
        assert torch.equal(torch.isfinite(x), fine), s
        assert float(((x - w).abs() / w.abs().clamp(min=1.0))[fine].max()) < tol, s
        at += n
