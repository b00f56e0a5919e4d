"""Prompt portions of ops.attn_generic in fp32 on the tensor cores (csrc/attn_split.cu): rows and keys around its 128-row and 64-key
tiles, head sizes that are padded, sinks, gates, values inside the key rows, packed and paged keys, against a 64-bit evaluation;
and values that three bf16 terms cannot carry. Tolerance: fp32 scores of a few units sum up to 128 products and enter an exponential."""
import math

import pytest
import torch
from test_attn_tiled_gpu import _want

pytestmark = pytest.mark.gpu
F64 = torch.float64


def _run(H, G, dim, dv, spans, paged, sink=False, gate=False, latent=False, poke=None, scale=None):
    from nanovllm import ops
    g = torch.Generator().manual_seed(dim * dv + H + len(spans))
    rnd = lambda *s: torch.randn(*s, generator=g)  # noqa: E731
    T, scale = sum(n for n, _ in spans), dim ** -0.5 if scale is None else scale
    q, sk, gt = rnd(T, H, dim), rnd(H) if sink else None, rnd(T, H) if gate else None
    ks = [rnd(m, G, dim) for _, m in spans]
    vs = [k[:, :, :dv] if latent else rnd(m, G, dv) for k, (_, m) in zip(ks, spans)]
    if poke:
        poke(q, ks, vs)
    cu = lambda i: torch.tensor([0] + [s[i] for s in spans]).cumsum(0).to(torch.int32).cuda()  # noqa: E731
    sp = ops.StepSpans(cu(0), cu(1), None, max(n for n, _ in spans))
    extra = dict(sink=None if sk is None else sk.cuda(), gate=None if gt is None else gt.cuda())
    if paged:
        need = [-(-m // paged) for _, m in spans]
        order = torch.randperm(sum(need) + 2, generator=g).tolist()
        table = torch.full((len(spans), max(need)), -1, dtype=torch.int32)
        kc, vc = (torch.full((len(order), paged, G * n), math.nan) for n in (dim, dv))   # what no sequence owns is never used
        for s, n in enumerate(need):
            for b in range(n):
                blk = order.pop()
                table[s, b] = blk
                for c, x in ((kc, ks), (vc, vs)):
                    rows = x[s][b * paged:(b + 1) * paged]
                    c[blk, :len(rows)] = rows.reshape(len(rows), -1)
        got = ops.attn_generic(q.cuda(), kc.cuda(), vc.cuda(), sp, scale, G, dv, block_tables=table.cuda(), **extra)
    else:
        got = ops.attn_generic(q.cuda(), torch.cat(ks).cuda(), None if latent else torch.cat(vs).cuda(), sp, scale, G, dv, **extra)
    at, out = 0, []
    for s, (n, m) in enumerate(spans):
        w = _want(q[at:at + n], ks[s], vs[s], m - n, scale, 0, 0, 0, 0.0, sk, None if gt is None else gt[at:at + n])
        out.append((got[at:at + n].cpu().to(F64).view(n, H, dv), w))
        at += n
    return out


@pytest.mark.parametrize("H,G,dim,dv,spans,paged,kw", [
    (8, 2, 128, 128, [(32, 32), (33, 64), (65, 129), (1, 63)], 16, {}),
    (2, 2, 64, 64, [(127, 127), (129, 192), (64, 65)], 0, dict(sink=True)),
    (3, 3, 48, 48, [(130, 200)], 16, dict(gate=True)),
    (6, 2, 20, 124, [(100, 100), (43, 300)], 64, dict(sink=True, gate=True)),
    (5, 1, 128, 36, [(26, 26), (77, 90)], 0, dict(latent=True)),
    (4, 1, 68, 128, [(64, 700)], 16, {}),
])
def test_against_64_bit(H, G, dim, dv, spans, paged, kw):
    for s, (x, w) in enumerate(_run(H, G, dim, dv, spans, paged, **kw)):
        assert float(((x - w).abs() / w.abs().clamp(min=1.0)).max()) < 2e-5, s


@pytest.mark.parametrize("bad", [math.inf, -math.inf, math.nan, 1e-36])
@pytest.mark.parametrize("where", ["q", "k", "v"])
def test_what_three_terms_cannot_carry(bad, where):
    def poke(q, ks, vs):                                       # seen by the second half of the second sequence's rows
        if where == "q":
            q[200, 1, 5] = bad
        else:
            (ks if where == "k" else vs)[1][150, 0, 7] = bad
    for s, (x, w) in enumerate(_run(4, 2, 64, 64, [(100, 100), (180, 200)], 16, poke=poke)):
        fine = torch.isfinite(w)
        assert torch.equal(torch.isfinite(x), fine), s
        assert float(((x - w).abs() / w.abs().clamp(min=1.0))[fine].max()) < 2e-5, s


@pytest.mark.parametrize("scale", [1e-19, 2e-4, 0.3, -0.3, 8e5, -9.9e5, 1.01e6, 3e7, 5e9, -5e9])
def test_scales_up_to_the_guard_and_past_it(scale):
    """Scores of a few units at every scale; past the guard another kernel takes over."""
    def poke(q, ks, vs):
        q *= 0.125 / scale
    for s, (x, w) in enumerate(_run(4, 2, 64, 64, [(70, 70), (64, 200)], 16, sink=True, poke=poke, scale=scale)):
        assert float(((x - w).abs() / w.abs().clamp(min=1.0)).max()) < 2e-5, s


@pytest.mark.parametrize("dim,scale", [(128, None), (64, 0.1), (64, -0.1), (64, 1e5)])
def test_scores_that_overflow(dim, scale):
    """Finite operands, scores of -1e39: no weight, also where a whole tile of keys has nothing else."""
    sign = -1.0 if scale is not None and scale < 0 else 1.0

    def poke(q, ks, vs):
        q[:, :, 0], q[:, :, 1:] = 1e20, q[:, :, 1:] * 1e20
        for k in ks:
            k[:, :, 1:] *= 1e-20 if scale != 1e5 else 1e6      # others of a few units; of 1e31 and more
            k[:, :, 0] = 0.0
            k[:66, :, 0] = -1e20 * sign
            k[70::7, :, 0] = -1e20 * sign
    for s, (x, w) in enumerate(_run(4, 2, dim, 64, [(100, 200), (64, 130)], 16, poke=poke, scale=scale)):
        assert float(((x - w).abs() / w.abs().clamp(min=1.0)).max()) < 2e-5, s


@pytest.mark.parametrize("sink", [False, True])
def test_scores_of_many_digits(sink):
    """Scores around 1e10, whose spacing in fp32 is a thousand: the largest takes all (the next are millions below)."""
    def poke(q, ks, vs):
        q *= 1e5
        for k in ks:
            k *= 1e5
    for s, (x, w) in enumerate(_run(4, 2, 128, 128, [(100, 100), (64, 200)], 16, sink=sink, poke=poke)):
        assert float(((x - w).abs() / w.abs().clamp(min=1.0)).max()) < 2e-5, s


@pytest.mark.parametrize("qs,ks,vs", [(1, 1, 1e-36), (1, 1, 2e-42), (1e-37, 1, 1), (1, 1e-40, 1), (2.0 ** 76, 2.0 ** -76, 1), (2.0 ** 76, 2.0 ** -110, 1),
                                      (2.0 ** -110, 2.0 ** 100, 1), (1, 1, 2.0 ** 78), (1, 1, 2.0 ** 90), (1, 1, 2.0 ** 115)])
def test_small_and_large_operands(qs, ks, vs):
    """fp32 accuracy over fp32's range: one operand small or large, and small ones against large ones. Values end at 2^115, since the sums
    of up to 200 weights of at most 1 and values of up to 5 times that are kept in fp32 before they are divided (2^115 x 1000 < 2^128)."""
    def poke(q, kk, vv):
        q *= qs
        for k, v in zip(kk, vv):
            k *= ks
            v *= vs
    for s, (x, w) in enumerate(_run(4, 2, 64, 64, [(70, 70), (64, 200)], 16, poke=poke)):
        size = float(w.abs().max())
        floor = 2.0 ** -149 / size                             # one step of the smallest numbers
        assert float(((x - w).abs() / w.abs().clamp(min=0.3 * size)).max()) < 2e-5 + 4 * floor, s


# ---- row tiles whose keys two CTAs share: few of them, and spans of 384 rows and more (every test above stays below)
LONG = [(390, 900), (5, 5), (200, 333)]


@pytest.mark.parametrize("H,G,dim,dv,paged,kw", [(8, 2, 128, 128, 16, {}), (4, 2, 64, 64, 0, dict(sink=True)), (3, 3, 48, 48, 16, dict(gate=True)),
                                                 (2, 1, 20, 124, 64, dict(sink=True, gate=True)), (2, 1, 128, 36, 0, dict(latent=True))])
def test_shared_keys_against_64_bit(H, G, dim, dv, paged, kw):
    """Key tiles from one (a CTA alone) to fifteen, in odd and even numbers, parts that some rows see nothing of."""
    for s, (x, w) in enumerate(_run(H, G, dim, dv, LONG, paged, **kw)):
        assert float(((x - w).abs() / w.abs().clamp(min=1.0)).max()) < 2e-5, s
    (x, w), = _run(H, G, dim, dv, [(449, 449)], paged, **kw)
    assert float(((x - w).abs() / w.abs().clamp(min=1.0)).max()) < 2e-5


@pytest.mark.parametrize("bad", [math.inf, math.nan, 1e-36])
@pytest.mark.parametrize("where,at", [("q", 300), ("k", 10), ("k", 880), ("v", 10), ("v", 880)])
def test_shared_keys_that_three_terms_cannot_carry(bad, where, at):
    """Met by either of the two CTAs: the rows are computed once more, from all keys."""
    def poke(q, ks, vs):
        if where == "q":
            q[at, 1, 5] = bad
        else:
            (ks if where == "k" else vs)[0][at, 0, 7] = bad
    for s, (x, w) in enumerate(_run(4, 2, 64, 64, LONG, 16, poke=poke)):
        fine = torch.isfinite(w)
        assert torch.equal(torch.isfinite(x), fine), s
        assert float(((x - w).abs() / w.abs().clamp(min=1.0))[fine].max()) < 2e-5, s


@pytest.mark.parametrize("kind", ["far", "overflow", "one part has it all", "negative scale"])
@pytest.mark.parametrize("sink", [False, True])
def test_shared_keys_and_scores_of_any_size(kind, sink):
    scale = -0.3 if kind == "negative scale" else None

    def poke(q, ks, vs):
        if kind == "far":                                      # around 1e10: their spacing is a thousand
            q *= 1e5
            for k in ks:
                k *= 1e5
        elif kind == "overflow":                               # finite operands, scores of -1e39 in the first part alone
            q[:, :, 0], q[:, :, 1:] = 1e20, q[:, :, 1:] * 1e20
            for k in ks:
                k[:, :, 1:] *= 1e-20
                k[:, :, 0] = 0.0
                k[:len(k) // 3 if len(k) > 5 else 0, :, 0] = -1e20      # (the span of five has rows that would see nothing else)
        elif kind == "one part has it all":                    # a key of the second part, hundreds above the others
            q[:, :, 0] = 8.0
            ks[0][700, :, 0] = 1000.0
    for s, (x, w) in enumerate(_run(4, 2, 128, 128, LONG, 16, sink=sink, poke=poke, scale=scale)):
        assert float(((x - w).abs() / w.abs().clamp(min=1.0)).max()) < 2e-5, s


@pytest.mark.parametrize("score", [35, 350, 3500])
@pytest.mark.parametrize("seed", [1, 2])
def test_shared_keys_lose_nothing_where_both_parts_count(monkeypatch, score, seed):
    """The largest scores of a row's two parts lie 0.7 apart: merged, the row is as near to 64 bits as where one CTA has all keys (the same scores,
    whose own rounding is most of the error: a residual of the merge adds 8 to 20 % to it, its rounding nothing that shows)."""
    from types import SimpleNamespace

    from nanovllm import _C, ops
    g, lib = torch.Generator().manual_seed(seed), _C.load()
    H, G, d, n = 8, 2, 128, 600
    q, k, v = (torch.randn(n, h, d, generator=g) * s for h, s in ((H, 0.1), (G, 0.1), (G, 1.0)))
    u = torch.nn.functional.normalize(torch.randn(d, generator=g), dim=0) * 11.3
    k[10], k[500] = u, u * (1 + 0.7 / score)
    q += u * score * d ** 0.5 / 11.3 ** 2 * (1 + 0.01 * torch.rand(n, H, 1, generator=g))
    cu = torch.tensor([0, n], dtype=torch.int32).cuda()
    call = lambda: ops.attn_generic(q.cuda(), k.cuda(), v.cuda(), ops.StepSpans(cu, cu, None, n), d ** -0.5, G, d)  # noqa: E731
    want = _want(q, k, v, 0, d ** -0.5, 0, 0, 0, 0.0, None, None)
    off = lambda x: float((x.cpu().to(F64).view(want.shape) - want)[501:].norm())  # noqa: E731
    shared = call()
    monkeypatch.setattr(_C, "load", lambda: SimpleNamespace(b200_attn_generic_step=lambda *a: lib.b200_attn_generic_step(*a[:-2], 0, a[-1])))
    alone = call()
    assert not torch.equal(shared, alone)
    assert off(shared) <= 1.03 * off(alone), (off(shared), off(alone))
