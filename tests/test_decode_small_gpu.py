"""Paged decode attention of few rows (csrc/decode_small.cu: a cluster of CTAs per row and kv head) around the lines of its rule and the edges of its
units of 16 keys, against 64 bits; and against paged_decode_kernel (num_ctas given) where a table names no block, values are infinite, rows are empty."""
import math

import pytest
import torch

from test_decode_terms_gpu import _case, _want

pytestmark = pytest.mark.gpu


def _run(q, k, v, table, lens, G, ctas=0, **kw):
    from nanovllm import ops
    dev = lambda t: t.cuda()  # noqa: E731
    return ops.paged_decode_attn(dev(q), dev(k), dev(v), dev(table), torch.tensor(lens, dtype=torch.int32).cuda(), q.shape[2] ** -0.5, G, num_ctas=ctas, **kw).cpu()


# (heads, kv heads, size, lengths): 8, 4, 2 and 1 CTAs per cluster; one, two and 33 units of a warp; the widest tables of each line and one more
CASES = [(16, 8, 128, [1]), (16, 8, 128, [16, 17]), (16, 8, 128, [128, 129, 1, 100]), (16, 8, 128, [4096]), (16, 8, 128, [4097]), (8, 1, 128, [4090]),
         (32, 4, 128, [333, 2, 1025]), (16, 8, 128, [2048, 5, 700, 31, 33, 1, 64, 90]), (16, 8, 128, [2049] * 8), (8, 8, 64, [8192]), (8, 8, 64, [8193]),
         (32, 8, 64, [500, 1024, 15, 511, 513]), (8, 8, 64, [700] * 9), (8, 8, 64, [1000 - 30 * i for i in range(32)]), (8, 2, 128, [900] * 40),
         (8, 2, 128, [100] * 65), (32, 8, 64, [90] * 33)]


@pytest.mark.parametrize("H,G,D,lens", CASES)
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_the_result_is_the_rounded_one(H, G, D, lens, dtype):
    q, k, v, table = _case(H, G, D, lens, dtype, len(lens) + D)
    got, want = _run(q, k, v, table, lens, G), _want(q, k, v, table, lens, H, G, D).to(dtype)
    share = 0.04 if dtype == torch.bfloat16 else 0.01        # as in test_decode_terms_gpu.py: two terms of a probability
    assert float((got != want).float().mean()) < share


@pytest.mark.parametrize("H,G,D,lens", [(16, 8, 128, [1500]), (32, 4, 128, [700, 33, 0]), (8, 8, 64, [300] * 20)])
@pytest.mark.parametrize("softcap,with_sink", [(30.0, False), (0.0, True), (20.0, True)])
def test_cap_sink_and_empty_rows(H, G, D, lens, softcap, with_sink):
    q, k, v, table = _case(H, G, D, lens, torch.bfloat16, 3)
    sink = torch.linspace(-3, 3, H) if with_sink else None
    got = _run(q, k, v, table, lens, G, softcap=softcap, sink=sink.cuda() if with_sink else None)
    for b, n in enumerate(lens):
        if n == 0:
            assert torch.equal(got[b], torch.zeros_like(got[b]))
            continue
        kk, vv = (c[table[b, :-(-n // 16)].long()].reshape(-1, G, D)[:n].double().repeat_interleave(H // G, 1) for c in (k, v))
        s = torch.einsum("hd,nhd->hn", q[b].double(), kk) * D ** -0.5
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if with_sink:
            s = torch.cat([s, sink.double()[:, None]], 1)
        want = torch.einsum("hn,nhd->hd", torch.softmax(s, 1)[:, :n], vv).reshape(-1)
        assert float((got[b].double() - want).norm() / want.norm()) < 2.5e-3     # the rounding of the result (2^-9 at most, 2^-9 / sqrt 3 on average)


def test_blocks_that_are_not_there_and_infinite_values():
    H, G, D, lens = 16, 8, 128, [200, 40, 90]
    q, k, v, table = _case(H, G, D, lens, torch.bfloat16, 5)
    flat = v[table[0, 3]]
    flat[7, 5], flat[9, 200], flat[11, 300] = math.inf, -math.inf, math.nan
    v[table[0, 3]] = flat
    table[1, 1], table[2, 0] = -1, k.shape[0] + 5             # (zero keys and values)
    got, want = (_run(q, k, v, table, lens, G, c) for c in (0, 148))
    fine = torch.isfinite(want)
    assert torch.equal(torch.isnan(got), torch.isnan(want)) and torch.equal(got[torch.isinf(want)], want[torch.isinf(want)])
    assert float((got[fine].double() - want[fine].double()).abs().max()) < 8e-3
    # nothing past a row's length is read into it: stale values there may be anything
    k2, v2 = k.clone(), v.clone()
    k2[table[1, 2], 8:], v2[table[1, 2], 8:] = math.nan, math.nan
    assert torch.equal(_run(q, k2, v2, table, lens, G)[1], got[1])


def test_strided_queries_and_a_replayed_graph():
    from nanovllm import ops
    H, G, D, lens = 16, 8, 128, [700, 80]
    q, k, v, table = (t.cuda() for t in _case(H, G, D, lens, torch.bfloat16, 9))
    ctx = torch.tensor(lens, dtype=torch.int32, device="cuda")
    wide = torch.randn(2, H * D + 512, device="cuda").bfloat16()
    wide[:, :H * D] = q.reshape(2, -1)
    view = wide[:, :H * D].unflatten(1, (H, D))
    want = ops.paged_decode_attn(q, k, v, table, ctx, D ** -0.5, G)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = ops.paged_decode_attn(view, k, v, table, ctx, D ** -0.5, G)
    for _ in range(3):
        out.zero_()
        graph.replay()
        assert torch.equal(out, want)


# an e4m3 cache: 8, 4, 2 and 1 CTAs, one and several units of a warp, the widest tables of each line and one more
@pytest.mark.parametrize("H,G,D,lens", [(16, 8, 128, [1]), (16, 8, 128, [16, 17, 0, 129]), (8, 2, 128, [4096, 31]), (16, 8, 128, [4097]), (32, 4, 128, [333, 2, 1025]),
                                        (16, 8, 128, [2048, 5, 700, 31, 33, 1, 64, 90]), (16, 8, 128, [500] * 32), (8, 8, 64, [8192]), (32, 8, 64, [500, 1024, 15, 511, 513]),
                                        (8, 2, 64, [700] * 9), (8, 8, 64, [1000 - 15 * i for i in range(64)]), (32, 8, 64, [90] * 65)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_e4m3_cache(H, G, D, lens, dtype):
    """As close to 64 bits as paged_decode_fp8_kernel (num_ctas given): probabilities are f16 in both, 2^-11; results are rounded to `dtype`."""
    from nanovllm import ops
    q, k, v, table = _case(H, G, D, lens, dtype, len(lens) + D)
    k8, v8, ctx = k.to(torch.float8_e4m3fn), v.to(torch.float8_e4m3fn), torch.tensor(lens, dtype=torch.int32)
    for row in (i for i, n in enumerate(lens) if n % 16):     # stale bytes past a row's length decode to NaN
        block = table[row, lens[row] // 16]
        k8[block, lens[row] % 16:] = v8[block, lens[row] % 16:] = float("nan")
    run = lambda ctas: ops.paged_decode_attn_fp8(q.cuda(), k8.cuda(), v8.cuda(), table.cuda(), ctx.cuda(), D ** -0.5, G, k_scale=0.5, v_scale=2.0, num_ctas=ctas).cpu()  # noqa: E731
    got, ref = run(0), run(148)
    live = [i for i, n in enumerate(lens) if n]
    want = 2 * _want(q[live], k8.float() * 0.5, v8.float(), table[live], [lens[i] for i in live], H, G, D)
    off = lambda x: float((x[live].double() - want).norm() / want.norm())  # noqa: E731
    assert off(got) <= off(ref) * 1.05 + 1e-5, (off(got), off(ref))
    for i, n in enumerate(lens):
        if n == 0:
            assert torch.equal(got[i], torch.zeros_like(got[i]))


def test_the_workspace_is_asked_for_by_wide_steps_alone(monkeypatch):
    """Through the native call: one row takes none, more (row, kv head) pairs than the rule holds do; no rows at all are refused as they were."""
    from nanovllm import _C, ops
    if _C.calls() is None:
        pytest.skip("no native calls")
    H, G, D, asked, real = 16, 8, 128, [], ops.decode_workspace
    monkeypatch.setattr(ops, "decode_workspace", lambda *a: asked.append(a) or real(*a))
    for rows, wanted in ((1, 0), (40, 1)):
        q, k, v, table = (t.cuda() for t in _case(H, G, D, [90] * rows, torch.bfloat16, 1))
        ops.paged_decode_attn(q, k, v, table, torch.full((rows,), 90, dtype=torch.int32, device="cuda"), D ** -0.5, G)
        assert len(asked) == wanted
    with pytest.raises(_C.B200Error):
        ops.paged_decode_attn(q[:0], k, v, table[:0], torch.empty(0, dtype=torch.int32, device="cuda"), D ** -0.5, G)
