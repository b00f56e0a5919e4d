"""-m gpu: the sparse-MoE kernels (csrc/moe.cu, csrc/moe_umma.cu) and the Qwen3-MoE engine against
the reference-generated goldens (tests/golden/moe.pt) and the CPU oracle (oracle/moe_ref.py).

Tolerances. Routing: expert ids must equal the reference's wherever the reference's own
probabilities are not tied at the top-k boundary; weights within one rounding of the model dtype.
Expert MLPs: the product accumulates each GEMM in fp32 on tensor cores, the CPU reference in its
own blocking; both round to bf16 at the same points (gate_up, silu, h, expert output, weighted
output, every combine add), so elementwise differences are a few bf16 ulps of the largest
magnitude: max |diff| <= 3e-2 * max |ref|, mean |diff| <= 4e-3 * mean |ref|.
"""
import os

import pytest
import torch

from oracle import moe_ref

pytestmark = pytest.mark.gpu

BLOCK_CASES = ("e8_k2", "e32_k4", "e128_k8", "single_token")


def moe_block_weights(E, hidden, inter, seed, dtype=torch.bfloat16):
    g = torch.Generator().manual_seed(seed)
    gate = torch.randn(E, hidden, generator=g).to(dtype)
    w13 = (0.1 * torch.randn(E, 2 * inter, hidden, generator=g)).to(dtype)
    w2 = (0.1 * torch.randn(E, hidden, inter, generator=g)).to(dtype)
    return gate, w13, w2


def _close(got, want, what):
    got, want = got.float().cpu(), want.float().cpu()
    d = (got - want).abs()
    assert d.max() <= 3e-2 * want.abs().max() + 1e-6, (what, float(d.max()), float(want.abs().max()))
    assert d.mean() <= 4e-3 * want.abs().mean() + 1e-7, (what, float(d.mean()), float(want.abs().mean()))


@pytest.mark.parametrize("name", BLOCK_CASES)
def test_route_matches_reference(golden_moe, name):
    from nanovllm import ops
    g = golden_moe[name]
    ids, w = ops.moe_route(g["logits"].cuda(), g["top_k"])
    ids, w = ids.cpu(), w.cpu()
    # rows whose k-th and (k+1)-th probabilities differ (and no duplicates inside the top k) are decided
    p = torch.softmax(g["logits"].float(), dim=1)
    top = p.topk(min(g["top_k"] + 1, p.shape[1]), dim=1).values
    decided = (top[:, :-1] > top[:, 1:]).all(dim=1)
    assert decided.float().mean() > 0.5
    assert torch.equal(ids[decided], g["topk_ids"][decided])
    dw = (w.float() - g["topk_weights"].float()).abs()[decided]
    assert dw.max() <= 2 ** -7 * g["topk_weights"].float().max(), float(dw.max())
    # undecided rows: still a valid top-k set of the same probabilities
    for t in (~decided).nonzero().flatten().tolist():
        assert sorted(p[t, ids[t].long()].tolist(), reverse=True) == pytest.approx(
            sorted(p[t, g["topk_ids"][t].long()].tolist(), reverse=True), rel=1e-5)


def test_route_fp16_and_odd_expert_counts():
    from nanovllm import ops
    g = torch.Generator().manual_seed(5)
    for E, k, T, dt in ((5, 2, 9, torch.float16), (48, 6, 70, torch.bfloat16), (256, 8, 33, torch.bfloat16),
                        (33, 1, 4, torch.float16)):
        logits = (2 * torch.randn(T, E, generator=g)).to(dt)
        ids, w = ops.moe_route(logits.cuda(), k)
        p = torch.softmax(logits.float(), dim=1)
        wv, wi = p.topk(k, dim=1)
        want_w = (wv / wv.sum(-1, keepdim=True)).to(dt)
        # values of the selected experts must be the k largest (ties may pick another index)
        sel = p.gather(1, ids.cpu().long())
        assert torch.allclose(sel, wv, rtol=1e-5, atol=0)
        assert (w.cpu().float() - want_w.float()).abs().max() <= 2 ** -7
        assert (w.cpu().float().sum(-1) - 1).abs().max() < 0.02


@pytest.mark.parametrize("T,k,E,begin,n", [(37, 2, 8, 0, 8), (256, 8, 128, 0, 128), (256, 8, 128, 32, 16),
                                            (1, 8, 128, 112, 16), (50, 4, 32, 8, 8), (4096, 8, 128, 0, 128),
                                            (300, 8, 128, 0, 16), (16384, 8, 128, 64, 64)])
def test_align_is_the_oracle_dispatch_plan(T, k, E, begin, n):
    from nanovllm import ops
    g = torch.Generator().manual_seed(T + k)
    ids = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(min(T, 512))]).to(torch.int32)
    if T > 512:
        ids = ids.repeat((T + 511) // 512, 1)[:T].contiguous()
    plan = ops.moe_align(ids.cuda(), begin, n)
    off, sp, pos = moe_ref.dispatch_plan(ids, begin, n)
    nl = int(off[-1])
    assert torch.equal(plan.offsets.cpu(), off)
    assert torch.equal(plan.sorted_pair.cpu()[:nl], sp)
    assert torch.equal(plan.pos_of_pair.cpu(), pos)


@pytest.mark.parametrize("name", BLOCK_CASES)
def test_expert_mlps_and_combine_match_reference_block(golden_moe, name):
    """Reference routing fed in (no near-tie ambiguity): gate_up GEMM + SiluAndMul, down GEMM +
    routing weight, ascending-expert combine against Qwen3MoeSparseMoeBlock's output."""
    from nanovllm import ops
    g = golden_moe[name]
    E = g["experts"]
    _, w13, w2 = moe_block_weights(E, g["hidden"], g["inter"], g["seed"])
    x, ids, w = g["x"].cuda(), g["topk_ids"].cuda(), g["topk_weights"].cuda()
    plan = ops.moe_align(ids, 0, E)
    y = ops.moe_experts(x, w13.cuda(), w2.cuda(), ids, w, plan)
    _close(y, g["out"], name)
    # expert-parallel partials (2 and 4 ranks): each equals the oracle's partial, and they sum to the whole
    for world in (2, 4):
        if E % world:
            continue
        total = torch.zeros_like(g["out"], dtype=torch.float32)
        for r in range(world):
            n = E // world
            plan = ops.moe_align(ids, r * n, n)
            part = ops.moe_experts(x, w13[r * n:(r + 1) * n].contiguous().cuda(),
                                   w2[r * n:(r + 1) * n].contiguous().cuda(), ids, w, plan)
            want = moe_ref.sparse_moe_block(g["x"], moe_block_weights(E, g["hidden"], g["inter"], g["seed"])[0],
                                            w13, w2, g["top_k"], experts=set(range(r * n, (r + 1) * n)))
            _close(part, want, f"{name} rank {r}/{world}")
            total += part.float().cpu()
        _close(total, g["out"], f"{name} sum of {world} partials")


@pytest.mark.parametrize("T,k,E,hidden,inter", [(256, 8, 128, 512, 256),      # decode-like: ~16 rows per expert
                                                 (64, 8, 128, 2048, 768),      # Qwen3-30B-A3B expert shapes
                                                 (700, 2, 4, 256, 128),        # ~350 rows per expert: many passes
                                                 (97, 1, 3, 128, 64)])         # top-1, ragged
def test_expert_mlps_against_fp32_evaluation(T, k, E, hidden, inter):
    """Larger shapes than the goldens hold: against an fp32 evaluation of the same block on the GPU
    with the reference's rounding points restated in torch."""
    from nanovllm import ops
    g = torch.Generator().manual_seed(E * 1000 + T)
    bf = torch.bfloat16
    x = torch.randn(T, hidden, generator=g).to(bf).cuda()
    w13 = (hidden ** -0.5 * torch.randn(E, 2 * inter, hidden, generator=g)).to(bf).cuda()
    w2 = (inter ** -0.5 * torch.randn(E, hidden, inter, generator=g)).to(bf).cuda()
    ids = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)]).to(torch.int32).cuda()
    w = torch.rand(T, k, generator=g)
    w = (w / w.sum(-1, keepdim=True)).to(bf).cuda()
    plan = ops.moe_align(ids, 0, E)
    y = ops.moe_experts(x, w13, w2, ids, w, plan)
    want = torch.zeros(T, hidden, dtype=bf, device="cuda")
    for e in range(E):
        tok, slot = torch.where(ids == e)
        if tok.numel() == 0:
            continue
        gu = (x[tok].float() @ w13[e].float().T).to(bf)
        h = torch.nn.functional.silu(gu[:, :inter]) * gu[:, inter:]
        out = (h.float() @ w2[e].float().T).to(bf) * w[tok, slot, None]
        want.index_add_(0, tok, out)
    _close(y, want, (T, k, E, hidden, inter))
    # rows of the plan beyond the local pairs must never be touched: all experts local here -> T*k rows
    assert int(plan.offsets[-1]) == T * k


def test_tiny_qwen3_moe_engine_against_reference_run(golden_moe):
    """LLM('tiny-qwen3-moe') teacher-forced along the reference run. A router near-tie resolved the
    other way changes a token's experts (and its logits visibly), so the bound is statistical: the
    median row error must be at the bf16 noise level and >= 85 % of the (step, sequence) rows must
    be within the dense-model bound and pick the reference token."""
    from nanovllm import LLM, SamplingParams
    g = golden_moe["tiny_qwen3_moe"]
    llm = LLM("tiny-qwen3-moe", seed=g["seed"], norm_jitter=g["norm_jitter"], enforce_eager=True,
              kvcache_block_size=16, max_num_seqs=8, max_model_len=256, max_num_batched_tokens=1024,
              num_kvcache_blocks=128)
    runner = llm.model_runner
    orig, logs, picked, step = runner.sampler.forward, [], [], [0]

    def spy(logits, *a, **kw):
        logs.append(logits.float().cpu())
        out = orig(logits, *a, **kw)
        picked.append(out.cpu().tolist())
        if step[0] < g["max_tokens"]:
            out.copy_(torch.tensor([t[step[0]] for t in g["tokens"]], dtype=out.dtype, device=out.device))
        step[0] += 1
        return out
    runner.sampler.forward = spy
    llm.generate(g["prompts"], SamplingParams(temperature=1.0, max_tokens=g["max_tokens"], ignore_eos=True,
                                              greedy=True), use_tqdm=False)
    llm.exit()
    got = torch.stack(logs)                                   # [steps, B, vocab]
    row_err = (got - g["logits"]).abs().amax(-1).flatten()
    same_tok = torch.tensor([[picked[s][b] == g["tokens"][b][s] for b in range(len(g["prompts"]))]
                             for s in range(g["max_tokens"])]).flatten()
    assert row_err.median() < 0.03, float(row_err.median())
    assert (row_err < 0.06).float().mean() >= 0.85, row_err
    assert same_tok.float().mean() >= 0.85, same_tok


def test_tiny_qwen3_moe_cuda_graph_equals_eager():
    import random
    from nanovllm import LLM, SamplingParams
    rnd = random.Random(4)
    prompts = [[rnd.randint(0, 511) for _ in range(n)] for n in (9, 40, 16, 3)]
    sp = SamplingParams(temperature=1.0, max_tokens=24, ignore_eos=True, greedy=True)
    outs = []
    for eager in (True, False):
        llm = LLM("tiny-qwen3-moe", seed=2, norm_jitter=0.1, enforce_eager=eager, kvcache_block_size=16,
                  max_num_seqs=8, max_model_len=256, max_num_batched_tokens=1024, num_kvcache_blocks=128)
        outs.append([o["token_ids"] for o in llm.generate(prompts, sp, use_tqdm=False)])
        llm.exit()
    assert outs[0] == outs[1]


@pytest.mark.parametrize("big", ["umma", "library"])
def test_big_gemm_paths_match_the_streaming_kernels(monkeypatch, big):
    """ops._MOE_BIG_GEMM: prefill-sized batches through the tcgen05 grouped GEMM (csrc/moe_umma.cu) or
    through torch._grouped_mm must agree with the weight-streaming expert GEMMs -- full and
    expert-parallel plans, row counts that are not multiples of the 128-row tile, an empty expert."""
    from nanovllm import ops
    g = torch.Generator().manual_seed(9)
    bf = torch.bfloat16
    for T, k, E, hidden, inter in ((1500, 4, 8, 256, 128), (333, 2, 4, 2048, 768), (700, 1, 3, 128, 64)):
        x = torch.randn(T, hidden, generator=g).to(bf).cuda()
        w13 = (hidden ** -0.5 * torch.randn(E, 2 * inter, hidden, generator=g)).to(bf).cuda()
        w2 = (inter ** -0.5 * torch.randn(E, hidden, inter, generator=g)).to(bf).cuda()
        ids = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)]).to(torch.int32)
        if E == 3:
            ids[ids == 1] = 2                           # expert 1 receives nothing
        ids = ids.cuda()
        w = torch.rand(T, k, generator=g)
        w = (w / w.sum(-1, keepdim=True)).to(bf).cuda()
        for begin, n in ((0, E), (E // 2, E - E // 2)):
            plan = ops.moe_align(ids, begin, n)
            wa, wb = w13[begin:begin + n].contiguous(), w2[begin:begin + n].contiguous()
            monkeypatch.setattr(ops, "_MOE_BIG_GEMM", "stream")
            a = ops.moe_experts(x, wa, wb, ids, w, plan)
            monkeypatch.setattr(ops, "_MOE_BIG_GEMM", big)
            monkeypatch.setattr(ops, "_MOE_BIG_GEMM_ROWS", 1)
            b = ops.moe_experts(x, wa, wb, ids, w, plan)
            _close(b, a, f"{big} vs streaming kernel, T={T} experts [{begin},{begin + n})")


@pytest.mark.parametrize("M,K,inter", [(256, 1024, 3072), (7, 128, 64), (300, 5120, 3200), (128, 2048, 768)])
def test_dense_layers_on_the_grouped_tcgen05_kernel(M, K, inter):
    """ops.gate_up_silu_umma / ops.linear_umma: the grouped kernel as a one-expert group = an ordinary
    (fused) linear layer; against cuBLAS + the validated silu_and_mul kernel."""
    from nanovllm import ops
    g = torch.Generator().manual_seed(M + K)
    bf = torch.bfloat16
    x = torch.randn(M, K, generator=g).to(bf).cuda()
    w = (K ** -0.5 * torch.randn(2 * inter, K, generator=g)).to(bf).cuda()
    _close(ops.gate_up_silu_umma(x, w), ops.silu_and_mul(torch.nn.functional.linear(x, w)), ("gate_up", M, K, inter))
    if (2 * inter) % 128 == 0:
        _close(ops.linear_umma(x, w), torch.nn.functional.linear(x, w), ("linear", M, K, inter))


@pytest.mark.parametrize("dtype,k,hidden,inter,weigh_input", [
    (torch.bfloat16, 1, 256, 128, False), (torch.float16, 2, 512, 256, True), (torch.bfloat16, 1, 768, 384, False)])
def test_persistent_256_column_tiles(monkeypatch, dtype, k, hidden, inter, weigh_input):
    """moe_umma_wide_kernel at its edges: an empty expert, experts of 1, 127, 128, 129 and many rows, fewer K blocks than
    ring stages, one column band and several, weights on the input or the output; against the weight-streaming kernels."""
    from nanovllm import ops
    g = torch.Generator().manual_seed(hidden + k)
    counts = [0, 1, 127, 128, 129, 640, 0, 18975 // k]
    E, T = len(counts), max(sum(counts), 19000 // k)
    first = torch.repeat_interleave(torch.arange(E), torch.tensor(counts[:-1] + [T - sum(counts[:-1])]))
    ids = first[torch.randperm(T, generator=g)].view(T, 1)
    if k == 2:
        ids = torch.cat([ids, (ids + 1 + torch.randint(0, E - 1, (T, 1), generator=g)) % E], 1)
    ids = ids.to(torch.int32).cuda()
    x = torch.randn(T, hidden, generator=g).to(dtype).cuda()
    w13 = (hidden ** -0.5 * torch.randn(E, 2 * inter, hidden, generator=g)).to(dtype).cuda()
    w2 = (inter ** -0.5 * torch.randn(E, hidden, inter, generator=g)).to(dtype).cuda()
    w = torch.rand(T, k, generator=g).to(torch.float32 if weigh_input else dtype).cuda()
    plan = ops.moe_align(ids, 0, E)
    monkeypatch.setattr(ops, "_MOE_BIG_GEMM", "stream")
    a = ops.moe_experts(x, w13, w2, ids, w, plan, weigh_input=weigh_input)
    monkeypatch.setattr(ops, "_MOE_BIG_GEMM", "umma")
    b = ops.moe_experts(x, w13, w2, ids, w, plan, weigh_input=weigh_input)
    _close(b, a, f"hidden {hidden}, inter {inter}")


@pytest.mark.parametrize("T,k,E,begin,n,shift", [(1, 1, 1, 0, 1, 0), (16, 8, 128, 0, 128, 0), (127, 1, 8, 2, 5, 1),
                                                 (513, 8, 128, 96, 32, 3), (5000, 4, 256, 0, 256, 0), (9001, 1, 3, 1, 2, 2)])
def test_plan_is_a_stable_sort_by_expert(T, k, E, begin, n, shift):
    """b200_moe_align on short and long pair lists, at the edges of the 128-pair vectors, with ids that do not start on a
    16-byte boundary and experts that live elsewhere: exactly numpy's stable sort."""
    import numpy as np
    from nanovllm import ops
    g = torch.Generator().manual_seed(T)
    ids = torch.randint(0, E, (T, k), generator=g, dtype=torch.int32)
    store = torch.zeros(T * k + 4, dtype=torch.int32, device="cuda")
    dev = store[shift:shift + T * k].view(T, k)
    dev.copy_(ids)
    plan = ops.moe_align(dev, begin, n)
    flat = ids.flatten().numpy()
    local = np.flatnonzero((flat >= begin) & (flat < begin + n))
    order = local[np.argsort(flat[local], kind="stable")]
    pos = np.full(T * k, -1)
    pos[order] = np.arange(len(order))
    assert (plan.sorted_pair.cpu().numpy()[:len(order)] == order).all()
    assert (plan.pos_of_pair.cpu().numpy() == pos).all()
    counts = np.bincount(flat[local] - begin, minlength=n)
    assert (plan.offsets.cpu().numpy() == np.concatenate([[0], np.cumsum(counts)])).all()


def test_a_wait_that_runs_out_is_reported():
    """The persistent grouped GEMM with no patience at all: it leaves with copies and products under way, the status word is
    set, the next call raises, and the one after it is right."""
    from nanovllm import _C, ops
    lib = _C.load()
    M, K, N = 20000, 768, 512
    g = torch.Generator().manual_seed(3)
    x, w = (torch.randn(r, K, generator=g).bfloat16().cuda() for r in (M, N))
    want = (x.float() @ w.float().T).bfloat16()
    offsets, out = torch.tensor([0, M], dtype=torch.int32, device="cuda"), torch.zeros(M, N, dtype=x.dtype, device="cuda")
    torch.cuda.synchronize()
    ops.check_waits()
    _C.check(lib.b200_moe_gemm_down_umma_bounded(out.data_ptr(), x.data_ptr(), w.data_ptr(), offsets.data_ptr(), M, K, N, 1,
                                                 _C.BF16, 0, torch.cuda.current_stream().cuda_stream), "bounded")
    torch.cuda.synchronize()
    with pytest.raises(_C.B200Error, match="ran out"):
        ops.linear_umma(x, w)
    _close(ops.linear_umma(x, w), want, "after it")
    torch.cuda.synchronize()
    ops.check_waits()


@pytest.mark.parametrize("dtype,M,K,inter", [(torch.bfloat16, 19000, 64, 128), (torch.float16, 9600, 320, 256), (torch.bfloat16, 18945, 256, 256)])
def test_persistent_tiles_against_plain_products(dtype, M, K, inter):
    """The persistent 256-column kernel as dense layers (one group; full row tiles give every SM one) against fp32 products:
    one K block and more, M at and off a multiple of 128."""
    from nanovllm import ops
    g = torch.Generator().manual_seed(M)
    x = torch.randn(M, K, generator=g).to(dtype).cuda()
    w = (K ** -0.5 * torch.randn(2 * inter, K, generator=g)).to(dtype).cuda()
    product = (x.float() @ w.float().T).to(dtype)
    _close(ops.linear_umma(x, w), product, ("linear", M, K, inter))
    gate, up = product.float().split(inter, 1)
    _close(ops.gate_up_silu_umma(x, w), (torch.nn.functional.silu(gate).to(dtype).float() * up).to(dtype), ("gate_up", M, K, inter))
